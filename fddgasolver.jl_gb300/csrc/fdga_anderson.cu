// fdga_anderson.cu -- device-resident Anderson acceleration (NLsolve method=:anderson).
//
// The update of one Anderson step (NLsolve 4.5.1 anderson.jl, Walker & Ni 2011; driven by
// src/solve.jl:179-188 of the reference) runs without a host round trip: the QR factor R, the
// Givens parameters of a column deletion, the Gram-Schmidt coefficients and γ = R⁻¹ Qᴴ f live in
// device memory, and each long-vector pass reduces its block partials into the coefficient it
// needs at the start of the next pass.  Every block reduces the same partials in the same fixed
// order, so all blocks use bit-identical coefficients.  Arithmetic order per element matches the
// serial restatement: modified Gram-Schmidt one column at a time, rotations i = 1..m-1 in order,
// x -= γ_i Δg_i for i = 0..m_eff-1 in order.
#include "fdga_kernels.h"

namespace fdga {

namespace {

constexpr int RT = 256;  // threads of every reduction block

// The long-vector passes are bound by GB300's FP64 pipe: complex products are written as FMAs.
// conj(a) b + c
__device__ __forceinline__ cplx cfma_conj(cplx a, cplx b, cplx c) {
    return mk(fma(a.x, b.x, fma(a.y, b.y, c.x)), fma(a.x, b.y, fma(-a.y, b.x, c.y)));
}
// c - a b
__device__ __forceinline__ cplx cfnma(cplx a, cplx b, cplx c) {
    return mk(fma(-a.x, b.x, fma(a.y, b.y, c.x)), fma(-a.x, b.y, fma(-a.y, b.x, c.y)));
}

// Block sum of per-thread values in a fixed order, valid in all threads: shuffles within the warps, then the
// warps' sums in order.  One barrier; sh (one entry per warp) is used once per kernel.
__device__ __forceinline__ cplx block_sum(cplx v, cplx (&sh)[RT / 32]) {
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    cplx r = sh[0];
#pragma unroll
    for (int w = 1; w < RT / 32; ++w) r += sh[w];
    return r;
}
// Sum of part[0..np), identical in every block.
__device__ __forceinline__ cplx block_reduce_parts(const cplx* part, int np, cplx (&sh)[RT / 32]) {
    cplx s = mk(0.0, 0.0);
    for (int i = threadIdx.x; i < np; i += RT) s += ld16(part + i);
    return block_sum(s, sh);
}
// Block partial of a per-thread value, written to out[blockIdx.x].
__device__ __forceinline__ void block_store_partial(cplx v, cplx (&sh)[RT / 32], cplx* out) {
    const cplx r = block_sum(v, sh);
    if (threadIdx.x == 0) out[blockIdx.x] = r;
}

// Storage of the vectors.  Without symmetry groups every vector has one value per state element.
// With them, every iterate is a complex combination of class-symmetric vectors, so all members of a
// class that carry the same conjugation hold the same value up to their sign: the vectors keep one
// value per (class, conjugation) pair, the "keys" (key = 2·class + conj), and inner products weight a
// key by its number of members.  That is the full-vector arithmetic, elementwise the same operations,
// on 1/8 to 1/16 of the elements (Hubbard 8x8, nK3 = (8, 12): 1.87 M elements, 0.19 M keys).

// code of a state element (class * 4 + op) -> its key and sign
__device__ __forceinline__ uint32_t key_of(uint32_t code) { return ((code >> 2) << 1) | ((code >> 1) & 1u); }
__device__ __forceinline__ cplx signed_(cplx v, uint32_t neg) {
    return neg ? mk(neg_exact(v.x), neg_exact(v.y)) : v;
}
// first member and number of members of each key (src preset to 0xffffffff, w to 0)
__global__ void __launch_bounds__(RT) k_aa_keys(const uint32_t* code, uint32_t* src, double* w, size_t n) {
    for (size_t j = blockIdx.x * (size_t)RT + threadIdx.x; j < n; j += (size_t)gridDim.x * RT) {
        const uint32_t k = key_of(code[j]);
        atomicMin(&src[k], (uint32_t)j);
        atomicAdd(&w[k], 1.0);
    }
}
// number of elements of x that differ from their key's value (a NaN differs)
__global__ void __launch_bounds__(RT) k_aa_check(const cplx* x, const uint32_t* code, const uint32_t* src,
                                                 unsigned int* count, size_t n) {
    unsigned int bad = 0;
    for (size_t j = blockIdx.x * (size_t)RT + threadIdx.x; j < n; j += (size_t)gridDim.x * RT) {
        const uint32_t c = code[j], s = src[key_of(c)];
        const cplx a = signed_(x[j], c & 1u), b = signed_(x[s], code[s] & 1u);
        if (!(a.x == b.x && a.y == b.y)) ++bad;
    }
    if (bad) atomicAdd(count, bad);
}
// value of key k of the full vector x (0 for a key without members)
__device__ __forceinline__ cplx key_value(const cplx* x, const uint32_t* code, const uint32_t* src, size_t k) {
    const uint32_t s = src[k];
    return s == 0xffffffffu ? mk(0.0, 0.0) : signed_(x[s], code[s] & 1u);
}
__global__ void __launch_bounds__(RT) k_aa_gather(cplx* xr, const cplx* x, const uint32_t* code, const uint32_t* src,
                                                  size_t nr) {
    for (size_t k = blockIdx.x * (size_t)RT + threadIdx.x; k < nr; k += (size_t)gridDim.x * RT)
        xr[k] = key_value(x, code, src, k);
}
__global__ void __launch_bounds__(RT) k_aa_expand(cplx* x, const cplx* xr, const uint32_t* code, size_t n) {
    for (size_t j = blockIdx.x * (size_t)RT + threadIdx.x; j < n; j += (size_t)gridDim.x * RT) {
        const uint32_t c = code[j];
        st16(x + j, signed_(ld16(xr + key_of(c)), c & 1u));
    }
}
// fx = y - x ; g = x + beta fx ; block maxima of |fx|², NaN kept (y full, x one value per key)
__global__ void __launch_bounds__(RT) k_aa_residual(const cplx* y, const cplx* xr, const uint32_t* code,
                                                    const uint32_t* src, cplx* fx, cplx* g, double beta, double* pmax,
                                                    size_t nr) {
    __shared__ double red[RT / 32];
    double mx = 0.0;
    for (size_t k = blockIdx.x * (size_t)RT + threadIdx.x; k < nr; k += (size_t)gridDim.x * RT) {
        const cplx x = xr[k], f = key_value(y, code, src, k) - x;
        fx[k] = f;
        g[k] = x + f * beta;
        mx = max_mag(mx, f.x * f.x + f.y * f.y);
    }
    for (int o = 16; o > 0; o >>= 1) mx = max_mag(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
    __syncthreads();
    if (threadIdx.x) return;
    for (int w = 1; w < RT / 32; ++w) mx = max_mag(mx, red[w]);
    pmax[blockIdx.x] = mx;
}

// What bounds the step: at full length the FP64 pipe (about 200 FP64 instructions per element at
// m = 8: 1.0 ms at 1.87 M elements); at one value per key the launches.  So a pass does all the work
// that its vectors allow: the Givens rotations of a column deletion, Δg and Δf and the first
// projection run in one pass, every Gram-Schmidt pass also takes the partial of <Q_i, f> (no separate
// pass of dot products), and γ and the next deletion's rotations come from one single-block kernel.
// A step beside the map at m = 8 on GB300, on full vectors with separate passes -> now: Hubbard 8x8,
// nK3 = (8, 12): 1.03 -> 0.21 ms; Hubbard 8x8, nK3 = (20, 40), 49 M elements: 22 -> 1.8 ms; SIAM,
// nK3 = (16, 16), 0.1 M elements: 0.26 -> 0.16 ms.

// Column rotations (nrot > 0: the nrot = m - 1 rotations of a deletion, applied to Q in order), then
// Δg = g - gold ; Δf = fx - fxold (in place in fxold) ; partial of <Q_0, Δf>, or of |Δf|² when Q has no
// column left (k = 0).
__global__ void __launch_bounds__(RT) k_aa_diff(cplx* dg, const cplx* g, const cplx* gold, cplx* df, const cplx* fx,
                                                AAVecsW Q, int k, int nrot, const cplx* rot, const double* wgt,
                                                cplx* part_out, size_t n) {
    __shared__ cplx sh[RT / 32];
    __shared__ cplx rs[2 * AA_MAX];
    for (int i = threadIdx.x; i < 2 * nrot; i += RT) rs[i] = rot[i];
    __syncthreads();
    cplx s = mk(0.0, 0.0);
    for (size_t t = blockIdx.x * (size_t)RT + threadIdx.x; t < n; t += (size_t)gridDim.x * RT) {
        cplx q0 = mk(0.0, 0.0);
        if (nrot > 0) {
            cplx a = Q.v[0][t];
            for (int i = 1; i <= nrot; ++i) {
                const double c = rs[2 * (i - 1)].x;
                const cplx sn = rs[2 * (i - 1) + 1];
                const cplx b = Q.v[i][t];
                // Q_{i-1} = c a + conj(s) b ; a = -s a + c b
                const cplx r = mk(fma(a.x, c, fma(sn.x, b.x, sn.y * b.y)), fma(a.y, c, fma(sn.x, b.y, -sn.y * b.x)));
                Q.v[i - 1][t] = r;
                if (i == 1) q0 = r;
                // (the last column of a deletion is overwritten by the new one: not formed)
                if (i < nrot) a = mk(fma(b.x, c, fma(-sn.x, a.x, sn.y * a.y)), fma(b.y, c, fma(-sn.x, a.y, -sn.y * a.x)));
            }
        } else if (k > 0) {
            q0 = Q.v[0][t];
        }
        dg[t] = g[t] - gold[t];
        const cplx v = fx[t] - df[t];
        df[t] = v;
        const cplx wv = wgt ? v * wgt[t] : v;
        if (k > 0) s = cfma_conj(q0, wv, s);
        else s.x = fma(v.x, wv.x, fma(v.y, wv.y, s.x));
    }
    block_store_partial(s, sh, part_out);
}

// One modified Gram-Schmidt step: r = Σ part_in (= <Qa, Δf>), R entry = r, Δf -= r Qa; then the
// partials of the next projection <Qb, Δf> (or |Δf|² when Qb is null) and of <Qa, fx>.
__global__ void __launch_bounds__(RT) k_aa_mgs(cplx* df, const cplx* Qa, const cplx* part_in, int np, cplx* Rentry,
                                               const cplx* Qb, const cplx* fx, const double* wgt, cplx* part_out,
                                               cplx* pdot, size_t n) {
    __shared__ cplx sh[3][RT / 32];
    // (an element's loads are issued before the sum it waits for)
    size_t i = blockIdx.x * (size_t)RT + threadIdx.x;
    const size_t step = (size_t)gridDim.x * RT;
    cplx a, v, wf, b;
    double w = 1.0;
    auto load = [&]() {
        a = ld16(Qa + i); v = ld16(df + i); wf = ld16(fx + i);
        if (Qb) b = ld16(Qb + i);
        if (wgt) w = wgt[i];
    };
    if (i < n) load();
    const cplx r = block_reduce_parts(part_in, np, sh[0]);
    if (blockIdx.x == 0 && threadIdx.x == 0) *Rentry = r;
    cplx s = mk(0.0, 0.0), q = mk(0.0, 0.0);
    while (i < n) {
        v = cfnma(r, a, v);
        st16(df + i, v);
        cplx wv = v;
        if (wgt) { wv = wv * w; wf = wf * w; }
        q = cfma_conj(a, wf, q);
        if (Qb) s = cfma_conj(b, wv, s);
        else s.x = fma(v.x, wv.x, fma(v.y, wv.y, s.x));
        i += step;
        if (i < n) load();
    }
    block_store_partial(s, sh[1], part_out);
    block_store_partial(q, sh[2], pdot);
}

// ‖Δf‖ = sqrt(Σ part_in), R(k,k) = ‖Δf‖, Q_k = Δf / ‖Δf‖, partial of <Q_k, fx>.
__global__ void __launch_bounds__(RT) k_aa_qnew(cplx* Qk, const cplx* df, const cplx* part_in, int np, cplx* Rkk,
                                                const cplx* fx, const double* wgt, cplx* pdot, size_t n) {
    __shared__ cplx sh[2][RT / 32];
    size_t i = blockIdx.x * (size_t)RT + threadIdx.x;
    const size_t step = (size_t)gridDim.x * RT;
    cplx v, wf;
    double w = 1.0;
    auto load = [&]() {
        v = ld16(df + i); wf = ld16(fx + i);
        if (wgt) w = wgt[i];
    };
    if (i < n) load();
    const double nr = sqrt(fmax(0.0, block_reduce_parts(part_in, np, sh[0]).x));
    if (blockIdx.x == 0 && threadIdx.x == 0) *Rkk = mk(nr, 0.0);
    const double inv = 1.0 / nr;  // one division per block, not two per element
    cplx q = mk(0.0, 0.0);
    while (i < n) {
        const cplx u = mk(v.x * inv, v.y * inv);
        st16(Qk + i, u);
        if (wgt) wf = wf * w;
        q = cfma_conj(u, wf, q);
        i += step;
        if (i < n) load();
    }
    block_store_partial(q, sh[1], pdot);
}

__device__ __forceinline__ double cabs_(cplx a) { return hypot(a.x, a.y); }
// Deletion of the first column of the m x m QR factor by Givens rotations (NLsolve qrdelete!):
// rotation i = 1..m-1 acts on rows (i-1, i) of R; the parameters go to rot[2(i-1)] = (c, -) and
// rot[2(i-1)+1] = s; then the columns shift left by one.  One warp, a column of R per lane: the rotations
// are a serial chain, the columns are not (one thread took 66 us at m = 8).  Rs is the copy of R in shared
// memory that the chain works on.
__device__ __forceinline__ void givens_delete(cplx* Rs, cplx* R, int m, cplx* rot) {
    const int lane = threadIdx.x & 31;
    auto Rr = [&](int i, int j) -> cplx& { return Rs[i + (size_t)m * j]; };
    for (int i = 1; i < m; ++i) {
        const cplx f = Rr(i - 1, i), g = Rr(i, i);
        const double af = cabs_(f), ag = cabs_(g);
        double c;
        cplx sn;
        if (ag == 0.0) { c = 1.0; sn = mk(0.0, 0.0); }
        else if (af == 0.0) { c = 0.0; sn = mk(g.x / ag, -g.y / ag); }
        else {
            const double rr = hypot(af, ag);
            c = af / rr;
            const cplx fa = mk(f.x / af, f.y / af);
            sn = fa * conjg(g);
            sn = mk(sn.x / rr, sn.y / rr);
        }
        __syncwarp();
        for (int j = lane; j < m; j += 32) {
            const cplx a = Rr(i - 1, j), b = Rr(i, j);
            Rr(i - 1, j) = a * c + sn * b;
            Rr(i, j) = (-conjg(sn)) * a + b * c;
        }
        if (lane == 0) {
            rot[2 * (i - 1)] = mk(c, 0.0);
            rot[2 * (i - 1) + 1] = sn;
        }
        __syncwarp();
    }
    for (int e = lane; e < m * m; e += 32) {
        const int i = e % m, j = e / m;
        R[e] = i < m - 1 && j < m - 1 ? Rr(i, j + 1) : Rr(i, j);
    }
}
__global__ void k_aa_givens(cplx* R, int m, cplx* rot) {
    extern __shared__ __align__(16) unsigned char aa_sm[];
    cplx* Rs = reinterpret_cast<cplx*>(aa_sm);
    for (int e = threadIdx.x; e < m * m; e += 32) Rs[e] = R[e];
    __syncwarp();
    givens_delete(Rs, R, m, rot);
}

// γ = R⁻¹ (Σ_blocks part): one block; a warp per column of partials, then warp 0 back-substitutes
// (a row of R per lane).  R is column-major m x m.  del: the rotations of the next step's column
// deletion in the same launch, on warp 1 and a second copy of R beside the rest (R is not read by the
// update in between).  Serial chains of FP64 divisions bound it: R lies in shared memory and the parts of
// the divisions by R_ii that do not wait for γ are done ahead for all rows at once.
__global__ void __launch_bounds__(RT) k_aa_gamma(const cplx* part, int stride, int np, cplx* R, int m, int meff,
                                                 cplx* gam, int del, cplx* rot) {
    extern __shared__ __align__(16) unsigned char aa_sm[];
    __shared__ cplx g[AA_MAX];
    __shared__ cplx dv[AA_MAX];  // Smith's ratio and denominator of R_ii
    cplx* Rs = reinterpret_cast<cplx*>(aa_sm);
    cplx* Rg = Rs + (size_t)m * m;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int e = threadIdx.x; e < m * m; e += RT) {
        const cplx v = ld16(R + e);
        Rs[e] = v;
        if (del) Rg[e] = v;
    }
    __syncthreads();
    if (warp == 1) {
        if (del) givens_delete(Rg, R, m, rot);
        return;
    }
    constexpr int NW = RT / 32 - 1;  // the other warps
    for (int i = warp ? warp - 1 : 0; i < meff; i += NW) {
        cplx s = mk(0.0, 0.0);
        for (int b = lane; b < np; b += 32) s += ld16(part + (size_t)i * stride + b);
        s = warp_sum(s);
        if (lane == 0) g[i] = s;
    }
    if (warp == 0)
        for (int i = lane; i < meff; i += 32) {
            const cplx b = Rs[i + (size_t)m * i];
            const bool big = fabs(b.x) >= fabs(b.y);
            const double r = big ? b.y / b.x : b.x / b.y;
            dv[i] = mk(r, big ? b.x + b.y * r : b.x * r + b.y);
        }
    asm volatile("bar.sync 1, %0;" ::"n"(32 * NW) : "memory");
    if (warp != 0) return;
    for (int i = meff - 1; i >= 0; --i) {
        const cplx a = g[i], b = Rs[i + (size_t)m * i];
        const double r = dv[i].x, den = dv[i].y;
        const cplx x = fabs(b.x) >= fabs(b.y) ? mk((a.x + a.y * r) / den, (a.y - a.x * r) / den)
                                              : mk((a.x * r + a.y) / den, (a.y * r - a.x) / den);
        __syncwarp();
        if (lane == 0) gam[i] = x;
        for (int j = lane; j < i; j += 32) g[j] = cfnma(Rs[j + (size_t)m * i], x, g[j]);
        __syncwarp();
    }
}

// x = g - Σ_i γ_i Δg_i (i in order) ; fxold = fx ; gold = g.
__global__ void __launch_bounds__(RT) k_aa_update(cplx* x, const cplx* g, AAVecs dG, const cplx* gam, int meff,
                                                  const cplx* fx, cplx* fxold, cplx* gold, size_t n) {
    __shared__ cplx gs[AA_MAX];
    for (int i = threadIdx.x; i < meff; i += RT) gs[i] = gam[i];
    __syncthreads();
    for (size_t i = blockIdx.x * (size_t)RT + threadIdx.x; i < n; i += (size_t)gridDim.x * RT) {
        const cplx gi = g[i];
        cplx v = gi;
        for (int j = 0; j < meff; ++j) v = cfnma(gs[j], dG.v[j][i], v);
        x[i] = v;
        fxold[i] = fx[i];
        gold[i] = gi;
    }
}

}  // namespace

#define AA_CHECK()                                   \
    do {                                             \
        cudaError_t e__ = cudaGetLastError();        \
        if (e__ != cudaSuccess) return e__;          \
    } while (0)

cudaError_t launch_aa_keys(cudaStream_t s, int nblk, const uint32_t* code, uint32_t* src, double* w, size_t n) {
    k_aa_keys<<<nblk, RT, 0, s>>>(code, src, w, n);
    AA_CHECK(); return cudaSuccess;
}
cudaError_t launch_aa_check(cudaStream_t s, int nblk, const cplx* x, const uint32_t* code, const uint32_t* src,
                            unsigned int* count, size_t n) {
    k_aa_check<<<nblk, RT, 0, s>>>(x, code, src, count, n);
    AA_CHECK(); return cudaSuccess;
}
cudaError_t launch_aa_gather(cudaStream_t s, int nblk, cplx* xr, const cplx* x, const uint32_t* code,
                             const uint32_t* src, size_t nr) {
    k_aa_gather<<<nblk, RT, 0, s>>>(xr, x, code, src, nr);
    AA_CHECK(); return cudaSuccess;
}
cudaError_t launch_aa_expand(cudaStream_t s, cplx* x, const cplx* xr, const uint32_t* code, size_t n) {
    const size_t nb = (n + RT - 1) / RT;
    k_aa_expand<<<(unsigned)(nb < 4864 ? nb : 4864), RT, 0, s>>>(x, xr, code, n);  // 32 CTAs per SM of 152
    AA_CHECK(); return cudaSuccess;
}
cudaError_t launch_aa_residual(cudaStream_t s, int nblk, const cplx* y, const cplx* xr, const uint32_t* code,
                               const uint32_t* src, cplx* fx, cplx* g, double beta, double* pmax, size_t nr) {
    k_aa_residual<<<nblk, RT, 0, s>>>(y, xr, code, src, fx, g, beta, pmax, nr);
    AA_CHECK(); return cudaSuccess;
}
cudaError_t launch_aa_diff(cudaStream_t s, int nblk, cplx* dg, const cplx* g, const cplx* gold, cplx* df,
                           const cplx* fx, const AAVecsW& Q, int k, int nrot, const cplx* rot, const double* wgt,
                           cplx* part_out, size_t n) {
    if (k < 0 || k >= AA_MAX || nrot < 0 || nrot >= AA_MAX) return cudaErrorInvalidValue;
    k_aa_diff<<<nblk, RT, 0, s>>>(dg, g, gold, df, fx, Q, k, nrot, rot, wgt, part_out, n);
    AA_CHECK(); return cudaSuccess;
}
cudaError_t launch_aa_mgs(cudaStream_t s, int nblk, cplx* df, const cplx* Qa, const cplx* part_in, cplx* Rentry,
                          const cplx* Qb, const cplx* fx, const double* wgt, cplx* part_out, cplx* pdot, size_t n) {
    k_aa_mgs<<<nblk, RT, 0, s>>>(df, Qa, part_in, nblk, Rentry, Qb, fx, wgt, part_out, pdot, n);
    AA_CHECK(); return cudaSuccess;
}
cudaError_t launch_aa_qnew(cudaStream_t s, int nblk, cplx* Qk, const cplx* df, const cplx* part_in, cplx* Rkk,
                           const cplx* fx, const double* wgt, cplx* pdot, size_t n) {
    k_aa_qnew<<<nblk, RT, 0, s>>>(Qk, df, part_in, nblk, Rkk, fx, wgt, pdot, n);
    AA_CHECK(); return cudaSuccess;
}
cudaError_t launch_aa_update(cudaStream_t s, int nblk, cplx* x, const cplx* g, const AAVecs& dG, const cplx* gam,
                             int meff, const cplx* fx, cplx* fxold, cplx* gold, size_t n) {
    if (meff > AA_MAX) return cudaErrorInvalidValue;
    k_aa_update<<<nblk, RT, 0, s>>>(x, g, dG, gam, meff, fx, fxold, gold, n);
    AA_CHECK(); return cudaSuccess;
}
cudaError_t launch_aa_givens(cudaStream_t s, cplx* R, int m, cplx* rot) {
    if (m < 2 || m > AA_MAX) return cudaErrorInvalidValue;
    const size_t smem = (size_t)m * m * sizeof(cplx);
    static SmemRecord raised;
    const cudaError_t e = raise_smem_limit(k_aa_givens, raised, smem);
    if (e != cudaSuccess) return e;
    k_aa_givens<<<1, 32, smem, s>>>(R, m, rot);
    AA_CHECK(); return cudaSuccess;
}
cudaError_t launch_aa_gamma(cudaStream_t s, const cplx* part, int stride, int np, cplx* R, int m, int meff, cplx* gam,
                            int del, cplx* rot) {
    if (meff < 1 || meff > m || m > AA_MAX || (del && (m < 2 || meff != m))) return cudaErrorInvalidValue;
    const size_t smem = 2 * (size_t)m * m * sizeof(cplx);
    static SmemRecord raised;
    const cudaError_t e = raise_smem_limit(k_aa_gamma, raised, smem);
    if (e != cudaSuccess) return e;
    k_aa_gamma<<<1, RT, smem, s>>>(part, stride, np, R, m, meff, gam, del, rot);
    AA_CHECK(); return cudaSuccess;
}

}  // namespace fdga
