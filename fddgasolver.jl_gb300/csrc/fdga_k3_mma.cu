// fdga_k3_mma.cu -- the K3 Bethe-Salpeter contractions of the FP64 map for small blocks (Nν3 ≤ 32) on
// warp-level tensor-core products, by exact digit slicing (the Ozaki scheme): FP64 results from FP16
// products.
//
// Per (channel, representative (P, Ω) block) the BSE is one complex product C = A·M of Nν3 x Nν3
// matrices (src/BSEa/BSEa_K3.jl:1-128), M formed elementwise in FP64 from the caches, Π, Π0 and FL.  On
// the CUDA cores it is bound by the FP64 pipe (1/64 of the FP32 rate); the tcgen05 kernel of
// fdga_k3_oz.cu has 128-row accumulators, of which a 24 x 24 block fills 24 rows, and a fixed cost per
// CTA (tensor-memory allocation, the pre-pass of A digits, mbarrier round trips) that a block of three
// K steps does not carry.  mma.sync.m16n8k16 fits these blocks without waste: one warp owns one 8 x 8
// complex output tile, whose real and imaginary parts are the two 8-row halves of the MMA's 16 rows.
//
// Exact slicing.  Row ν of A and column ν' of M each have a power-of-two bound 2^(F-1022) from the
// largest exponent field of their entries (integer maxima, no FP64 work).  An entry is rounded to the
// fixed-point integer Y = v 2^(62+1022-F), |Y| < 2^62 (exact for every entry within 2^9 of its row's or
// column's largest), taken from the FP64 significand by a shift, and Y is cut into S = 8 balanced
// base-256 digits: adding 0x80 to every byte makes byte s, less 128, the digit d_s in [-128, 127].  A
// digit is an FP16 number exactly (0x6400 | byte is 1024 + byte; one packed subtraction of 1152 leaves
// the digit).  The products of digit pairs (s, t) with s + t = g ≤ 7 share one FP32 accumulator:
// products are at most 2^14 and at most 8·64 of them meet in one accumulator, so every partial sum is an
// integer of at most 2^23 and exact.  The pairs with s + t ≥ 8 are dropped; with the rounding of Y they
// leave below 2^-58.9 of (row bound)·(column bound) per product term, and the 36 digit products replace the
// FP64 operations (three real products per complex one, 64 issue slots each).  The epilogue joins the
// eight integers exactly in two 64-bit integers and one FP64 addition, then applies T and γL as the
// CUDA-core kernel does.
//
// To what the accuracy is relative.  Where a row and a column have large entries at a common ω, the bounds are
// about Σ_ω |A||M| and the digits beat an FP64 sum's rounding.  Operands graded against each other (A falls along
// ω as M rises) have bounds far above it: entries 2^k below theirs keep 62 - k bits.  So one more product, of the
// top digits in magnitude, sees whether any ω has a nonzero top digit on both sides, that is Σ |A||M| ≥ 2^-14 of
// the bounds and an error below 2 Nν3 2^-45 of it; an output without one is summed again in FP64, one ω per lane
// (A falling by 2^39 as M rises, Nν3 = 24: error 8e-9 of the largest output -> an FP64 sum's).  That is so in the
// adjoint and below Nν3 = 32, where FP64 sums ran before.  Of the lattice workloads' maps 0.2 % of the outputs are
// summed again (Hubbard 8x8, nK3 = (8, 12): K3 38 us with and without; the residual call 584 -> 587 us), of the
// adjoint's 3.6 %, far from the diagonal of one product (700 -> 719 us; one output at a time, each part by itself,
// 776).  At Nν3 = 32 the map's digits stand by themselves, as did the form before with bounds of whole blocks: a
// SIAM has outputs far from the diagonal that would be summed again (K3 18 -> 43 us one at a time).  A row of A or a
// column of M that holds an infinity or NaN, or products near the end of the normal range, are summed in FP64
// everywhere.
//
// What bounds it: forming M (8 to 14 FP64 operations per entry) and the latency of one pass load ->
// digits -> MMA -> store; a CTA of NC·NC warps (NC = ⌈Nν3/8⌉) does one block, each warp staging one 8 x 8
// chunk of M and of A and then one output tile, so that no warp idles in either phase.
// On GB300, CUDA cores -> this kernel, L_K3 / K3 in us: Hubbard 8x8, nK3 = (8, 12) (675 blocks of
// 24 x 24) 78 / 98 -> 23 / 37; Hubbard 6x6, nK3 = (7, 11) 50 / 59 -> 19 / 25; 5x5 without groups,
// nK3 = (5, 7) (675 blocks of 14 x 14) 28 / 34 -> 13 / 16; SIAM, nK3 = (6, 6) 18 / 20 -> 9 / 11.  At
// Nν3 = 24 the tcgen05 kernel takes 79 / 97.
#include <algorithm>

#include "fdga_digits.cuh"
#include "fdga_kernels.h"

namespace fdga {

namespace {

constexpr int S = 8;  // digits per operand
// bytes between rows of a digit plane: an odd multiple of 16, so that the eight 16-byte rows of an 8 x 8
// matrix (ldmatrix) and the 4-byte stores of 8 columns x 4 ω pairs fall on distinct banks
template <int NC> constexpr int PITCH = NC == 1 ? 16 : (NC == 4 ? 80 : 48);
template <int NC> constexpr int PLANE = 8 * NC * PITCH<NC>;
// planes [A or M][digit][re, im]
template <int NC> constexpr int SMEM = 2 * S * 2 * PLANE<NC>;

// the digits of two neighbouring ω of one row, both parts, stored to the planes at byte offset o
template <int NC>
__device__ __forceinline__ void store_digits(uint8_t* planes, int o, cplx v0, cplx v1, int F) {
    const unsigned long long r0 = (unsigned long long)fixed_digits<S>(v0.x, F) + DIGIT_BIAS, i0 = (unsigned long long)fixed_digits<S>(v0.y, F) + DIGIT_BIAS;
    const unsigned long long r1 = (unsigned long long)fixed_digits<S>(v1.x, F) + DIGIT_BIAS, i1 = (unsigned long long)fixed_digits<S>(v1.y, F) + DIGIT_BIAS;
#pragma unroll
    for (int s = 0; s < S; ++s) {
        uint8_t* p = planes + (2 * s) * PLANE<NC> + o;
        *reinterpret_cast<uint32_t*>(p) = digit_pair(r0, r1, S - 1 - s);
        *reinterpret_cast<uint32_t*>(p + PLANE<NC>) = digit_pair(i0, i1, S - 1 - s);
    }
}

// Warp sums of eight values: that of x[i] in x[0] of the lanes 4i .. 4i + 3 (9 additions for the 40 of eight sums by
// themselves: FP64 bounds an output summed again).
__device__ __forceinline__ void sum8(double (&x)[8], int lane) {
#pragma unroll
    for (int h = 4; h >= 1; h >>= 1) {  // lanes 4h apart exchange halves
        const bool up = (lane & (4 * h)) != 0;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const double keep = up ? x[i + h] : x[i], send = up ? x[i] : x[i + h];
            x[i] = keep + __shfl_xor_sync(0xffffffffu, send, 4 * h);
        }
    }
    x[0] += __shfl_xor_sync(0xffffffffu, x[0], 2);
    x[0] += __shfl_xor_sync(0xffffffffu, x[0], 1);
}

// One N x N complex product per CTA of NC·NC warps: av = two neighbouring k of row cl of the left operand,
// mv = the same k of column cl of the right one; out(row, column, value) is called by the lane that holds an
// element, term(row, column, k) is the product of the two operands' elements at k in FP64, for outputs of operands
// graded against each other (where `graded`) or not finite.  fmax_ is zero on entry and a __syncthreads lies behind
// that.
template <int NC, class TERM, class OUT>
__device__ __forceinline__ void digit_product(uint8_t* sm, int (*fmax_)[8 * NC], int N, int cl, int w0, bool graded,
                                              const cplx (&av)[2], const cplx (&mv)[2], TERM&& term, OUT&& out) {
    uint8_t* Mp = sm;
    uint8_t* Ap = sm + 2 * S * PLANE<NC>;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int em = max(cexpo(mv[0]), cexpo(mv[1])), ea = max(cexpo(av[0]), cexpo(av[1]));
#pragma unroll
    for (int o = 8; o <= 16; o <<= 1) {
        em = max(em, __shfl_xor_sync(0xffffffffu, em, o));
        ea = max(ea, __shfl_xor_sync(0xffffffffu, ea, o));
    }
    if (lane < 8) {
        atomicMax(&fmax_[0][cl], ea);
        atomicMax(&fmax_[1][cl], em);
    }
    __syncthreads();
    const int so = cl * PITCH<NC> + 2 * w0;
    store_digits<NC>(Ap, so, av[0], av[1], fmax_[0][cl]);
    store_digits<NC>(Mp, so, mv[0], mv[1], fmax_[1][cl]);
    __syncthreads();
    // warp = (ν' chunk j, ν chunk nt): D rows 0-7 = Re, rows 8-15 = Im of the outputs ν' = 8j.., columns ν
    const int j = warp % NC, nt = warp / NC;
    float acc[S][4];
#pragma unroll
    for (int g = 0; g < S; ++g)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[g][i] = 0.0f;
    float mag[4] = {0.0f, 0.0f, 0.0f, 0.0f};  // Σ of the top digits' products in magnitude
    auto mma = [](float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
        asm volatile(
            "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    };
    // lane l addresses row l % 8 of matrix l / 8: M re, M im, A re, A im of one digit
    const uint32_t laddr = (uint32_t)__cvta_generic_to_shared(
        (lane < 16 ? Mp + (8 * j + (lane & 7)) * PITCH<NC> : Ap + (8 * nt + (lane & 7)) * PITCH<NC>) +
        ((lane >> 3) & 1) * PLANE<NC>);
#pragma unroll 1
    for (int c = 0; c < NC; ++c) {
        uint32_t mr[S], mi[S], ar[S], ai[S];
#pragma unroll
        for (int s = 0; s < S; ++s)
            asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                         : "=r"(mr[s]), "=r"(mi[s]), "=r"(ar[s]), "=r"(ai[s])
                         : "r"(laddr + (uint32_t)(2 * s * PLANE<NC> + 16 * c))
                         : "memory");
        // k = (ω chunk; Re A, Im A): rows Re: [Re M, -Im M], rows Im: [Im M, Re M]
#pragma unroll
        for (int s = 0; s < S; ++s)
#pragma unroll
            for (int t = 0; s + t < S; ++t) mma(acc[s + t], mr[s], mi[s], mi[s] ^ 0x80008000u, mr[s], ar[t], ai[t]);
        const uint32_t pm = 0x7fff7fffu;
        mma(mag, mr[0] & pm, mi[0] & pm, mi[0] & pm, mr[0] & pm, ar[0] & pm, ai[0] & pm);
    }
    const int col = 8 * j + (lane >> 2);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int nu = 8 * nt + 2 * (lane & 3) + e;
        const bool in = col < N && nu < N;
        cplx v = mk(0.0, 0.0);
        bool weak = false;
        if (in) {
            const int FA = fmax_[0][nu], FM = fmax_[1][col], E = FA + FM;
            double p[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const float a[8] = {acc[0][2 * q + e], acc[1][2 * q + e], acc[2][2 * q + e], acc[3][2 * q + e],
                                    acc[4][2 * q + e], acc[5][2 * q + e], acc[6][2 * q + e], acc[7][2 * q + e]};
                p[q] = join_digits<S>(a, E);
            }
            v = mk(p[0], p[1]);
            // (a row or column of zeros has F = 0: its sums are 0)
            // (E below 1100: outputs near the end of the normal range, where the join flushes)
            weak = FA != 0 && FM != 0 &&
                   (FA == 0x7ff || FM == 0x7ff || E < 1100 || (graded && mag[e] == 0.0f && mag[2 + e] == 0.0f));
        }
        for (unsigned todo = __ballot_sync(0xffffffffu, weak); todo;) {  // four outputs at a time, one k per lane
            int src[4];
            double x[8];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                src[i] = todo ? __ffs(todo) - 1 : src[0];
                todo &= todo - 1;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                cplx t = mk(0.0, 0.0);
                if (lane < N) t = term(8 * nt + 2 * (src[i] & 3) + e, 8 * j + (src[i] >> 2), lane);
                x[2 * i] = t.x;
                x[2 * i + 1] = t.y;
            }
            sum8(x, lane);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const cplx t = mk(__shfl_sync(0xffffffffu, x[0], 8 * i), __shfl_sync(0xffffffffu, x[0], 8 * i + 4));
                if (lane == src[i]) v = t;
            }
        }
        if (in) out(nu, col, v);
    }
}

// MODE 0: L_K3, 1: K3 (and the dA·M part of the tangent), 3: the A·dM part of the tangent
template <int MODE, int NC>
__global__ void __launch_bounds__(32 * NC * NC) k_bse_K3_mma(K3Args3 args, Dims d) {
    extern __shared__ __align__(16) uint8_t sm[];
    __shared__ cplx qf[8 * NC][2];  // the ω factors of M with their signs, as in k_bse_K3_oz
    __shared__ int fmax_[2][8 * NC];  // largest exponent fields: [0] rows ν of A, [1] columns ν' of M
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int N = d.N3n;
    const int slot = blockIdx.x / args.nblocks, bi = blockIdx.x % args.nblocks;
    const int blk = args.blocks ? args.blocks[bi] : bi;
    const K3Args& a = args.a[slot];
    const int CH = args.ch[slot];
    const int m = blk % d.N3O - (d.n3O - 1), P = blk / d.N3O;
    const size_t base = (size_t)blk * N * N;
    const double s1 = (CH == CH_A) ? 1.0 : -1.0, s2 = (CH == CH_T) ? -1.0 : 1.0;
    const bool full = MODE == 3 || (MODE == 1 && (a.flags & K3F_1LOOP) == 0);
    auto gl_of = [&](const cplx* FLc, const cplx* FLt, const cplx* FLa, size_t i) -> cplx {
        if (CH == CH_T) {
            const cplx t = ldg(FLt + i), u = ldg(FLa + i);
            return cplx{fma(t.x, 2.0, -u.x), fma(t.y, 2.0, -u.y)};
        }
        return ldg(FLc + i);
    };
    if (tid < 8 * NC) {
        fmax_[0][tid] = fmax_[1][tid] = 0;
        cplx q0 = mk(0.0, 0.0), q1 = mk(0.0, 0.0);
        if (tid < N) {
            const size_t ip = ixPi(d, P, m, tid - d.n3n);
            q0 = (MODE != 3 && a.Pi0) ? ldg(a.Pi0 + ip) : mk(0.0, 0.0);
            if (MODE >= 1) {
                const cplx pi = ldg(a.Pi + ip);
                q1 = pi * s1;
                q0 = (MODE == 3) ? ldg(a.tPi + ip) * s1 : (pi - q0) * s1;
            }
        }
        qf[tid][0] = q0;
        qf[tid][1] = q1;
    }
    // entry (ω, ν') of M: q[0] x0 + q[1] x1
    auto load_M = [&](int w, int cl, cplx& x0, cplx& x1) {
        x0 = ldg(a.B0 + base + (size_t)w * N + cl);
        if (!full) return;
        // s2 Π = ±s1 Π: the γL terms join the Γ terms before the products
        const size_t ig = (CH == CH_P) ? base + (size_t)w * N + cl : base + (size_t)cl * N + w;
        const int ot = cross(CH, m, w - d.n3n);
        const bool hl = fin(ot, d.n3n);
        const size_t il = base + (size_t)(ot + d.n3n) * N + cl;
        cplx g = ldg(a.G + ig);
        if (hl) {
            const cplx l = gl_of(a.FLc, a.FLt, a.FLa, il);
            g = (s1 == s2) ? g + l : g - l;
        }
        if (MODE == 3) {  // dM = s1 dΠ (F0 + Γ ± γL) + s1 Π (dΓ ± dγL)
            x0 += g;
            g = ldg(a.tG + ig);
            if (hl) {
                const cplx l = gl_of(a.tFLc, a.tFLt, a.tFLa, il);
                g = (s1 == s2) ? g + l : g - l;
            }
        }
        x1 = g;
    };
    auto form_M = [&](int w, cplx x0, cplx x1) { return full ? cfma(qf[w][0], x0, qf[w][1] * x1) : qf[w][0] * x0; };
    // staging: warp = (column chunk, ω chunk); a lane holds one column (row of A) and two neighbouring ω
    const int cl = 8 * (warp % NC) + (lane & 7), w0 = 8 * (warp / NC) + 2 * (lane >> 3);
    cplx av[2], x0[2], x1[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int w = w0 + i;
        av[i] = x0[i] = x1[i] = mk(0.0, 0.0);
        if (cl >= N || w >= N) continue;
        av[i] = ldg(a.A + base + (size_t)cl * N + w);
        load_M(w, cl, x0[i], x1[i]);
    }
    __syncthreads();
    cplx mv[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) mv[i] = cl < N && w0 + i < N ? form_M(w0 + i, x0[i], x1[i]) : mk(0.0, 0.0);
    auto term = [&](int nu, int col, int w) {
        cplx y0, y1 = mk(0.0, 0.0);
        load_M(w, col, y0, y1);
        return ldg(a.A + base + (size_t)nu * N + w) * form_M(w, y0, y1);
    };
    digit_product<NC>(sm, fmax_, N, cl, w0, N < 32, av, mv, term, [&](int nu, int col, cplx cv) {
        const size_t io = base + (size_t)nu * N + col;
        cplx o;
        if (MODE == 0) {
            o = cv * (d.T * ((CH == CH_A) ? 1.0 : -1.0));
        } else if (a.flags & K3F_NOEPI) {
            o = cv * d.T;
        } else {
            const cplx g = (MODE == 3) ? gl_of(a.tFLc, a.tFLt, a.tFLa, io) : gl_of(a.FLc, a.FLt, a.FLa, io);
            o = cplx{fma(cv.x, d.T, g.x), fma(cv.y, d.T, g.y)};
        }
        if (a.flags & K3F_ACC) o = a.out[io] + o;
        a.out[io] = o;
    });
}

// The products of the adjoint contraction: OPA = 0: C = α A Bᴴ, OPA = 1: C = α Aᴴ B (C += when
// accumulating).  Adjoint GEMMs of Hubbard 8x8, nK3 = (8, 12) on GB300: 72 us each on the CUDA cores,
// 23 us here.
template <int OPA, int NC>
__global__ void __launch_bounds__(32 * NC * NC) k_adj_mma(GemmBatch g, Dims d) {
    extern __shared__ __align__(16) uint8_t sm[];
    __shared__ int fmax_[2][8 * NC];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int N = d.N3n, slot = blockIdx.z;
    const int blk = g.blocks ? g.blocks[blockIdx.x] : blockIdx.x;
    const size_t base = (size_t)blk * N * N;
    const cplx* A = (slot == 0 ? g.A[0] : slot == 1 ? g.A[1] : g.A[2]) + base;
    const cplx* B = (slot == 0 ? g.B[0] : slot == 1 ? g.B[1] : g.B[2]) + base;
    cplx* C = (slot == 0 ? g.C[0] : slot == 1 ? g.C[1] : g.C[2]) + base;
    const double alpha = slot == 0 ? g.alpha[0] : slot == 1 ? g.alpha[1] : g.alpha[2];
    if (tid < 8 * NC) fmax_[0][tid] = fmax_[1][tid] = 0;
    auto left = [&](int r, int w) { return OPA == 0 ? ldg(A + (size_t)r * N + w) : conjg(ldg(A + (size_t)w * N + r)); };
    auto right = [&](int c, int w) { return OPA == 0 ? conjg(ldg(B + (size_t)c * N + w)) : ldg(B + (size_t)w * N + c); };
    const int cl = 8 * (warp % NC) + (lane & 7), w0 = 8 * (warp / NC) + 2 * (lane >> 3);
    cplx av[2], mv[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int w = w0 + i;
        const bool in = cl < N && w < N;
        av[i] = in ? left(cl, w) : mk(0.0, 0.0);
        mv[i] = in ? right(cl, w) : mk(0.0, 0.0);
    }
    __syncthreads();
    digit_product<NC>(sm, fmax_, N, cl, w0, true, av, mv, [&](int r, int c, int w) { return left(r, w) * right(c, w); },
                      [&](int r, int c, cplx cv) {
                          cplx* o = C + (size_t)r * N + c;
                          const cplx v = cv * alpha;
                          *o = g.accumulate ? *o + v : v;
                      });
}

template <int MODE, int NC>
cudaError_t run_mma(cudaStream_t s, const K3Args3& a, int nslots, const Dims& d) {
    k_bse_K3_mma<MODE, NC><<<(unsigned)(nslots * a.nblocks), 32 * NC * NC, SMEM<NC>, s>>>(a, d);
    return cudaGetLastError();
}
template <int MODE>
cudaError_t run_mode(cudaStream_t s, const K3Args3& a, int nslots, const Dims& d) {
    switch ((d.N3n + 7) / 8) {
        case 1: return run_mma<MODE, 1>(s, a, nslots, d);
        case 2: return run_mma<MODE, 2>(s, a, nslots, d);
        case 3: return run_mma<MODE, 3>(s, a, nslots, d);
        default: return run_mma<MODE, 4>(s, a, nslots, d);
    }
}

}  // namespace

template <int OPA>
static cudaError_t run_adj(cudaStream_t s, const GemmBatch& g, const Dims& d) {
    const dim3 grid((unsigned)g.nblocks, 1, 3);
    switch ((d.N3n + 7) / 8) {
        case 1: k_adj_mma<OPA, 1><<<grid, 32, SMEM<1>, s>>>(g, d); break;
        case 2: k_adj_mma<OPA, 2><<<grid, 128, SMEM<2>, s>>>(g, d); break;
        case 3: k_adj_mma<OPA, 3><<<grid, 288, SMEM<3>, s>>>(g, d); break;
        default: k_adj_mma<OPA, 4><<<grid, 512, SMEM<4>, s>>>(g, d); break;
    }
    return cudaGetLastError();
}
cudaError_t launch_adj_mma(cudaStream_t s, int opa, const GemmBatch& g, const Dims& d) {
    return opa ? run_adj<1>(s, g, d) : run_adj<0>(s, g, d);
}

bool k3_mma_supported(const Dims& d) { return d.N3n <= 32; }

// raises the shared-memory limit of the four-chunk instantiations (82 KB); the others fit the default
cudaError_t prepare_bse_K3_mma(const Dims& d) {
    if (d.N3n <= 24) return cudaSuccess;
    static SmemRecord set0, set1, set3, seta, setb;
    cudaError_t e = raise_smem_limit(k_bse_K3_mma<0, 4>, set0, SMEM<4>, 0);
    if (e == cudaSuccess) e = raise_smem_limit(k_bse_K3_mma<1, 4>, set1, SMEM<4>, 0);
    if (e == cudaSuccess) e = raise_smem_limit(k_bse_K3_mma<3, 4>, set3, SMEM<4>, 0);
    if (e == cudaSuccess) e = raise_smem_limit(k_adj_mma<0, 4>, seta, SMEM<4>, 0);
    if (e == cudaSuccess) e = raise_smem_limit(k_adj_mma<1, 4>, setb, SMEM<4>, 0);
    return e;
}

// mode 0 (BSE_L_K3), 1 (BSE_K3), 2 (the tangent dK3 = T (dA·M + A·dM) + dγL, as two launches with their
// own scales: dA and A need not share a magnitude)
cudaError_t launch_bse_K3_mma(cudaStream_t s, int mode, const K3Args3& a, int nslots, const Dims& d) {
    if (!k3_mma_supported(d) || mode < 0 || mode > 2) return cudaErrorInvalidValue;
    if (mode == 0) return run_mode<0>(s, a, nslots, d);
    if (mode == 1) return run_mode<1>(s, a, nslots, d);
    K3Args3 a1 = a, a3 = a;
    for (int i = 0; i < nslots; ++i) {
        if (a.a[i].flags & K3F_1LOOP) return cudaErrorInvalidValue;  // no tangent of the one-loop form
        a1.a[i].A = a.a[i].tA;
        a1.a[i].flags |= K3F_NOEPI;
        a3.a[i].flags |= K3F_ACC;
    }
    const cudaError_t e = run_mode<1>(s, a1, nslots, d);
    return e != cudaSuccess ? e : run_mode<3>(s, a3, nslots, d);
}

}  // namespace fdga
