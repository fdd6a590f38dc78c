// fdga_k3_oz.cu -- the K3 Bethe-Salpeter contractions of the FP64 map on the tcgen05 tensor cores,
// by exact digit slicing (the Ozaki scheme): FP64 results from FP16 products.
//
// Per (channel, representative (P, Ω) block) the BSE is one complex product C = A·M of Nν3 x Nν3
// matrices (src/BSEa/BSEa_K3.jl:1-128; M formed elementwise in FP64 from the caches, Π, Π0 and FL).  It runs
// as the real GEMM D[ν][n] = Σ_k A_r[ν][k] B_r[k][n] in 2x2 real form (k = 2ω + q, n = 2ν' + p), split in
// column tiles of NT = 64 real columns.
//
// Exact slicing.  Row ν of A and column ν' of M each have a bound 2^(F-1022) from the largest exponent
// field of their entries.  An entry becomes a 62-bit fixed-point integer relative to its bound and is cut
// into S = 8 balanced base-256 digits, FP16 numbers exactly (fdga_digits.cuh).  The products of digit
// pairs (s, t) with s + t = g share one FP32 accumulator in tensor memory (g = 0..7, 8 x 64 columns: all of
// it).  The top digits are at most 64 and the others 128, so a diagonal of K products is at most g K 2^14: all
// are exact for K ≤ 128 (Nν3 ≤ 64), and the diagonals g ≤ 4 for K ≤ 256; the others pass 2^24 there only when
// nearly all digits of a row and a column have full size and equal signs, and then round by a unit of a
// diagonal g ≥ 5 (2^-52 of the bounds).  The pairs with s + t ≥ 8 are dropped; with the rounding of the entries
// they leave below 2^-58.9 of (row bound)·(column bound) per product term, which is less than an FP64 product's
// rounding for terms within 2^5 of the bounds.  (Seven digits, 54 bits, left up to 2^-51.2, more than the 2^-53.2
// of the 8 x 7-bit form before them, and took 302 / 442 us where eight take 331 / 496: 4x4, nK3 = (20, 40).)
// The epilogue joins the diagonals exactly in two 64-bit integers with one FP64 addition, then applies T and γL,
// as the FP64 kernel does.  A row of A or column of M with an infinity or NaN gives NaN there, as the FP64 sums do.
//
// Per launch and group of blocks: k_oz_adigits finds F of every row of every A block and writes its digit
// operands to a global buffer, once per block, in the shared-memory operand layout; then the contraction
// runs one CTA per (channel slot, block, column tile), two CTAs per SM: eight worker warps and a control
// warp.  A worker forms N/8 entries of the tile of M in FP64 in registers, all their loads independent, and
// the workers find the column bounds; then, K in chunks of 16 (8 ω, one entry per worker), they digitise
// chunk after chunk into one of the stages (three for L_K3 up to Nν3 = 80, else two) while the control thread
// keeps the A digits of the next chunks in flight (cp.async.bulk on an mbarrier) and issues the 36 MMAs of a
// chunk when both have arrived (kind::f16, FP32 accumulation, committed to the stage's mbarrier).  The
// accumulators take the whole tensor memory of an SM, so the CTA allocates it only once its M is formed and
// gives it back as soon as the accumulators are joined into shared memory: the MMAs of one CTA run while its
// neighbour on the SM forms M or writes its results.  The rows above N of the 128-row A operands are whatever
// lies behind them in their stage: they reach only rows of D that are not read.  Every wait on an mbarrier is
// bounded (a timeout sets *err and the CTA's abort flag; the control thread still waits, bounded, for its copies
// and MMAs in flight before the tensor memory is released).
//
// What bounds it: the MMAs, which cost about the same for 32 columns as for 64 (the 128-row A operand is
// read for each), then the FP64 pipe (8 to 12 operations per entry of M and 2 to 6 per output).  The form
// before had 32-column tiles, 36 BF16 MMAs of 7-bit digits, an FP32 bound pass over the operands of M, and M
// formed and digitised per chunk between two CTA barriers.  L_K3 / K3 stage in us on GB300, that form -> this:
// 4x4, nK3 = (20, 40) (Nν3 = 80, 702 blocks) 429 / 607 -> 331 / 496; 8x8, nK3 = (20, 40) 1030 / 1460 -> 789 / 1160.
#include <algorithm>

#include "fdga_digits.cuh"
#include "fdga_kernels.h"
#include "fdga_ring.h"

namespace fdga {

namespace {

constexpr int WORKERS = 256;              // threads that form and digitise M
constexpr int OZ_THREADS = WORKERS + 32;  // and the control warp
constexpr int S = 8;                      // digits per operand
constexpr int KC = 16;                    // real K per chunk (one FP16 MMA)
constexpr int CW = KC / 2;                // ω per chunk
constexpr int NT = 64;                    // real columns per tile
constexpr int TCOLS = S * NT;             // tensor-memory columns (512: all of them)
constexpr int B_DIG = NT * KC * 2;        // one B digit operand: 64 rows x 16 FP16 = 2 KB
constexpr int CPITCH = NT / 2 + 1;        // complex values between rows of the results (one pad: 16-byte stores
                                          // of neighbouring rows fall on distinct banks)
// one stage: the S digit operands of A (N rows x 16 FP16 each), then those of B
__host__ __device__ constexpr uint32_t stage_bytes(int N) { return (uint32_t)S * (uint32_t)(N * KC * 2 + B_DIG); }
constexpr uint32_t SPIN_LIMIT = 1u << 22;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// byte offset of element (row r, k) in a K-major no-swizzle operand of 16-bit elements, KC columns:
// 8-row x 16-byte core matrices, K-adjacent ones 128 B apart, 8-row groups KC·16 = 256 B apart
__device__ __forceinline__ uint32_t op16(int r, int k) {
    return (uint32_t)((((r >> 3) * (KC / 8) + (k >> 3)) << 7) + ((r & 7) << 4) + ((k & 7) << 1));
}
__device__ __forceinline__ uint64_t sdesc16(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)((KC * 16) >> 4) << 32) |
           (1ull << 46);
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, const volatile int* stop) {
    for (uint32_t i = 0; i < SPIN_LIMIT; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
        if (stop && *stop) return false;
    }
    return false;
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// global -> shared bulk copy (16-byte aligned addresses, a multiple of 16 bytes), completing on bar
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void mma_f16(uint32_t dt, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
        :
        : "r"(dt), "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}

// The A digit operands of the blocks r0, r0 + 1, ..: one CTA per block, one warp per eight rows.  Four lanes
// share a row, four neighbouring ω each per step; the row's largest exponent field (fa[block][row], read by the
// contraction's epilogue) comes first, then the lanes write, per chunk of 8 ω, 16 bytes of each of the S digit
// operands in the K-major no-swizzle layout of op16 (N·32 bytes each): eight lanes fill a 128-byte core matrix.
__global__ void __launch_bounds__(256) k_oz_adigits(K3Args3 args, Dims d, int* __restrict__ fa, uint8_t* adig, int r0) {
    const int N = d.N3n, nchunks = N / CW, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rr = blockIdx.x, rest = r0 + rr, nb = args.nblocks;
    const int slot = rest / nb, bi = rest % nb;
    const int blk = args.blocks ? args.blocks[bi] : bi;
    const cplx* A = (slot == 0 ? args.a[0].A : slot == 1 ? args.a[1].A : args.a[2].A) + (size_t)blk * N * N;
    const size_t arow = (size_t)N * 32;
    for (int rg = warp; rg < N / 8; rg += 8) {
        const int row = 8 * rg + (lane & 7), w00 = 4 * (lane >> 3);
        const cplx* src = A + (size_t)row * N;
        int mx = 0;
        for (int w = w00; w < N; w += 16)
#pragma unroll
            for (int i = 0; i < 4; ++i) mx = max(mx, cexpo(ldg(src + w + i)));
        mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
        mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
        if (lane < 8) fa[(size_t)rest * N + row] = mx;
        for (int w = w00; w < N; w += 16) {
            unsigned long long re[4], im[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const cplx x = ldg(src + w + i);
                re[i] = (unsigned long long)fixed_digits<S>(x.x, mx) + DIGIT_BIAS;
                im[i] = (unsigned long long)fixed_digits<S>(x.y, mx) + DIGIT_BIAS;
            }
            uint8_t* dst = adig + ((size_t)rr * nchunks + (w >> 3)) * S * arow + op16(row, 2 * (w & 4));
#pragma unroll
            for (int s = 0; s < S; ++s)
                *reinterpret_cast<uint4*>(dst + (size_t)s * arow) =
                    make_uint4(digit_pair(re[0], im[0], S - 1 - s), digit_pair(re[1], im[1], S - 1 - s),
                               digit_pair(re[2], im[2], S - 1 - s), digit_pair(re[3], im[3], S - 1 - s));
        }
    }
}

// MAXC: the largest number of chunks (N/8) of an instantiation, the entries of M a worker holds; NS: stages
template <int MODE, int MAXC, int NS>
__global__ void __launch_bounds__(OZ_THREADS, 2)
    k_bse_K3_oz(K3Args3 args, Dims d, int ntile, const int* __restrict__ fa, const uint8_t* __restrict__ adig, int r0,
                int* err) {
    extern __shared__ __align__(128) uint8_t sm[];  // NS stages; later the results; behind them qf
    __shared__ uint64_t done_[NS];   // per stage: the chunk's MMAs are done (tcgen05.commit)
    __shared__ uint64_t afull_[NS];  // per stage: the chunk's A digit operands have arrived
    __shared__ uint64_t bfull_[NS];  // per stage: the workers have written the chunk's B digit operands
    __shared__ uint32_t tmem_base;
    __shared__ int abort_;
    __shared__ int committed_;  // chunks whose MMAs were committed
    __shared__ int cmax[NT / 2];  // largest exponent fields of the columns of M
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const bool worker = warp < WORKERS / 32;
    const int N = d.N3n;
    const int nchunks = N / CW;  // N is a multiple of 8
    const int nb = args.nblocks;
    const int tile = blockIdx.x % ntile;
    const int rest = r0 + (int)(blockIdx.x / ntile);
    const int slot = rest / nb;
    const int blk = args.blocks ? args.blocks[rest % nb] : (int)(rest % nb);
    const K3Args& a = args.a[slot];
    const int CH = args.ch[slot];
    const int m = blk % d.N3O - (d.n3O - 1), P = blk / d.N3O;
    const size_t base = (size_t)blk * N * N;
    const int col0 = tile * NT;                      // first real column of the tile
    const int ncol = min(NT, 2 * N - col0);          // 16, 32, 48 or 64
    const int cc0 = col0 / 2, ncc = ncol / 2;        // complex columns ν'
    const double s1 = (CH == CH_A) ? 1.0 : -1.0, s2 = (CH == CH_T) ? -1.0 : 1.0;
    // M has the Γ and γL terms (mode 1 but the one-loop form; mode 3 always)
    const bool full = MODE == 3 || (MODE == 1 && (a.flags & K3F_1LOOP) == 0);
    auto done = [&](int st) { return smem_u32(done_ + st); };
    auto afull = [&](int st) { return smem_u32(afull_ + st); };
    auto bfull = [&](int st) { return smem_u32(bfull_ + st); };
    const uint32_t arow = (uint32_t)N * 32u, stage = stage_bytes(N);
    // the ω factors of M with their signs: [0] Π0 (mode 0), s1 (Π - Π0) (mode 1) or s1 dΠ (mode 3),
    // [1] s1 Π
    cplx(*qf)[2] = reinterpret_cast<cplx(*)[2]>(sm + max(NS * stage, (uint32_t)(N * CPITCH) * (uint32_t)sizeof(cplx)));
    // A: row ν, k = 2ω_l holds Re A, 2ω_l + 1 holds Im A; the S operands of a chunk arrive by one copy
    auto copy_A = [&](int c) {
        const int st = ring_stage(c, NS);
        mbar_expect_tx(afull(st), (uint32_t)S * arow);
        bulk_g2s(smem_u32(sm + (size_t)st * stage), adig + ((size_t)(rest - r0) * nchunks + c) * S * arow,
                 (uint32_t)S * arow, afull(st));
    };
    if (!worker && lane == 0) {
        abort_ = 0;
        for (int i = 0; i < NS; ++i) {
            mbar_init(done(i), 1);
            mbar_init(afull(i), 1);
            mbar_init(bfull(i), WORKERS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (int c = 0; c < min(nchunks, NS); ++c) copy_A(c);
    }
    if (tid < N) {
        const size_t ip = ixPi(d, P, m, tid - d.n3n);
        const cplx pi0 = (MODE != 3 && a.Pi0) ? ldg(a.Pi0 + ip) : mk(0.0, 0.0);
        cplx q0 = pi0, q1 = mk(0.0, 0.0);
        if (MODE >= 1) {
            const cplx pi = ldg(a.Pi + ip);
            q1 = pi * s1;
            q0 = (MODE == 3) ? ldg(a.tPi + ip) * s1 : (pi - pi0) * s1;
        }
        qf[tid][0] = q0;
        qf[tid][1] = q1;
    }
    if (tid < NT / 2) cmax[tid] = 0;
    __syncthreads();
    // γL at a K3 index in the channel's spin combination (t: 2 FL.γt - FL.γa), of FL or of the tangent's dFL
    auto gl_of = [&](const cplx* FLc, const cplx* FLt, const cplx* FLa, size_t i) -> cplx {
        if (CH == CH_T) {
            const cplx t = ldg(FLt + i), u = ldg(FLa + i);
            return cplx{fma(t.x, 2.0, -u.x), fma(t.y, 2.0, -u.y)};
        }
        return ldg(FLc + i);
    };
    // a worker's column of the tile and its ω within a chunk (narrow last tiles take fewer, full warps); its
    // entries of M, one per chunk
    const int csh = ncc <= 8 ? 3 : (ncc <= 16 ? 4 : 5);
    const int wl = tid >> csh, cl = tid & ((1 << csh) - 1);
    const bool have = worker && cl < ncc && wl < CW;
    cplx mv[MAXC];
    int em = 0;
#pragma unroll
    for (int c = 0; c < MAXC; ++c) {
        mv[c] = mk(0.0, 0.0);
        if (have && c < nchunks) {
            const int w = CW * c + wl, col = cc0 + cl;
            cplx x0 = ldg(a.B0 + base + (size_t)w * N + col);
            if (full) {
                // s2 Π = ±s1 Π: the γL terms join the Γ terms before the products
                const size_t ig = (CH == CH_P) ? base + (size_t)w * N + col : base + (size_t)col * N + w;
                const int ot = cross(CH, m, w - d.n3n);
                const bool hl = fin(ot, d.n3n);
                const size_t il = base + (size_t)(ot + d.n3n) * N + col;
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
                mv[c] = cfma(qf[w][0], x0, qf[w][1] * g);
            } else {
                mv[c] = qf[w][0] * x0;
            }
            em = max(em, cexpo(mv[c]));
        }
    }
    if (have) atomicMax(&cmax[cl], em);
    __syncthreads();
    bool ok = true;
    if (!worker) {
        // the whole tensor memory: waits for the neighbour CTA of the SM to give it back
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                     "n"(TCOLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
            const uint32_t tmem = *(volatile uint32_t*)&tmem_base;
            // instruction descriptor: D FP32, A and B FP16, both K-major, N = ncol, M = 128
            const uint32_t idesc = (1u << 4) | ((uint32_t)(ncol >> 3) << 17) | ((128u >> 4) << 24);
            // shared-memory descriptors of the first A and B digit operands of stage 0 (the start address
            // field, bits 0-13, takes the byte offsets of the other operands >> 4 without carry: all of the
            // shared memory lies below 2^18 bytes)
            const uint64_t dA0 = sdesc16(smem_u32(sm)), dB0 = sdesc16(smem_u32(sm) + S * arow);
            int copied = min(nchunks, NS), committed = 0;
            for (int c = 0; c < nchunks && ok; ++c) {
                const int st = ring_stage(c, NS);
                const uint32_t par = ring_parity(c, NS);
                ok = mbar_wait(afull(st), par, &abort_) && mbar_wait(bfull(st), par, &abort_);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t so = (uint64_t)((uint32_t)st * stage >> 4);
#pragma unroll
                for (int s = 0; s < S; ++s)
#pragma unroll
                    for (int t = 0; t + s < S; ++t)
                        mma_f16(tmem + (uint32_t)((s + t) * NT), dA0 + so + (uint64_t)((uint32_t)s * arow >> 4),
                                dB0 + so + (uint64_t)((t * B_DIG) >> 4), idesc, (c > 0 || s > 0) ? 1u : 0u);
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(done(st))
                             : "memory");
                committed = c + 1;
                if (c >= 1 && c - 1 + NS < nchunks) {  // the stage of chunk c - 1 is free once that is done
                    ok = mbar_wait(done(ring_stage(c - 1, NS)), ring_parity(c - 1, NS), &abort_);
                    if (ok) {
                        copy_A(c - 1 + NS);
                        ++copied;
                    }
                }
            }
            if (!ok) {
                // a wait gave up: report it, stop the workers, and wait (bounded) for the copies in flight;
                // the MMAs in flight end before the tensor memory is released (below)
                abort_ = 1;
                atomicExch(err, 1);
                for (int c = max(0, copied - NS); c < copied; ++c)
                    mbar_wait(afull(ring_stage(c, NS)), ring_parity(c, NS), nullptr);
            }
            committed_ = committed;
        }
        __syncwarp();
    } else {
        // B (rows n = 2ν'_l + p of the tile, k = 2ω_l + q): row 2ν'_l holds [Re M, -Im M], row 2ν'_l + 1 holds
        // [Im M, Re M]
        const int F = have ? cmax[cl] : 0;
        const uint32_t o0 = op16(2 * cl, 2 * wl), o1 = op16(2 * cl + 1, 2 * wl);
#pragma unroll
        for (int c = 0; c < MAXC; ++c) {
            if (c < nchunks && ok) {
                const int st = ring_stage(c, NS);
                if (c >= NS) ok = mbar_wait(done(st), ring_parity(c - NS, NS), &abort_);
                if (ok) {
                    if (have) {
                        const unsigned long long yr = (unsigned long long)fixed_digits<S>(mv[c].x, F) + DIGIT_BIAS;
                        const unsigned long long yi = (unsigned long long)fixed_digits<S>(mv[c].y, F) + DIGIT_BIAS;
                        uint8_t* b = sm + (size_t)st * stage + S * arow;
#pragma unroll
                        for (int s = 0; s < S; ++s) {
                            const uint32_t p = digit_pair(yr, yi, S - 1 - s);
                            *reinterpret_cast<uint32_t*>(b + s * B_DIG + o0) = p ^ 0x80000000u;
                            *reinterpret_cast<uint32_t*>(b + s * B_DIG + o1) = __byte_perm(p, p, 0x1032);
                        }
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    mbar_arrive(bfull(st));
                }
            }
        }
        // (commits complete in order: the last one is the end of all)
        if (ok) ok = mbar_wait(done(ring_stage(nchunks - 1, NS)), ring_parity(nchunks - 1, NS), &abort_);
        if (!ok) {  // (any lane's: the control thread may have ended its part)
            abort_ = 1;
            atomicExch(err, 1);
        }
    }
    ok = __all_sync(0xffffffffu, ok);  // (a wait may give up in some lanes only)
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const int q = warp & 3, h = warp >> 2;
    const int nu = 32 * q + lane;
    cplx* Cs = reinterpret_cast<cplx*>(sm);  // (all chunks are done: the stages are free)
    if (ok && worker && 32 * q < N) {
        // warp w reads TMEM lanes 32(w%4).. (rows ν) and the 32-column half w/4 of the tile, 8 columns at a time
        const uint32_t tmem = *(volatile uint32_t*)&tmem_base;
        const int FA = nu < N ? fa[(size_t)rest * N + nu] : 0;
#pragma unroll 1
        for (int cb = 32 * h; cb < min(32 * h + 32, ncol); cb += 8) {
            float r[S][8];
#pragma unroll
            for (int g = 0; g < S; ++g) {
                const uint32_t taddr = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(g * NT + cb);
                asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                             : "=f"(r[g][0]), "=f"(r[g][1]), "=f"(r[g][2]), "=f"(r[g][3]), "=f"(r[g][4]), "=f"(r[g][5]),
                               "=f"(r[g][6]), "=f"(r[g][7])
                             : "r"(taddr)
                             : "memory");
            }
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (nu < N) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int col = cb / 2 + j, FM = cmax[col];
                    cplx o;
                    if (FA == 0x7ff || FM == 0x7ff) {
                        const double qn = __longlong_as_double(0x7ff8000000000000ll);
                        o = mk(qn, qn);
                    } else {
                        float x[S], y[S];
#pragma unroll
                        for (int g = 0; g < S; ++g) { x[g] = r[g][2 * j]; y[g] = r[g][2 * j + 1]; }
                        o = mk(join_digits<S>(x, FA + FM), join_digits<S>(y, FA + FM));
                    }
                    st16(Cs + (size_t)nu * CPITCH + col, o);
                }
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    __syncthreads();
    if (!worker) {
        // after an abort the MMAs of the last chunks committed may still run: a bounded wait before the release for
        // the last one (commits complete in order, and its stage's earlier uses were waited for before it)
        if (abort_ && committed_ > 0)
            mbar_wait(done(ring_stage(committed_ - 1, NS)), ring_parity(committed_ - 1, NS), nullptr);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(*(volatile uint32_t*)&tmem_base), "n"(TCOLS));
        return;
    }
    if (abort_ || cl >= ncc) return;
#pragma unroll 4
    for (int r = wl; r < N; r += WORKERS >> csh) {
        const size_t io = base + (size_t)r * N + cc0 + cl;
        const cplx cv = ld16(Cs + (size_t)r * CPITCH + cl);
        cplx o;
        if (MODE == 0) {
            o = cv * (d.T * ((CH == CH_A) ? 1.0 : -1.0));
        } else if (a.flags & K3F_NOEPI) {
            o = cv * d.T;
        } else {
            const cplx g = (MODE == 3) ? gl_of(a.tFLc, a.tFLt, a.tFLa, io) : gl_of(a.FLc, a.FLt, a.FLa, io);
            o = cplx{fma(cv.x, d.T, g.x), fma(cv.y, d.T, g.y)};
        }
        if (a.flags & K3F_ACC) o = ld16(a.out + io) + o;
        st16(a.out + io, o);
    }
}

}  // namespace

bool k3_oz_supported(const Dims& d) {
    // rows ν < N of the 128-lane accumulator; column tiles of 64, the last one of a multiple of 16 (MMA N % 16)
    return d.N3n >= 8 && d.N3n <= 128 && (d.N3n % 8) == 0;
}

// the stages (an A operand is read up to row 127: behind the last digit's N rows into the stage's 16 KB of B), or
// the results; then the ω factors
static size_t k3_oz_smem(const Dims& d, int ns) {
    const size_t N = (size_t)d.N3n;
    return std::max(ns * (size_t)stage_bytes(d.N3n), N * CPITCH * sizeof(cplx)) + 2 * N * sizeof(cplx);
}

// NS: stages of mode 0, where the MMAs wait for the operands; modes 1 and 3 are bound by forming M, whose loads
// want the L1 cache that a third stage takes (4x4, nK3 = (20, 40): K3 kernel, at seven digits, 394 us with two
// stages, 407 with three; L_K3 stage 392 and 331).  Above Nν3 = 80 three stages leave room for one CTA on an SM only.
template <int MAXC, int NS>
static cudaError_t prepare_oz(const Dims& d) {
    cudaError_t e = raise_smem_limit_of<k_bse_K3_oz<0, MAXC, NS>>(k3_oz_smem(d, NS), 0);
    if (e == cudaSuccess) e = raise_smem_limit_of<k_bse_K3_oz<1, MAXC, 2>>(k3_oz_smem(d, 2), 0);
    if (e == cudaSuccess) e = raise_smem_limit_of<k_bse_K3_oz<3, MAXC, 2>>(k3_oz_smem(d, 2), 0);
    return e;
}
cudaError_t prepare_bse_K3_oz(const Dims& d) {
    if (d.N3n <= 64) return prepare_oz<8, 3>(d);
    if (d.N3n <= 80) return prepare_oz<12, 3>(d);
    return d.N3n <= 96 ? prepare_oz<12, 2>(d) : prepare_oz<16, 2>(d);
}

// mode 0 (BSE_L_K3), 1 (BSE_K3), 2 (the tangent dK3 = T (dA·M + A·dM) + dγL): mode 2 runs as two
// launches, each with its own bounds (dA and A need not share a magnitude): the mode-1 kernel
// on dA with the epilogue term left out, then the A·dM kernel adding T C + dγL into the output
template <int MAXC, int NS>
static cudaError_t launch_oz(cudaStream_t s, int mode, const K3Args3& a, int nslots, const Dims& d, int* err,
                             int* fa_scratch, uint8_t* adig, int adig_blocks) {
    const int ntile = (2 * d.N3n + NT - 1) / NT;
    const int nblk = nslots * a.nblocks;
    // per launch: groups of at most adig_blocks blocks (the size of the digit buffer), each
    // digitised (with its exponent bounds) and contracted in stream order
    auto run = [&](auto kernel, size_t smem, const K3Args3& ka) -> cudaError_t {
        cudaError_t e = cudaSuccess;
        for (int r0 = 0; e == cudaSuccess && r0 < nblk; r0 += adig_blocks) {
            const int cnt = std::min(adig_blocks, nblk - r0);
            k_oz_adigits<<<(unsigned)cnt, 256, 0, s>>>(ka, d, fa_scratch, adig, r0);
            e = cudaGetLastError();
            if (e != cudaSuccess) break;
            kernel<<<(unsigned)(cnt * ntile), OZ_THREADS, smem, s>>>(ka, d, ntile, fa_scratch, adig, r0, err);
            e = cudaGetLastError();
        }
        return e;
    };
    if (mode == 2) {
        K3Args3 a1 = a, a3 = a;
        for (int i = 0; i < nslots; ++i) {
            if (a.a[i].flags & K3F_1LOOP) return cudaErrorInvalidValue;  // no tangent of the one-loop form
            a1.a[i].A = a.a[i].tA;
            a1.a[i].flags |= K3F_NOEPI;
            a3.a[i].flags |= K3F_ACC;
        }
        // stream order: the second launch's pre-pass overwrites the scratch after the first
        // contraction has read it
        const cudaError_t e = run(k_bse_K3_oz<1, MAXC, 2>, k3_oz_smem(d, 2), a1);
        if (e != cudaSuccess) return e;
        return run(k_bse_K3_oz<3, MAXC, 2>, k3_oz_smem(d, 2), a3);
    }
    return mode == 1 ? run(k_bse_K3_oz<1, MAXC, 2>, k3_oz_smem(d, 2), a) : run(k_bse_K3_oz<0, MAXC, NS>, k3_oz_smem(d, NS), a);
}
cudaError_t launch_bse_K3_oz(cudaStream_t s, int mode, const K3Args3& a, int nslots, const Dims& d, int* err,
                             int* fa_scratch, uint8_t* adig, int adig_blocks) {
    if (!k3_oz_supported(d) || mode < 0 || mode > 2 || !fa_scratch || !adig || adig_blocks < 1)
        return cudaErrorInvalidValue;
    if (d.N3n <= 64) return launch_oz<8, 3>(s, mode, a, nslots, d, err, fa_scratch, adig, adig_blocks);
    if (d.N3n <= 80) return launch_oz<12, 3>(s, mode, a, nslots, d, err, fa_scratch, adig, adig_blocks);
    if (d.N3n <= 96) return launch_oz<12, 2>(s, mode, a, nslots, d, err, fa_scratch, adig, adig_blocks);
    return launch_oz<16, 2>(s, mode, a, nslots, d, err, fa_scratch, adig, adig_blocks);
}

size_t k3_oz_digit_bytes(const Dims& d) { return (size_t)4 * S * d.N3n * d.N3n; }

}  // namespace fdga
