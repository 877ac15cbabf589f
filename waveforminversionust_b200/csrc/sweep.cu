// Batched forward and adjoint block-tridiagonal sweeps of applyBlockLU
// (Runtime/solver/applyBlockLU.cu:433-467), complex single on CUDA cores.
//
// Forward (H u = src):
//   j = 1..Nx-1 :  tmp = SRC_j - L_{j-1} u_{j-1};   u_j  = invT_j tmp       [stencil, GEMM]
//   j = Nx-2..0 :  tmp = U_j u_{j+1};               u_j -= invT_j tmp       [stencil, GEMM]
// Adjoint (H^H u = src):
//   j = 1..Nx-1 :  tmp = invT_{j-1}^H u_{j-1};      u_j  = SRC_j - U_{j-1}^H tmp   [GEMM, stencil]
//   j = Nx-2..0 :  tmp = u_j - L_j^H u_{j+1};       u_j  = invT_j^H tmp     [stencil, GEMM]
//
// The sources are independent of one another, so a thread-block cluster takes
// a few of them through every column of both substitutions in one launch
// (sweep_cluster_kernel).  Pages too tall for it take two launches per column
// step: a tridiagonal stencil over (y, source) that writes the dense operand
// tmp, and a 32 x 32-tile complex GEMM over the interior rows (invT pages
// have zero borders) whose K loop prefetches the next A and B slabs into
// registers while the current slab is multiplied from double-buffered shared
// memory.  Threads run along y, so every field access is a contiguous,
// coalesced column segment.
#include <cuda.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"
#include "tc.cuh"
#include "tcstep.cuh"

namespace wust {

constexpr int SBM = 32, SBN = 32, SBK = 32, STHREADS = 256;

struct SweepParams {
    Coefs<float2> co;
    const float2 *invT;
    float2 *u;          // [ny, nx, S]
    float2 *tmp;        // [ny, S]
    SrcView src;
    int ny, nx, S, j;
};

// ---------------------------------------------------------------------------
// Tridiagonal stencils (rows 1..ny-2 unless stated), one thread per (y, s).
// ---------------------------------------------------------------------------
enum StencilMode { ST_L = 0, ST_U = 1, ST_LH = 2, ST_UH = 3 };

template <int MODE>
__global__ void stencil_kernel(SweepParams p) {
    const int ny = p.ny, j = p.j;
    const int s = blockIdx.y;
    const size_t fs = (size_t)ny * p.nx * s;
    if (MODE == ST_UH) {
        // u(:, j, s) = SRC(:, j, s) - U_{j-1}^H tmp(:, s) on every row, border
        // included (applyBlockLU.cu:159-202)
        const int y = blockIdx.x * blockDim.x + threadIdx.x;
        if (y >= ny || s >= p.S) return;
        const float2 *t = p.tmp + (size_t)ny * s;
        float2 acc = make_float2(0.f, 0.f);
        cfma_conj(acc, p.co.ud(y, j - 1), t[y]);
        if (y > 0) cfma_conj(acc, p.co.uu(y - 1, j - 1), t[y - 1]);
        if (y < ny - 1) cfma_conj(acc, p.co.ul(y, j - 1), t[y + 1]);
        p.u[fs + (size_t)ny * j + y] = csub(p.src.get(y, j, s, ny, p.nx), acc);
        return;
    }
    const int y = blockIdx.x * blockDim.x + threadIdx.x + 1;
    if (y >= ny - 1 || s >= p.S) return;
    float2 out;
    if (MODE == ST_L) {          // SRC_j - L_{j-1} u_{j-1}   (applyBlockLU.cu:29-73)
        const float2 *uc = p.u + fs + (size_t)ny * (j - 1);
        float2 acc = cmul(p.co.ld(y, j - 1), uc[y]);
        cfma(acc, p.co.ll(y - 1, j - 1), uc[y - 1]);
        cfma(acc, p.co.lu(y, j - 1), uc[y + 1]);
        out = csub(p.src.get(y, j, s, ny, p.nx), acc);
    } else if (MODE == ST_U) {   // U_j u_{j+1}   (applyBlockLU.cu:95-137)
        const float2 *uc = p.u + fs + (size_t)ny * (j + 1);
        out = cmul(p.co.ud(y, j), uc[y]);
        cfma(out, p.co.ul(y - 1, j), uc[y - 1]);
        cfma(out, p.co.uu(y, j), uc[y + 1]);
    } else {                     // u_j - L_j^H u_{j+1}   (applyBlockLU.cu:224-267)
        const float2 *un = p.u + fs + (size_t)ny * (j + 1);
        float2 acc = make_float2(0.f, 0.f);
        cfma_conj(acc, p.co.ld(y, j), un[y]);
        cfma_conj(acc, p.co.lu(y - 1, j), un[y - 1]);
        cfma_conj(acc, p.co.ll(y, j), un[y + 1]);
        out = csub(p.u[fs + (size_t)ny * j + y], acc);
    }
    p.tmp[y + (size_t)ny * s] = out;
}

// ---------------------------------------------------------------------------
// C(r, s) (op)= op(A)(r, k) B(k, s) over interior r, k in [1, ny-1).
// A: one invT page, column-major ld ny; op = identity or conjugate transpose.
// B(k, s) = Bp[k + ldb * s]; C(r, s) = Cp[r + ldc * s].
// EPI: 0 store, 1 subtract; RING: also zero C rows 0 and ny-1.
// ---------------------------------------------------------------------------
template <bool CONJT, int EPI, bool RING>
__global__ void __launch_bounds__(STHREADS) cgemm_step_kernel(const float2 *__restrict__ A, const float2 *Bp,
                                                              size_t ldb, float2 *Cp, size_t ldc, int ny, int S) {
    __shared__ float2 As[2][SBK][SBM + 1];   // As[buf][k][r] = op(A)(r, k)
    __shared__ float2 Bs[2][SBK][SBN + 1];   // Bs[buf][k][s]
    const int tid = threadIdx.x, tr = tid % 16, tc = tid / 16;
    const int r0 = 1 + blockIdx.x * SBM;
    const int s0 = blockIdx.y * SBN;
    const int nslab = (ny - 2 + SBK - 1) / SBK;
    constexpr int PER = SBM * SBK / STHREADS;   // 4

    float2 ra[PER], rb[PER];
    auto fetch = [&](int slab) {
        const int k0 = 1 + slab * SBK;
#pragma unroll
        for (int m = 0; m < PER; ++m) {
            const int e = tid + m * STHREADS;
            int rr, kk;
            if (CONJT) { kk = e % SBK; rr = e / SBK; }
            else { rr = e % SBM; kk = e / SBM; }
            const int r = r0 + rr, k = k0 + kk;
            float2 v = make_float2(0.f, 0.f);
            if (r < ny - 1 && k < ny - 1) v = CONJT ? cconj(A[k + (size_t)ny * r]) : A[r + (size_t)ny * k];
            ra[m] = v;
            const int kb = e % SBK, sb = e / SBK;
            const int kg = k0 + kb, sg = s0 + sb;
            rb[m] = (kg < ny - 1 && sg < S) ? Bp[kg + ldb * sg] : make_float2(0.f, 0.f);
        }
    };
    auto stash = [&](int buf) {
#pragma unroll
        for (int m = 0; m < PER; ++m) {
            const int e = tid + m * STHREADS;
            if (CONJT) As[buf][e % SBK][e / SBK] = ra[m];
            else As[buf][e / SBM][e % SBM] = ra[m];
            Bs[buf][e % SBK][e / SBK] = rb[m];
        }
    };

    float2 acc[2][2];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int jj = 0; jj < 2; ++jj) acc[i][jj] = make_float2(0.f, 0.f);

    fetch(0);
    for (int slab = 0; slab < nslab; ++slab) {
        const int buf = slab & 1;
        stash(buf);
        __syncthreads();
        if (slab + 1 < nslab) fetch(slab + 1);
#pragma unroll 8
        for (int kk = 0; kk < SBK; ++kk) {
            const float2 a0 = As[buf][kk][tr], a1 = As[buf][kk][tr + 16];
            const float2 b0 = Bs[buf][kk][tc], b1 = Bs[buf][kk][tc + 16];
            cfma(acc[0][0], a0, b0);
            cfma(acc[0][1], a0, b1);
            cfma(acc[1][0], a1, b0);
            cfma(acc[1][1], a1, b1);
        }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
#pragma unroll
        for (int jj = 0; jj < 2; ++jj) {
            const int r = r0 + tr + 16 * i, s = s0 + tc + 16 * jj;
            if (r >= ny - 1 || s >= S) continue;
            float2 *dst = Cp + r + ldc * s;
            *dst = (EPI == 1) ? csub(*dst, acc[i][jj]) : acc[i][jj];
        }
    }
    if (RING && blockIdx.x == 0 && tid < 2 * SBN) {
        const int s = s0 + tid / 2;
        if (s < S) Cp[((tid % 2) ? ny - 1 : 0) + ldc * s] = make_float2(0.f, 0.f);
    }
}

template <int MODE>
static void launch_stencil(const SweepParams &p, cudaStream_t st) {
    const int rows = (MODE == ST_UH) ? p.ny : p.ny - 2;
    dim3 grid(ceil_div(rows, 128), p.S);
    stencil_kernel<MODE><<<grid, 128, 0, st>>>(p);
    ++g_kernel_launches;
}

template <bool CONJT, int EPI, bool RING>
static void launch_gemm(const float2 *A, const float2 *B, size_t ldb, float2 *C, size_t ldc, int ny, int S,
                        cudaStream_t st) {
    if (ny <= 2) return;
    dim3 grid(ceil_div(ny - 2, SBM), ceil_div(S, SBN));
    cgemm_step_kernel<CONJT, EPI, RING><<<grid, STHREADS, 0, st>>>(A, B, ldb, C, ldc, ny, S);
    ++g_kernel_launches;
}

// ---------------------------------------------------------------------------
// One launch per solve: a cluster of CL CTAs takes NS sources through all
// 2 (nx - 1) column steps.  Every CTA holds its rows of the page's product;
// the finished column goes to the shared memory of all CTAs of the cluster,
// which then form the next right-hand side (the tridiagonal stencil) for all
// rows on their own, so that a step has one exchange.  Per step and CTA:
//   GEMM     its RB rows x NS sources over all n, in eight partial tiles over
//            K, RW x NSW per thread.  H: warp w takes an eighth of the page
//            columns and all rows.  H^H, whose operand has K contiguous: warp
//            w takes an eighth of the rows and lane phase ph the page rows
//            ph, ph + 8, ...  Each warp streams its share of the page through
//            a ring of its own, two TMA boxes per stage (they do not depend on
//            the state, so the next step's first ones, and its page into L2,
//            are on their way during the exchange).  A box starts on 16
//            bytes, a page column (8 ny bytes) wherever the parity puts it:
//            the tensor map takes two columns as one row, so that one box
//            holds a stage's even columns and one its odd ones, each copied
//            from the boundary before and read from an offset of one entry.
//            (16-byte cp.async instead, by the same warps: 10 us of issue on
//            top of the 15 that the multiply-adds take; 8-byte ones, bulk
//            copies per column or loads into registers: as much or more.)
//   exchange the eight partial tiles are summed in a fixed order, subtracted
//            from the old column where the substitution says so, written to u
//            and to every CTA's copy of the column;
//   stencil  B = base - W c for all rows (base and weights were fetched
//            before the cluster barrier).
// What bounds it: at 552^2 x 256 the FP32 multiply-adds of the GEMM (a
// 6 x 6 tile per thread takes 2.7 bytes from L1 and shared memory per complex
// multiply-add, where 4 would balance the two); on small pages the chain
// exchange - barrier - stencil.  The cluster barrier is the hardware's, and
// every thread of the cluster reaches it; there is no other wait.
// Measured, us per column step before (two launches) -> now: 552^2 x 256 H
// 35 -> 23, H^H 44 -> 25; 224^2 x 32 18 -> 3.7, 20 -> 4.9; 64^2 x 6 9.3 -> 1.8,
// 8.6 -> 2.5.
// ---------------------------------------------------------------------------
constexpr int CT = 256, CW = CT / 32;    // threads, warps
constexpr int kCsMaxCl = 8;

struct __align__(64) SweepClusterParams {
    Coefs<float2> co;
    const float2 *invT;
    float2 *u;          // [ny, nx, S]
    SrcView src;
    int *err;
    int ny, nx, S, n, RB, stages;
    int s0;             // first source of the launch
    unsigned long long timeout_ns;
    CUtensorMap pages;  // invT as rows of two page columns, a box of one parity of a stage's columns
};

template <bool ADJ, int RW, int NSW>
struct SweepShape {
    static constexpr int TR = 16 * RW, NS = 2 * NSW;
    static constexpr int WR = TR / CW;                       // H^H: rows per warp
    static constexpr int SK = ADJ ? 32 : 8;                  // K per stage
    static constexpr int COLS = ADJ ? WR : SK;               // page columns per stage, half of them per box
    // entries of a column in a box: the part read, one of offset; H^H: 16 words between the row groups of a warp
    static constexpr int INN = ADJ ? (RW == 6 || RW == 2 ? 40 : 36) : TR + 2;
    static constexpr int box = (int)sizeof(float2) * INN * (COLS / 2);
    static constexpr int box_at = (box + 127) / 128 * 128;
    static constexpr size_t stage = 2 * box_at;
    static_assert(COLS % 2 == 0 && INN % 2 == 0 && INN <= 256, "a box of whole 16-byte units");
    static constexpr int ITEMS = RW * NSW > 16 ? 5 : 6;      // stencil items per thread: 2 n <= ITEMS * CT
    static constexpr int NSP = NS > 2 ? NS + 2 : NS;         // entries per row of B: rows of a quarter-warp in distinct banks
    static constexpr int PS = NS * TR + 2;                   // entries per partial tile, likewise
    // K of a warp (H: an eighth) in whole stages
    __host__ __device__ static int kper(int n) { return ADJ ? (n + SK - 1) / SK * SK : ((n + CW - 1) / CW + SK - 1) / SK * SK; }
    __host__ __device__ static int ldc(int ny) { return (ny + 3) / 2 * 2; }
    __host__ __device__ static size_t col(int ny) { return sizeof(float2) * (size_t)NS * ldc(ny); }
    __host__ __device__ static size_t work(int n) {          // B, or the partial tiles
        const size_t b = sizeof(float2) * (size_t)n * NSP, q = sizeof(float2) * (size_t)CW * PS;
        return b > q ? b : q;
    }
    __host__ __device__ static size_t ring(int ny) { return (col(ny) + work(ny - 2) + 127) / 128 * 128; }
    static size_t bytes(int ny, int stages) { return ring(ny) + (size_t)CW * stages * (stage + sizeof(uint64_t)); }
};

template <int N>
__device__ __forceinline__ void load_pairs(float2 (&v)[N], const float2 *p) {
    if constexpr (N % 2 == 0) {
#pragma unroll
        for (int i = 0; i < N; i += 2) {
            const float4 q = *reinterpret_cast<const float4 *>(p + i);
            v[i] = make_float2(q.x, q.y);
            v[i + 1] = make_float2(q.z, q.w);
        }
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = p[i];
    }
}

template <bool ADJ, int RW, int NSW>
__global__ void __launch_bounds__(CT, 1) sweep_cluster_kernel(const __grid_constant__ SweepClusterParams p) {
    using Sh = SweepShape<ADJ, RW, NSW>;
    constexpr int TR = Sh::TR, NS = Sh::NS, NSP = Sh::NSP, HS = NS / 2, PS = Sh::PS, ITEMS = Sh::ITEMS;
    constexpr int SK = Sh::SK, INN = Sh::INN;
    // The last stage of K holds more than the interior: the page's border and entries of its neighbours, which nobody has
    // said are finite.  Tiny tiles take it whole with zeros for them, larger ones as far as it goes, after the loop over
    // full stages.  The widest tile, which uses its last register, ends it by a loop within that loop instead (552^2 H
    // 23.1 us a step, 26.4 to 27.0 in the other ways, which take up to 12 % off the small ones' 3.85 to 13.4).
    constexpr bool kTiny = RW * NSW <= 4, kWide = RW * NSW > 16;
    enum { kWhole, kLast, kAny };
    extern __shared__ __align__(128) uint8_t cs_smem[];
    const int ny = p.ny, nx = p.nx, n = p.n, ldc = Sh::ldc(ny), kper = Sh::kper(n);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float2 *C = reinterpret_cast<float2 *>(cs_smem) + 1;                   // the column: [source][y], y = 1 on 16 bytes
    float2 *X = reinterpret_cast<float2 *>(cs_smem + Sh::col(ny));         // B [k][NSP], or partials [8][source][row]
    unsigned rank, ncta;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(ncta));
    const int s_first = p.s0 + (int)(blockIdx.x / ncta) * NS, ns = min(NS, p.S - s_first);
    const int r0 = (int)rank * p.RB, rows = min(p.RB, n - r0);             // interior rows r0 .. r0 + rows - 1
    const size_t page_sz = (size_t)ny * ny, plane = (size_t)ny * nx;
    const int steps = 2 * (nx - 1);
    // this thread's entries of the tile: rows trow(x), sources tsrc .., partial tile part
    auto trow = [&](int x) { return ADJ ? 2 * RW * warp + RW * ((lane >> 3) & 1) + x : (lane & 15) + 16 * x; };
    const int tsrc = NSW * (lane >> 4), part = ADJ ? lane & 7 : warp;

    auto page_of = [&](int i) -> const float2 * {
        bool fwd;
        const int j = step_col(i, nx, fwd);
        return p.invT + page_sz * (size_t)(ADJ && fwd ? j - 1 : j);
    };
    // ---- the warp's page stream
    uint8_t *ring = cs_smem + Sh::ring(ny) + (size_t)warp * p.stages * Sh::stage;
    uint64_t *full = reinterpret_cast<uint64_t *>(cs_smem + Sh::ring(ny) + (size_t)CW * p.stages * Sh::stage) + warp * p.stages;
    // stages per step: H skips what lies beyond n
    const int k_own = warp * kper, per = ADJ ? kper / SK : max(0, min(kper, n - k_own) + SK - 1) / SK;
    int f_step = per ? 0 : steps, f_g = 0, f_slot = 0;
    int lost = 0;                                                          // stages from an expired wait to the end
    auto page_at = [&](int i) {                                            // first column of the page, of all pages
        bool fwd;
        const int j = step_col(i, nx, fwd);
        return ny * (ADJ && fwd ? j - 1 : j);
    };
    auto fetch = [&]() {
        if (f_step >= steps) return;
        if (lane == 0 && !lost) {
            const int first = page_at(f_step) + 1 + (ADJ ? r0 + Sh::WR * warp : k_own + f_g * SK);
            const int off = ADJ ? f_g * SK + 1 : r0 + 1;
            tc::mbar_expect_tx(full + f_slot, 2 * Sh::box);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int col = first + h, x = ((col & 1) * ny + off) & ~1;
                asm volatile(
                    "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                        tc::smem_u32(ring + (size_t)f_slot * Sh::stage + h * Sh::box_at)),
                    "l"(&p.pages), "r"(x), "r"(col >> 1), "r"(tc::smem_u32(full + f_slot)) : "memory");
            }
        }
        f_slot = f_slot + 1 == p.stages ? 0 : f_slot + 1;
        if (++f_g == per) { f_g = 0; ++f_step; }
    };

    // ---- stencil of step i: item it of this thread is row y of half the sources
    float2 wc[ITEMS], wm[ITEMS], wp[ITEMS], base[ITEMS][HS];
    auto item = [&](int it, int &y, int &h) {
        const int e = tid + it * CT;
        h = e >= n;
        y = e - (h ? n : 0) + 1;
        return e < 2 * n;
    };
    float wsx = 1.f, wsy = 1.f;                                            // signs of the weights
    auto fetch_stencil = [&](int i) {
        bool fwd;
        const int j = step_col(i, nx, fwd);
        // step_weights of tcstep.cuh, one pointer per weight
        const Coefs<float2> &co = p.co;
        const int jc = ADJ ? (fwd ? j - 2 : j) : (fwd ? j - 1 : j);
        const float2 *c0 = ADJ == fwd ? co.Ud : co.Ld, *c1, *c2;
        if (!ADJ) { c1 = fwd ? co.Ll : co.Ul; c2 = fwd ? co.Lu : co.Uu; }
        else { c1 = fwd ? co.Uu : co.Lu; c2 = fwd ? co.Ul : co.Ll; }
        const bool none = jc < 0;                                          // H^H, first column: c is zero
        c0 += (size_t)ny * (none ? 0 : jc);
        c1 += (size_t)(ny - 1) * (none ? 0 : jc);
        c2 += (size_t)(ny - 1) * (none ? 0 : jc);
        wsx = !ADJ && !fwd ? -1.f : 1.f;
        wsy = ADJ || !fwd ? -1.f : 1.f;
        // step_base: a column of a dense field, a receiver scatter, a point, or nothing
        const int jb = ADJ && fwd ? j - 1 : j;
        const bool from_u = ADJ && !fwd, from_src = fwd && !none;
        const float2 *D = from_u ? p.u : from_src && p.src.mode == SRC_DENSE ? p.src.dense : nullptr;
        if (D) D += plane * s_first + (size_t)ny * jb;
#pragma unroll
        for (int it = 0; it < ITEMS; ++it) {
            if (it * CT >= 2 * n) break;
            int y, h;
            const bool in = item(it, y, h);
            const float2 *Dh = D + plane * (size_t)(h * HS) + y;
#pragma unroll
            for (int q = 0; q < HS; ++q) {
                base[it][q] = f2(0.f, 0.f);
                if (in && D && h * HS + q < ns) base[it][q] = __ldcg(Dh + plane * q);
            }
            wc[it] = wm[it] = wp[it] = f2(0.f, 0.f);
            if (in && !none) {
                wc[it] = c0[y];
                wm[it] = c1[y - 1];
                wp[it] = c2[y];
            }
        }
        if (from_src && p.src.mode == SRC_POINT) {
            for (int s = 0; s < ns; ++s) {
                const int y0 = p.src.lin[s_first + s] - ny * jb;
                if (y0 < 1 || y0 > n) continue;
#pragma unroll
                for (int it = 0; it < ITEMS; ++it) {
                    int y, h;
                    const bool in = item(it, y, h) && y == y0;
#pragma unroll
                    for (int q = 0; q < HS; ++q)
                        if (in && h * HS + q == s) base[it][q] = f2(1.f, 0.f);
                }
            }
        } else if (from_src && p.src.mode == SRC_SCATTER) {
#pragma unroll
            for (int it = 0; it < ITEMS; ++it) {
                int y, h;
                const int k = item(it, y, h) ? p.src.at[(size_t)ny * jb + y] : -1;
                if (k < 0) continue;
#pragma unroll
                for (int q = 0; q < HS; ++q)
                    if (h * HS + q < ns) base[it][q] = p.src.vals[k + (size_t)p.src.n_slots * (s_first + h * HS + q)];
            }
        }
    };
    auto stencil = [&](int i) {
        bool fwd;
        const int j = step_col(i, nx, fwd);
        const bool wu = ADJ && fwd;                                        // B is also u(:, j - 1)
#pragma unroll
        for (int it = 0; it < ITEMS; ++it) {
            if (it * CT >= 2 * n) break;
            int y, h;
            if (!item(it, y, h)) continue;
            const float2 w0 = f2(wsx * wc[it].x, wsy * wc[it].y), w1 = f2(wsx * wm[it].x, wsy * wm[it].y);
            const float2 w2 = f2(wsx * wp[it].x, wsy * wp[it].y);
            const float2 *c = C + (size_t)(h * HS) * ldc + y;
            float2 b[HS];
#pragma unroll
            for (int q = 0; q < HS; ++q, c += ldc) {
                float2 acc = cmul(w0, c[0]);
                cfma(acc, w1, c[-1]);
                cfma(acc, w2, c[1]);
                b[q] = csub(base[it][q], acc);
            }
            float2 *dst = X + (size_t)(y - 1) * NSP + h * HS;
            if constexpr (HS % 2 == 0) {
#pragma unroll
                for (int q = 0; q < HS; q += 2)
                    *reinterpret_cast<float4 *>(dst + q) = make_float4(b[q].x, b[q].y, b[q + 1].x, b[q + 1].y);
            } else {
#pragma unroll
                for (int q = 0; q < HS; ++q) dst[q] = b[q];
            }
            if (wu && y > r0 && y <= r0 + rows) {
                float2 *uo = p.u + plane * (size_t)(s_first + h * HS) + (size_t)ny * (j - 1) + y;
#pragma unroll
                for (int q = 0; q < HS; ++q)
                    if (h * HS + q < ns) uo[plane * q] = b[q];
            }
        }
        if (wu && j >= 2) {
            // rows 0 and ny - 1 of u(:, j - 1), which no page reads
            for (int e = tid; e < 2 * ns; e += CT) {
                const int s = e >> 1, y = e & 1 ? ny - 1 : 0;
                if (rank != (e & 1 ? ncta - 1 : 0)) continue;
                float2 w0, w1, w2;
                step_weights<ADJ>(p.co, true, j, y, w0, w1, w2);
                const float2 *c = C + (size_t)s * ldc + y;
                float2 acc = f2(0.f, 0.f);
                cfma(acc, w0, c[0]);
                if (y > 0) cfma(acc, w1, c[-1]);
                else cfma(acc, w2, c[1]);
                p.u[plane * (s_first + s) + (size_t)ny * (j - 1) + y] =
                    csub(step_base<ADJ>(p.src, p.u, ny, nx, true, j, y, s_first + s), acc);
            }
        }
    };
    // The turn of the H^H solve: u(:, nx - 1) = SRC - U_{nx-2}^H c on every
    // row, which is the column that the first backward step depends on.
    auto turn = [&]() {
        constexpr int kPer = (ITEMS * CT / 2 + 2 + CT - 1) / CT;
        for (int s = 0; s < NS; ++s) {
            float2 v[kPer];
            float2 *c = C + (size_t)s * ldc;
#pragma unroll
            for (int m = 0; m < kPer; ++m) {
                const int y = tid + m * CT;
                v[m] = f2(0.f, 0.f);
                if (y >= ny || s >= ns) continue;
                float2 w0, w1, w2;
                step_weights<ADJ>(p.co, true, nx, y, w0, w1, w2);
                float2 acc = f2(0.f, 0.f);
                cfma(acc, w0, c[y]);
                if (y > 0) cfma(acc, w1, c[y - 1]);
                if (y < ny - 1) cfma(acc, w2, c[y + 1]);
                v[m] = csub(step_base<ADJ>(p.src, p.u, ny, nx, true, nx, y, s_first + s), acc);
                if ((y > r0 && y <= r0 + rows) || (y == 0 && rank == 0) || (y == ny - 1 && rank == ncta - 1))
                    p.u[plane * (s_first + s) + (size_t)ny * (nx - 1) + y] = v[m];
            }
            __syncthreads();
#pragma unroll
            for (int m = 0; m < kPer; ++m)
                if (tid + m * CT < ny) c[tid + m * CT] = v[m];
        }
        __syncthreads();
    };

    for (int e = tid; e < NS * ldc; e += CT) C[e - 1] = f2(0.f, 0.f);
    if (lane == 0)
        for (int c = 0; c < p.stages; ++c) tc::mbar_init(full + c, 1);
    tc::mbar_fence_init();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    for (int c = 0; c + 1 < p.stages; ++c) fetch();
    fetch_stencil(0);
    __syncthreads();
    stencil(0);
    // shared::cluster addresses of the column in every CTA
    unsigned col_at[kCsMaxCl];
#pragma unroll
    for (unsigned q = 0; q < kCsMaxCl; ++q)
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                     : "=r"(col_at[q]) : "r"((unsigned)__cvta_generic_to_shared(C)), "r"(q < ncta ? q : 0u));
    int slot = 0;
    uint32_t phase = 0;
    // every CTA of the cluster has started before any writes into another's shared memory
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    for (int i = 0; i < steps; ++i) {
        bool fwd;
        const int j = step_col(i, nx, fwd);
        const bool sub = !ADJ && !fwd;
        __syncthreads();                                   // B is complete
        // the next step's page into L2: each CTA of the launch its part
        if (i + 1 < steps) {
            const char *A = reinterpret_cast<const char *>(page_of(i + 1));
            const unsigned lines = (unsigned)((page_sz * sizeof(float2)) / 128);
            for (unsigned l = blockIdx.x * CT + tid; l < lines; l += gridDim.x * CT)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(A + (size_t)l * 128));
        }
        float2 acc[RW][NSW];
#pragma unroll
        for (int x = 0; x < RW; ++x)
#pragma unroll
            for (int y = 0; y < NSW; ++y) acc[x][y] = f2(0.f, 0.f);
        const int col0 = page_at(i) + 1 + (ADJ ? r0 + Sh::WR * warp : k_own);  // of this warp's columns
        // the next stage, once it has landed and the one before it is consumed
        auto next_stage = [&](int g) -> const uint8_t * {
            if (!lost && !tc::mbar_wait(full + slot, phase, p.timeout_ns)) {
                lost = (steps - i) * per - g;
                atomicCAS(p.err, 0, SITE_COPY);
            }
            __syncwarp();
            fetch();
            const uint8_t *stage = ring + (size_t)slot * Sh::stage;
            if (++slot == p.stages) {
                slot = 0;
                phase ^= 1u;
            }
            return stage;
        };
        // products of stage g: all of its K, the first `left` of it, or as many as there are
        auto multiply = [&](const uint8_t *stage, int g, auto which, int left) {
            constexpr int kWhich = decltype(which)::value;
            // column q of the stage: its box, its row, and the entry that the copy put in front of it or not
            auto column = [&](int q, int off) -> const float2 * {
                return reinterpret_cast<const float2 *>(stage + (q & 1) * Sh::box_at) + (q >> 1) * INN +
                       ((((col0 + q) & 1) * ny + off) & 1);
            };
            if constexpr (ADJ) {
                const float2 *Bs = X + (size_t)(g * SK + part) * NSP + tsrc;
                const float2 *Ar[RW];
#pragma unroll
                for (int x = 0; x < RW; ++x) Ar[x] = column(trow(x) - Sh::WR * warp, g * SK + 1) + part;
                auto product = [&](int kk, bool in) {
                    float2 b[NSW];
                    load_pairs(b, Bs + kk * NSP);
#pragma unroll
                    for (int y = 0; y < NSW; ++y) b[y] = in ? b[y] : f2(0.f, 0.f);
#pragma unroll
                    for (int x = 0; x < RW; ++x) {
                        const float2 a = in ? Ar[x][kk] : f2(0.f, 0.f);
#pragma unroll
                        for (int y = 0; y < NSW; ++y) cfma_conj(acc[x][y], a, b[y]);
                    }
                };
                if (kWhich == kWhole || (kWhich == kAny && left >= SK)) {
#pragma unroll
                    for (int kk = 0; kk < SK; kk += 8) product(kk, true);
                } else if constexpr (kWide) {
#pragma unroll 1
                    for (int kk = 0; kk < left - part; kk += 8) product(kk, true);
                } else {
#pragma unroll
                    for (int kk = 0; kk < SK; kk += 8)
                        if (kTiny || kk < left) product(kk, kk < left - part);
                }
            } else {
                const float2 *Bs = X + (size_t)(k_own + g * SK) * NSP + tsrc;
                const float2 *A0 = column(0, r0 + 1) + trow(0), *A1 = column(1, r0 + 1) + trow(0);   // SK is even
                auto product = [&](int kk, bool in) {
                    const float2 *Ak = (kk & 1 ? A1 : A0) + (kk >> 1) * INN;
                    float2 b[NSW];
                    load_pairs(b, Bs + kk * NSP);
#pragma unroll
                    for (int y = 0; y < NSW; ++y) b[y] = in ? b[y] : f2(0.f, 0.f);
#pragma unroll
                    for (int x = 0; x < RW; ++x) {
                        const float2 a = in ? Ak[16 * x] : f2(0.f, 0.f);
#pragma unroll
                        for (int y = 0; y < NSW; ++y) cfma(acc[x][y], a, b[y]);
                    }
                };
                if (kWhich == kWhole || (kWhich == kAny && left >= SK)) {
#pragma unroll
                    for (int kk = 0; kk < SK; ++kk) product(kk, true);
                } else if constexpr (kWide) {
#pragma unroll 1
                    for (int kk = 0; kk < left; ++kk) product(kk, true);
                } else {
#pragma unroll
                    for (int kk = 0; kk < SK; kk += 2)
                        if (kTiny || kk < left) {
                            product(kk, kk < left);
                            product(kk + 1, kk + 1 < left);
                        }
                }
            }
        };
        if constexpr (kWide) {
#pragma unroll 1
            for (int g = 0; g < per; ++g)
                multiply(next_stage(g), g, std::integral_constant<int, kAny>{}, n - (ADJ ? 0 : k_own) - g * SK);
        } else {
            const int k_mine = ADJ ? n : max(0, min(kper, n - k_own)), full_stages = k_mine / SK;
#pragma unroll 1
            for (int g = 0; g < full_stages; ++g) multiply(next_stage(g), g, std::integral_constant<int, kWhole>{}, SK);
            if (full_stages < per)
                multiply(next_stage(full_stages), full_stages, std::integral_constant<int, kLast>{}, k_mine - full_stages * SK);
        }
        // old column of the subtracting steps: on its way during the sums
        constexpr int MO = (TR * HS + CT - 1) / CT;
        float2 old[MO][2];
        float2 *ucol = p.u + plane * s_first + (size_t)ny * j + r0 + 1;
#pragma unroll
        for (int m = 0; m < MO; ++m) {
            const int e = tid + m * CT, r = 2 * (e % (TR / 2)), s = e / (TR / 2);
            old[m][0] = old[m][1] = f2(0.f, 0.f);
            if (sub && s < ns && r < rows) old[m][0] = __ldcg(ucol + plane * s + r);
            if (sub && s < ns && r + 1 < rows) old[m][1] = __ldcg(ucol + plane * s + r + 1);
        }
        __syncthreads();                                   // B is read: its room takes the partial tiles
#pragma unroll
        for (int y = 0; y < NSW; ++y)
#pragma unroll
            for (int x = 0; x < RW; ++x) X[(size_t)part * PS + (tsrc + y) * TR + trow(x)] = acc[x][y];
        __syncthreads();
        // every CTA has read the previous column
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        const bool wu = !ADJ || !fwd;
#pragma unroll
        for (int m = 0; m < MO; ++m) {
            const int e = tid + m * CT, r = 2 * (e % (TR / 2)), s = e / (TR / 2);
            if (s < NS && r < rows) {
                float4 v = *reinterpret_cast<const float4 *>(X + s * TR + r);
#pragma unroll
                for (int w = 1; w < CW; ++w) {
                    const float4 q = *reinterpret_cast<const float4 *>(X + (size_t)w * PS + s * TR + r);
                    v = make_float4(v.x + q.x, v.y + q.y, v.z + q.z, v.w + q.w);
                }
                if (sub) v = make_float4(old[m][0].x - v.x, old[m][0].y - v.y, old[m][1].x - v.z, old[m][1].y - v.w);
                const bool two = r + 1 < rows;
                if (!two) v.z = v.w = 0.f;                 // the next CTA's row, or the border row's zero
                if (wu && s < ns) {
                    ucol[plane * s + r] = f2(v.x, v.y);
                    if (two) ucol[plane * s + r + 1] = f2(v.z, v.w);
                }
                const unsigned at = 8u * (unsigned)(s * ldc + r0 + r + 1);
#pragma unroll
                for (unsigned q = 0; q < kCsMaxCl; ++q)
                    if (q < ncta)
                        asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(col_at[q] + at), "f"(v.x),
                                     "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
            }
        }
        if (ADJ && !fwd)                                   // border rows of u(:, j) are zero
            for (int e = tid; e < 2 * ns; e += CT)
                if (rank == (e & 1 ? ncta - 1 : 0)) p.u[plane * (s_first + (e >> 1)) + (size_t)ny * j + (e & 1 ? ny - 1 : 0)] = f2(0.f, 0.f);
        if (i + 1 < steps) fetch_stencil(i + 1);
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (i + 1 == steps) break;
        if (ADJ && i + 1 == nx - 1) turn();
        stencil(i + 1);
        if (ADJ && i + 1 == nx - 1) {                      // the columns that follow have zero border rows
            __syncthreads();
            for (int e = tid; e < 2 * NS; e += CT) C[(size_t)(e >> 1) * ldc + (e & 1 ? ny - 1 : 0)] = f2(0.f, 0.f);
        }
        __syncthreads();
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    }
    // after an expired wait: the copies issued ahead of it land (bounded) before the block ends
    if (lane == 0 && lost) {
        const int first = steps * per - lost;
        for (int c = first; c < first + min(p.stages - 1, lost); ++c)
            tc::mbar_wait(full + c % p.stages, (uint32_t)(c / p.stages) & 1u, p.timeout_ns);
    }
}

// Dynamic shared memory of any plan at most.  The kernels' attribute is set to
// this, not to the plan's: it belongs to the function, and another thread may
// be launching the same shape at another size.
constexpr size_t kSweepClusterSmem = 232448 - 1024;

// How a solve is split: cl CTAs per cluster, shape index, clusters in all and
// in one launch; cl == 0: none fits.
struct SweepPlan {
    int cl, shape, RB, clusters, per_launch, stages;
    size_t smem;
};
constexpr int kSweepShapes[][2] = {{6, 6}, {4, 4}, {3, 4}, {2, 2}, {1, 1}};    // RW, NSW

template <bool ADJ>
static size_t sweep_shape_bytes(int shape, int ny, int stages) {
    switch (shape) {
        case 0: return SweepShape<ADJ, 6, 6>::bytes(ny, stages);
        case 1: return SweepShape<ADJ, 4, 4>::bytes(ny, stages);
        case 2: return SweepShape<ADJ, 3, 4>::bytes(ny, stages);
        case 3: return SweepShape<ADJ, 2, 2>::bytes(ny, stages);
        default: return SweepShape<ADJ, 1, 1>::bytes(ny, stages);
    }
}

template <bool ADJ>
static const void *sweep_shape_kernel(int shape) {
    switch (shape) {
        case 0: return (const void *)sweep_cluster_kernel<ADJ, 6, 6>;
        case 1: return (const void *)sweep_cluster_kernel<ADJ, 4, 4>;
        case 2: return (const void *)sweep_cluster_kernel<ADJ, 3, 4>;
        case 3: return (const void *)sweep_cluster_kernel<ADJ, 2, 2>;
        default: return (const void *)sweep_cluster_kernel<ADJ, 1, 1>;
    }
}

// The shape with the least estimated time per step.  How many clusters of a
// size run at once is the B200's (148 SMs, clusters inside a GPC, one CTA per
// SM); a wrong count costs time, not correctness: the clusters do not wait on
// each other.  A cap of max_ctas CTAs is kept by launches of as many clusters
// as it holds, one after another on the stream.  Clocks per step: the
// multiply-adds at 128 per clock (1.3 of that as measured) or the page rows at
// 45 bytes per clock, the stencil of all rows, and 3000 for the sums, the
// exchange and the barriers.
template <bool ADJ>
static SweepPlan sweep_plan(int ny, int S, int max_ctas) {
    struct { int cl, at_once; } const sizes[] = {{1, 148}, {2, 70}, {4, 33}, {6, 22}, {8, 15}};
    SweepPlan best{};
    double best_t = 0;
    const int n = ny - 2;
    if (n < 1) return best;
    for (const auto &z : sizes) {
        const int at_once = max_ctas > 0 ? std::min(z.at_once, max_ctas / z.cl) : z.at_once;
        if (at_once < 1) continue;
        for (int s = 0; s < (int)(sizeof(kSweepShapes) / sizeof(kSweepShapes[0])); ++s) {
            const int TR = 16 * kSweepShapes[s][0], NS = 2 * kSweepShapes[s][1];
            const int RB = (ceil_div(n, z.cl) + 1) / 2 * 2;        // pairs of rows travel together
            if (RB > TR || RB * (z.cl - 1) >= n || 2 * n > (s == 0 ? 5 : 6) * CT) continue;
            int stages = 4;
            size_t smem = sweep_shape_bytes<ADJ>(s, ny, stages);
            while (smem > kSweepClusterSmem && stages > 2) smem = sweep_shape_bytes<ADJ>(s, ny, --stages);
            if (smem > kSweepClusterSmem) continue;
            const int clusters = ceil_div(S, NS);
            const double fma = 1.3 * 4.0 * TR * NS * n / 128.0, rows = 8.0 * RB * n / 45.0;
            const double t = (double)ceil_div(clusters, at_once) * (std::max(fma, rows) + 25.0 * n * NS / CT + 3000.0);
            if (best.cl == 0 || t < best_t) {
                best = SweepPlan{z.cl, s, RB, clusters, max_ctas > 0 ? std::min(clusters, at_once) : clusters, stages, smem};
                best_t = t;
            }
        }
    }
    return best;
}

// The tensor map of a shape's boxes; false where the pages cannot have one
// (not on 16 bytes) or the driver offers none.
template <bool ADJ, int RW, int NSW>
static bool sweep_page_map(CUtensorMap *map, const float2 *invT, int ny, int nx) {
    using Sh = SweepShape<ADJ, RW, NSW>;
    static_assert(sizeof(float2) == sizeof(double), "page entries go as 8-byte words");
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess || !fn) {
        (void)cudaGetLastError();
        return false;
    }
    const cuuint64_t dims[2] = {(cuuint64_t)2 * ny, (cuuint64_t)ny * nx / 2}, pitch[1] = {(cuuint64_t)16 * ny};
    const cuuint32_t box[2] = {(cuuint32_t)Sh::INN, (cuuint32_t)(Sh::COLS / 2)}, one[2] = {1, 1};
    return reinterpret_cast<decltype(&cuTensorMapEncodeTiled)>(fn)(
               map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, const_cast<float2 *>(invT), dims, pitch, box, one,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
template <bool ADJ>
static bool sweep_page_map(int shape, CUtensorMap *map, const float2 *invT, int ny, int nx) {
    switch (shape) {
        case 0: return sweep_page_map<ADJ, 6, 6>(map, invT, ny, nx);
        case 1: return sweep_page_map<ADJ, 4, 4>(map, invT, ny, nx);
        case 2: return sweep_page_map<ADJ, 3, 4>(map, invT, ny, nx);
        case 3: return sweep_page_map<ADJ, 2, 2>(map, invT, ny, nx);
        default: return sweep_page_map<ADJ, 1, 1>(map, invT, ny, nx);
    }
}

template <bool ADJ>
static bool sweep_cluster_solve(const Coefs<float2> &co, const float2 *invT, const SrcView &src, int S, float2 *u,
                                int *err, int max_ctas, cudaStream_t st) {
    const SweepPlan g = sweep_plan<ADJ>(co.ny, S, max_ctas);
    if (g.cl == 0 || (reinterpret_cast<uintptr_t>(invT) & 15) != 0) return false;
    SweepClusterParams p;
    if (!sweep_page_map<ADJ>(g.shape, &p.pages, invT, co.ny, co.nx)) return false;
    p.err = err;
    p.timeout_ns = 10ull * 1000 * 1000 * 1000;
    p.co = co;
    p.invT = invT;
    p.u = u;
    p.src = src;
    p.ny = co.ny;
    p.nx = co.nx;
    p.S = S;
    p.n = co.ny - 2;
    p.RB = g.RB;
    p.stages = g.stages;
    const void *kernel = sweep_shape_kernel<ADJ>(g.shape);
    WUST_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSweepClusterSmem));
    cudaLaunchConfig_t cfg{};
    cfg.blockDim = dim3(CT);
    cfg.dynamicSmemBytes = g.smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = g.cl;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    void *args[] = {&p};
    for (int c = 0; c < g.clusters; c += g.per_launch) {
        cfg.gridDim = dim3(std::min(g.per_launch, g.clusters - c) * g.cl);
        p.s0 = c * 2 * kSweepShapes[g.shape][1];
        WUST_CUDA(cudaLaunchKernelExC(&cfg, kernel, args));
        ++g_kernel_launches;
    }
    WUST_LAUNCH_CHECK();
    return true;
}

void sweep_solve(const Coefs<float2> &co, const float2 *invT, const SrcView &src, int S, bool adjoint,
                 float2 *u, float2 *tmp, int *err, cudaStream_t st, int max_ctas) {
    SweepParams p;
    p.co = co;
    p.invT = invT;
    p.u = u;
    p.tmp = tmp;
    p.src = src;
    p.ny = co.ny;
    p.nx = co.nx;
    p.S = S;
    const int ny = co.ny, nx = co.nx;
    const size_t page = (size_t)ny * ny, fld = (size_t)ny * nx;
    WUST_CUDA(cudaMemsetAsync(u, 0, sizeof(float2) * fld * S, st));
    if (adjoint ? sweep_cluster_solve<true>(co, invT, src, S, u, err, max_ctas, st)
                : sweep_cluster_solve<false>(co, invT, src, S, u, err, max_ctas, st))
        return;
    WUST_CUDA(cudaMemsetAsync(tmp, 0, sizeof(float2) * (size_t)ny * S, st));   // border rows of tmp stay zero
    if (!adjoint) {
        for (int j = 1; j < nx; ++j) {
            p.j = j;
            launch_stencil<ST_L>(p, st);
            launch_gemm<false, 0, true>(invT + page * j, tmp, ny, u + (size_t)ny * j, fld, ny, S, st);
        }
        for (int j = nx - 2; j >= 0; --j) {
            p.j = j;
            launch_stencil<ST_U>(p, st);
            launch_gemm<false, 1, false>(invT + page * j, tmp, ny, u + (size_t)ny * j, fld, ny, S, st);
        }
    } else {
        for (int j = 1; j < nx; ++j) {
            p.j = j;
            launch_gemm<true, 0, false>(invT + page * (j - 1), u + (size_t)ny * (j - 1), fld, tmp, ny, ny, S, st);
            launch_stencil<ST_UH>(p, st);
        }
        for (int j = nx - 2; j >= 0; --j) {
            p.j = j;
            launch_stencil<ST_LH>(p, st);
            launch_gemm<true, 0, true>(invT + page * j, tmp, ny, u + (size_t)ny * j, fld, ny, S, st);
        }
    }
    WUST_LAUNCH_CHECK();
}

}  // namespace wust
