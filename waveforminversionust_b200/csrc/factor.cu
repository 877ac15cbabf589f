// Block-LU factorization of the nine-point Helmholtz operator: the Schur
// recursion of decompBlockLU (Runtime/solver/decompBlockLU.cu:337-368)
//
//     T_0 = D_0,  invT_j = inv(T_j[1:Ny-1, 1:Ny-1]),
//     T_{j+1} = D_{j+1} - L_j invT_j U_j,
//
// as ONE persistent cooperative kernel (one CTA per SM, bounded grid barrier
// between phases).  Each page is inverted by an unpivoted blocked
// Gauss-Jordan sweep over NB-wide blocks K:
//
//     P = inv(A_KK);  R_K. = P A_K.  (R_KK = P);  C_.K = A_.K (rows of K zeroed)
//     A'_rc = (r in K) ? R_rc : ((c in K) ? 0 : A_rc) - sum_u C_ru R_uc
//
// The reference pivots (cusolverDnCgetrf); the Schur blocks of this operator
// keep their largest entry of each row on the diagonal and have condition
// numbers of 10..700 at 4+ points per wavelength, so partial pivoting selects
// the diagonal and the unpivoted sweep computes the same inverse.  A zero or
// non-finite pivot is reported as WUST_ERR_SINGULAR_SCHUR_BLOCK.
//
// Work split: every CTA owns G x G output tiles of the padded page.  The
// working page is double-buffered in global memory (L2-resident, 2 x 2.6 MB
// at 552^2), so a Gauss-Jordan step reads panels of step k from one buffer
// and writes step k+1 into the other: one grid barrier per step.  Each CTA
// inverts the small NB x NB pivot block itself (no extra barrier) and forms
// the row-panel slice its tile needs.  The tridiagonal Schur product
// L_j invT_j U_j needs only the 3x3 neighbourhood of each invT_j entry
// (decompBlockLU.cu:65-152) and is fused into the page prologue through a
// shared-memory halo tile.
#include "common.cuh"
#include "kernels.cuh"

namespace wust {

constexpr int G = kFactorTile;   // output tile edge
constexpr int NB = 24;           // Gauss-Jordan block (divides G)
constexpr int GT = 256;          // threads: (tr, tc) in 16 x 16, rows tr + 16 i, cols tc + 16 j, i, j < 3
static_assert(G % NB == 0 && G == 48, "tile mapping assumes G = 48");

struct FactorParams {
    Coefs<float2> co;
    float2 *invT;          // [ny, ny, nx] column-major pages
    float2 *ws0, *ws1;     // n_pad x n_pad working pages (column-major), ping-pong
    unsigned *counter;     // monotonic barrier counter
    int *err;              // barrier timeout site
    int *status;           // [0]: 1 + first page with a bad pivot; [1]: pivot index
    int n, n_pad;
    int j0, j1;            // pages [j0, j1); page j0 - 1 (if any) is already in invT
    unsigned long long timeout_ns;
#ifdef WUST_FACTOR_PROFILE
    unsigned long long *prof;   // [0] prologue, [1] pivot block, [2] tile work, [3] barriers (block 0, ns)
#endif
};

#ifdef WUST_FACTOR_PROFILE
#define PROF_MARK(slot)                                                     \
    do {                                                                    \
        if (blockIdx.x == 0 && threadIdx.x == 0) {                          \
            const unsigned long long now_ = global_timer_ns();              \
            p.prof[slot] += now_ - prof_t;                                  \
            prof_t = now_;                                                  \
        }                                                                   \
    } while (0)
#else
#define PROF_MARK(slot) do { } while (0)
#endif

// Grid barrier on a monotonic counter: arrive with a release reduction, wait
// with acquire loads until the counter reaches epoch * nblocks.  The wait is
// bounded by timeout_ns (%globaltimer); on expiry the site is recorded in
// *err and every CTA leaves.
__device__ __forceinline__ bool grid_barrier(unsigned *counter, int *err, unsigned nblocks, unsigned &epoch,
                                             unsigned long long timeout_ns, int site) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        ++epoch;
        const unsigned target = epoch * nblocks;
        asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(counter), "r"(1u) : "memory");
        int ok = 1;
        WaitBudget budget;
        for (unsigned spin = 0;; ++spin) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
            if ((int)(v - target) >= 0) break;
            if (*(volatile int *)err) { ok = 0; break; }
            if ((spin & 31u) == 31u && budget.spent(timeout_ns)) {
                atomicCAS(err, 0, site);
                ok = 0;
                break;
            }
        }
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// Shared-memory carve-up: the NB x (NB+1) pivot inverse, the double-buffered
// pivot column (in a second NB x (NB+1) slot), then three NB x (G+1) panels;
// the prologue's (G+2) x (G+3) halo tile aliases the panels.
constexpr int kPivElems = NB * (NB + 1);
constexpr int kPanelElems = NB * (G + 1);
constexpr int kHaloElems = (G + 2) * (G + 3);
constexpr int kFactorSmemElems = 2 * kPivElems + (3 * kPanelElems > kHaloElems ? 3 * kPanelElems : kHaloElems);
constexpr size_t kFactorSmemBytes = sizeof(float2) * kFactorSmemElems;

// Own G x G tile entries (rows tr + 16 i, cols tc + 16 j) into registers.
__device__ __forceinline__ void load_tile(const float2 *cur, int np_, int r0, int c0, int tr, int tc, float2 (&a)[3][3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int jj = 0; jj < 3; ++jj) a[i][jj] = cur[(r0 + tr + 16 * i) + (size_t)np_ * (c0 + tc + 16 * jj)];
}

// Panels of one tile: Kr[u][cl] = A[k0+u, c0+cl]; Cc[u][rl] = A[r0+rl, k0+u]
// (zero on the rows of K).  All loads of a thread are issued before its
// shared-memory stores.
template <int NTH>
__device__ __forceinline__ void stage_panels(const float2 *cur, int np_, int k0, int r0, int c0, float2 (*Kr)[G + 1],
                                             float2 (*Cc)[G + 1], int t0) {
    constexpr int PER = (NB * G + NTH - 1) / NTH;
    float2 kv[PER], cv[PER];
#pragma unroll
    for (int m = 0; m < PER; ++m) {
        const int e = t0 + m * NTH;
        if (e < NB * G) {
            const int u = e % NB, cl = e / NB;
            kv[m] = cur[(k0 + u) + (size_t)np_ * (c0 + cl)];
            const int rl = e % G, uu = e / G, r = r0 + rl;
            cv[m] = (r >= k0 && r < k0 + NB) ? make_float2(0.f, 0.f) : cur[r + (size_t)np_ * (k0 + uu)];
        }
    }
#pragma unroll
    for (int m = 0; m < PER; ++m) {
        const int e = t0 + m * NTH;
        if (e < NB * G) {
            Kr[e % NB][e / NB] = kv[m];
            Cc[e / G][e % G] = cv[m];
        }
    }
}

// 1/z as conj(z) / |z|^2 with the correctly rounded reciprocal intrinsic
// (pivot magnitudes of this operator are O(1/h^2), far from FP32 overflow).
__device__ __forceinline__ float2 crecip_fast(float2 z) {
    const float inv = __frcp_rn(fmaf(z.x, z.x, z.y * z.y));
    return make_float2(z.x * inv, -z.y * inv);
}

// Unpivoted Gauss-Jordan inverse of the NB x NB pivot block on warps 0-3:
// lane r holds row r, warp w holds columns [6w, 6w + 6).  Per pivot q the
// owner warp publishes column q through shared memory (one 128-thread named
// barrier per pivot, double-buffered), the pivot row travels by warp
// shuffles.  Result -> Pa[row][col].
__device__ __forceinline__ void invert_pivot_block(const float2 *cur, int np_, int k0, float2 (*Pa)[NB + 1],
                                                   float2 (*fcol)[NB], int *status, int page, bool report) {
    static_assert(NB == 24, "4 warps x 6 columns");
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int col0 = 6 * w;
    float2 a[6];
#pragma unroll
    for (int c = 0; c < 6; ++c)
        a[c] = (lane < NB) ? cur[(k0 + lane) + (size_t)np_ * (k0 + col0 + c)] : make_float2(0.f, 0.f);
#pragma unroll
    for (int q = 0; q < NB; ++q) {
        float2 *fc = fcol[q & 1];
        if (w == q / 6 && lane < NB) fc[lane] = a[q % 6];
        asm volatile("bar.sync 1, 128;" ::: "memory");
        const float2 piv = fc[q];
        if (report && threadIdx.x == 0) {
            const float mag = fabsf(piv.x) + fabsf(piv.y);
            if (!(mag > 0.f && isfinite(mag)) && atomicCAS(&status[0], 0, page + 1) == 0) status[1] = k0 + q;
        }
        const float2 ip = crecip_fast(piv);
        const float2 f = (lane < NB) ? fc[lane] : make_float2(0.f, 0.f);
        const float2 mf = make_float2(-f.x, -f.y);
#pragma unroll
        for (int c = 0; c < 6; ++c) {
            float2 pr;
            pr.x = __shfl_sync(0xffffffffu, a[c].x, q);
            pr.y = __shfl_sync(0xffffffffu, a[c].y, q);
            pr = cmul(pr, ip);
            float2 nv;
            if (col0 + c == q) nv = (lane == q) ? ip : cmul(mf, ip);
            else if (lane == q) nv = pr;
            else {
                nv = a[c];
                cfma(nv, mf, pr);
            }
            a[c] = nv;
        }
    }
#pragma unroll
    for (int c = 0; c < 6; ++c)
        if (lane < NB) Pa[lane][col0 + c] = a[c];
}

__global__ void __launch_bounds__(GT, 1) factor_kernel(FactorParams p) {
    extern __shared__ float2 smem[];
    float2(*Pa)[NB + 1] = reinterpret_cast<float2(*)[NB + 1]>(smem);
    float2(*fcol)[NB] = reinterpret_cast<float2(*)[NB]>(smem + kPivElems);          // pivot column, double-buffered
    float2(*Kr)[G + 1] = reinterpret_cast<float2(*)[G + 1]>(smem + 2 * kPivElems);   // A[K, tile cols]
    float2(*Rr)[G + 1] = Kr + NB;                                                   // R[u][tile col]
    float2(*Cc)[G + 1] = Kr + 2 * NB;                                               // C[tile row][u], as Cc[u][row]
    float2(*Xs)[G + 3] = reinterpret_cast<float2(*)[G + 3]>(smem + 2 * kPivElems);   // prologue halo, Xs[col][row]

    const int ny = p.co.ny, n = p.n, np_ = p.n_pad;
    const int nt = np_ / G, nsteps = np_ / NB;
    const unsigned nblocks = gridDim.x;
    const int tid = threadIdx.x, tr = tid % 16, tc = tid / 16;
    const size_t page_sz = (size_t)ny * ny;
    unsigned epoch = 0;
    int site = 0;
#ifdef WUST_FACTOR_PROFILE
    unsigned long long prof_t = global_timer_ns();
#endif

    // Border rows/columns of every page are zero (decompBlockLU.cu:284-288).
    const size_t gstride = (size_t)gridDim.x * blockDim.x;
    for (size_t idx = (size_t)blockIdx.x * blockDim.x + tid; idx < (size_t)(p.j1 - p.j0) * 4 * ny; idx += gstride) {
        const size_t page = p.j0 + idx / (4 * (size_t)ny);
        const int rem = (int)(idx % (4 * (size_t)ny));
        const int which = rem / ny, k = rem % ny;
        const size_t off = which == 0 ? (size_t)ny * k
                         : which == 1 ? (size_t)(ny - 1) + (size_t)ny * k
                         : which == 2 ? (size_t)k
                                      : (size_t)k + (size_t)ny * (ny - 1);
        p.invT[page * page_sz + off] = make_float2(0.f, 0.f);
    }

    for (int j = p.j0; j < p.j1; ++j) {
        // ---- prologue: ws0 = T_j interior (identity padding) ----------------
        const float2 *X = p.invT + (size_t)(j > 0 ? j - 1 : 0) * page_sz;
        for (int t = blockIdx.x; t < nt * nt; t += gridDim.x) {
            const int r0 = (t % nt) * G, c0 = (t / nt) * G;     // ws coordinates
            if (j > 0) {
                for (int e = tid; e < (G + 2) * (G + 2); e += GT) {
                    const int rr = e % (G + 2), cc = e / (G + 2);
                    const int R = r0 + rr, C = c0 + cc;          // grid indices of invT_{j-1}
                    Xs[cc][rr] = (R < ny && C < ny) ? X[R + (size_t)ny * C] : make_float2(0.f, 0.f);
                }
            }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < 3; ++i) {
#pragma unroll
                for (int jj = 0; jj < 3; ++jj) {
                    const int rl = tr + 16 * i, cl = tc + 16 * jj;
                    const int r = r0 + rl, c = c0 + cl;
                    float2 v;
                    if (r >= n || c >= n) {
                        v = make_float2(r == c ? 1.f : 0.f, 0.f);
                    } else {
                        const int R = r + 1, C = c + 1;          // grid row/col in [1, ny-2]
                        v = make_float2(0.f, 0.f);
                        if (R == C) v = p.co.dd(R, j);
                        else if (R == C + 1) v = p.co.dl(C, j);
                        else if (R + 1 == C) v = p.co.du(R, j);
                        if (j > 0) {
                            const int jm = j - 1;
                            const float2 udc = p.co.ud(C, jm), uuc = p.co.uu(C - 1, jm), ulc = p.co.ul(C, jm);
                            float2 right[3];
#pragma unroll
                            for (int d = 0; d < 3; ++d) {            // grid rows R-1, R, R+1
                                float2 acc = cmul(Xs[cl + 1][rl + d], udc);
                                cfma(acc, Xs[cl][rl + d], uuc);
                                cfma(acc, Xs[cl + 2][rl + d], ulc);
                                right[d] = acc;
                            }
                            float2 lr = cmul(p.co.ld(R, jm), right[1]);
                            cfma(lr, p.co.ll(R - 1, jm), right[0]);
                            cfma(lr, p.co.lu(R, jm), right[2]);
                            v = csub(v, lr);
                        }
                    }
                    p.ws0[r + (size_t)np_ * c] = v;
                }
            }
            __syncthreads();
        }
        PROF_MARK(0);
        if (!grid_barrier(p.counter, p.err, nblocks, epoch, p.timeout_ns, ++site)) return;
        PROF_MARK(3);

        // ---- blocked Gauss-Jordan inverse -----------------------------------
        for (int kb = 0; kb < nsteps; ++kb) {
            const float2 *cur = (kb & 1) ? p.ws1 : p.ws0;
            float2 *nxt = (kb & 1) ? p.ws0 : p.ws1;
            const int k0 = kb * NB;
            const bool last = (kb == nsteps - 1);

            // Warps 0-3 invert the pivot block A_KK in registers while warps 4-7
            // stage this CTA's first tile panels; all threads prefetch their
            // own tile entries first so every load is in flight at once.
            const int warp = tid >> 5;
            int t = blockIdx.x;
            float2 a[3][3];
            if (t < nt * nt) load_tile(cur, np_, (t % nt) * G, (t / nt) * G, tr, tc, a);
            if (warp < 4) {
                invert_pivot_block(cur, np_, k0, Pa, fcol, p.status, j, blockIdx.x == 0);
            } else if (t < nt * nt) {
                stage_panels<GT - 128>(cur, np_, k0, (t % nt) * G, (t / nt) * G, Kr, Cc, tid - 128);
            }
            __syncthreads();
            PROF_MARK(1);
            while (t < nt * nt) {
                const int I = t % nt, J = t / nt;
                const int r0 = I * G, c0 = J * G;
                // row panel slice R[u][cl] = (P A[K, .])_{u, c0+cl}; R = P on the columns of K
                if (tid < 8 * NB) {
                    const int u = tid % NB, cb = tid / NB;
                    float2 acc[G / 8];
#pragma unroll
                    for (int m = 0; m < G / 8; ++m) acc[m] = make_float2(0.f, 0.f);
#pragma unroll 4
                    for (int v = 0; v < NB; ++v) {
                        const float2 pv = Pa[u][v];
#pragma unroll
                        for (int m = 0; m < G / 8; ++m) cfma(acc[m], pv, Kr[v][cb + 8 * m]);
                    }
#pragma unroll
                    for (int m = 0; m < G / 8; ++m) {
                        const int cl = cb + 8 * m, c = c0 + cl;
                        Rr[u][cl] = (c >= k0 && c < k0 + NB) ? Pa[u][c - k0] : acc[m];
                    }
                }
                __syncthreads();
#pragma unroll
                for (int i = 0; i < 3; ++i) {
#pragma unroll
                    for (int jj = 0; jj < 3; ++jj) {
                        const int rl = tr + 16 * i, cl = tc + 16 * jj;
                        const int r = r0 + rl, c = c0 + cl;
                        const bool rk = (r >= k0 && r < k0 + NB), ck = (c >= k0 && c < k0 + NB);
                        float2 v = rk ? Rr[r - k0][cl] : (ck ? make_float2(0.f, 0.f) : a[i][jj]);
                        float2 dot = make_float2(0.f, 0.f);
#pragma unroll 8
                        for (int u = 0; u < NB; ++u) cfma(dot, Cc[u][rl], Rr[u][cl]);
                        v = csub(v, dot);
                        nxt[r + (size_t)np_ * c] = v;
                        if (last && r < n && c < n)
                            p.invT[(size_t)j * page_sz + (size_t)(r + 1) + (size_t)ny * (c + 1)] = v;
                    }
                }
                __syncthreads();
                t += gridDim.x;
                if (t < nt * nt) {          // more tiles than CTAs: stage the next one with all threads
                    load_tile(cur, np_, (t % nt) * G, (t / nt) * G, tr, tc, a);
                    stage_panels<GT>(cur, np_, k0, (t % nt) * G, (t / nt) * G, Kr, Cc, tid);
                    __syncthreads();
                }
            }
            PROF_MARK(2);
            if (!grid_barrier(p.counter, p.err, nblocks, epoch, p.timeout_ns, ++site)) return;
            PROF_MARK(3);
        }
    }
}

// ---------------------------------------------------------------------------
// Dataflow variant of the same elimination, for pages whose G x G tiles fit
// the grid one per CTA.  The kernel above spends its step (12.7 us, at every
// page size) on a chain of latencies: the grid barrier, the reload of tile
// and panels, the pivot block inverted by every CTA, the tile update.  Here
//   * the tile stays in registers for the whole page;
//   * after its update of step k a CTA publishes the rows and columns that
//     step k + 1 takes as panels, and the owner of the next diagonal block
//     publishes its inverse, as 16-byte words {re, tag, im, tag}: a reader
//     polls the data words themselves until their tag is the step's, so
//     there is no fence, no flag and no barrier between producer and reader
//     (each 8-byte half carries its own tag and is written at once).  Every
//     step has its own words, so nothing is overwritten before the page's
//     closing grid barrier;
//   * four extra warps (8 .. 11) hold no tile: in the CTA that owns the next
//     diagonal block they update that block alone and invert it while the
//     other warps update the tile.
// The remaining chain per step is the row panel, the diagonal block's update
// and its inverse, and one L2 round trip where the next block is another
// CTA's.  Blocks of 16 make it shortest (measured at 552^2, us per page: 24
// wide 161, 16 wide 138): an inverse costs about as many clocks per pivot at
// every width, wider blocks add to the panel and to the update, narrower
// ones to the round trips of the CTAs off the diagonal.
// ---------------------------------------------------------------------------
constexpr int FB = kFlowBlock;           // Gauss-Jordan block
constexpr int kFlowTileThreads = 256;    // warps 0-7: tile and panels, (tr, tc) as above
constexpr int kPivotThreads = 128;       // warps 8-11: pivot block
constexpr int FT = kFlowTileThreads + kPivotThreads;
static_assert(FB == 16 && G % FB == 0, "pivot warps: 4 x 4 rows, a column per half-warp lane");

struct FlowParams {
    Coefs<float2> co;
    float2 *invT;
    ulonglong2 *rowp;      // [step][column][FB]: rows of the pivot block
    ulonglong2 *colp;      // [step][FB][row]: columns of the pivot block
    ulonglong2 *pivp;      // [step][FB * FB]: inverse of the pivot block, column fastest
    unsigned *counter;
    int *err;
    unsigned *status;      // 0, or flow_bad_pivot of the first singular block
    int n, n_pad, nsteps, j0, j1;
    unsigned long long timeout_ns;
};

// page * kFlowPivots + pivot, such that the first one is the largest
constexpr unsigned kFlowPivots = kFlowMaxTiles * G;
__host__ __device__ constexpr unsigned flow_bad_pivot(int page, int pivot) {
    return 0xffffffffu - ((unsigned)page * kFlowPivots + (unsigned)pivot);
}

constexpr int kPStride = FB + 2;         // rows start on 16 bytes: pairs of entries in one load
constexpr int kCStride = G + 2;

struct __align__(16) FlowSmem {
    float2 P[2][FB][kPStride];     // inverse of the pivot block, by step parity
    float4 nrow[FB / 2][FB];       // scaled pivot rows of the inversion
    float2 S[FB][FB];              // the block being inverted
    float2 D[2][FB][FB];           // the next diagonal block before this step's update, by step parity
    float2 cf[9][G];               // ld ll lu dd dl du of this tile's rows, ud uu ul of its columns
    union {
        struct {
            float2 Kr[G][kPStride];    // pivot rows, [tile column][u]
            float2 Cc[FB][kCStride];   // pivot columns, [u][tile row], zero on the pivot rows
            float2 Rr[FB][G + 1];      // P Kr, [u][tile column]
        } s[2];
        float2 Xs[G + 2][G + 3];   // prologue halo, Xs[col][row]
    };
};
constexpr size_t kFlowSmemBytes = sizeof(FlowSmem);

__device__ __forceinline__ void flow_put(ulonglong2 *w, float2 v, unsigned tag) {
    const unsigned long long hi = (unsigned long long)tag << 32;
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(w), "l"(hi | __float_as_uint(v.x)),
                 "l"(hi | __float_as_uint(v.y)) : "memory");
}
__device__ __forceinline__ ulonglong2 flow_peek(const ulonglong2 *w) {
    ulonglong2 v;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(w) : "memory");
    return v;
}
__device__ __forceinline__ bool flow_ready(const ulonglong2 &v, unsigned tag) {
    return (unsigned)(v.x >> 32) == tag && (unsigned)(v.y >> 32) == tag;
}
__device__ __forceinline__ float2 flow_value(const ulonglong2 &v) {
    return make_float2(__uint_as_float((unsigned)v.x), __uint_as_float((unsigned)v.y));
}

// COUNT words per thread, all in flight at once; those that have not arrived
// are polled again.  false: gave up (timeout, or another CTA did).
template <int COUNT, typename Word, typename Store>
__device__ __forceinline__ bool flow_take(const FlowParams &p, unsigned tag, int site, Word word, Store store) {
    ulonglong2 v[COUNT];
#pragma unroll
    for (int m = 0; m < COUNT; ++m) v[m] = flow_peek(word(m));
    unsigned long long t0 = 0;
#pragma unroll
    for (int m = 0; m < COUNT; ++m) {
        ulonglong2 x = v[m];
        for (unsigned spin = 0; !flow_ready(x, tag); ++spin) {
            if ((spin & 63u) == 63u) {
                const unsigned long long now = global_timer_ns();
                if (t0 == 0) t0 = now;
                if (now - t0 > p.timeout_ns) atomicCAS(p.err, 0, site);
                if (*(volatile int *)p.err) return false;
            }
            x = flow_peek(word(m));
        }
        store(m, flow_value(x));
    }
    return true;
}

// Inverse w of the 2 x 2 pivot [e1; e2] in closed form; returns |det| (1-norm).
// 1 / det = conj(det) / |det|^2 at a scale of 2^-e, so that the range of
// pivots is that of one |pivot|^2; the reciprocal of a number in [1, 8] by
// the hardware's approximation and one Newton step.
__device__ __forceinline__ float invert_pair(float4 e1, float4 e2, float2 &w11, float2 &w12, float2 &w21, float2 &w22) {
    const float2 p11 = make_float2(e1.x, e1.y), p12 = make_float2(e1.z, e1.w);
    const float2 p21 = make_float2(e2.x, e2.y), p22 = make_float2(e2.z, e2.w);
    float2 det = cmul(p11, p22);
    cfma(det, make_float2(-p12.x, -p12.y), p21);
    const unsigned ex = max(__float_as_uint(det.x) & 0x7f800000u, __float_as_uint(det.y) & 0x7f800000u);
    const float sc = __uint_as_float(0x7f000000u - ex);
    const float dx = det.x * sc, dy = det.y * sc;
    const float m2 = fmaf(dx, dx, dy * dy);
    float inv;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(m2));
    inv = fmaf(inv, fmaf(-m2, inv, 1.f), inv) * sc;
    const float2 id = make_float2(dx * inv, -dy * inv);
    w11 = cmul(id, p22);
    w12 = cmul(id, make_float2(-p12.x, -p12.y));
    w21 = cmul(id, make_float2(-p21.x, -p21.y));
    w22 = cmul(id, p11);
    return fabsf(det.x) + fabsf(det.y);
}

// Unpivoted Gauss-Jordan inverse of an FB x FB block on the four pivot warps,
// two pivots at a time: warp w holds rows [4w, 4w + 4), a lane column c of
// rows pr and pr + 1.  The warp that owns a pair's rows inverts the 2 x 2
// pivot, scales its two rows, publishes them and goes on to its next pair at
// once; the others apply them when they come (one named barrier per pair, on
// which the owner only arrives), so that the chain of latencies runs inside
// one warp and crosses over three times in all.  The entries of the pivot
// columns and rows reach a warp's lanes through shared memory of its own (a
// shuffle costs 10 cycles of a single warp here, a broadcast read two).  The
// loop over the owners is not unrolled: copies of its body would push the
// tile's code out of the instruction caches.
__device__ __forceinline__ void invert_block_pairs(float2 (&a)[2], int pr, int c, float4 (*nrow)[FB], float2 (*S)[FB],
                                                   float2 (*P)[kPStride], unsigned *status, int page, int k0) {
    const int w = pr >> 2;
    int bad = -1;
    float4 f0, f1;                                // columns q, q + 1 of rows pr, pr + 1
    auto stage = [&](int q) {
        __syncwarp();
        S[pr][c] = a[0];
        S[pr + 1][c] = a[1];
        __syncwarp();
        f0 = *reinterpret_cast<const float4 *>(&S[pr][q]);
        f1 = *reinterpret_cast<const float4 *>(&S[pr + 1][q]);
        if (c == q || c == q + 1) a[0] = a[1] = make_float2(0.f, 0.f);
    };
    auto apply = [&](float2 n1, float2 n2) {
        cfma(a[0], make_float2(-f0.x, -f0.y), n1);
        cfma(a[1], make_float2(-f1.x, -f1.y), n1);
        cfma(a[0], make_float2(-f0.z, -f0.w), n2);
        cfma(a[1], make_float2(-f1.z, -f1.w), n2);
    };
#pragma unroll 1
    for (int ow = 0; ow < 4; ++ow) {
        if (w == ow) {
#pragma unroll
            for (int i = 0; i < 4; i += 2) {
                const int q = 4 * ow + i;
                stage(q);
                const float4 e1 = *reinterpret_cast<const float4 *>(&S[q][q]);
                const float4 e2 = *reinterpret_cast<const float4 *>(&S[q + 1][q]);
                float2 r1 = S[q][c], r2 = S[q + 1][c];
                float2 w11, w12, w21, w22;
                const float det = invert_pair(e1, e2, w11, w12, w21, w22);
                // the pivot columns turn into those of the identity times w
                if (c == q) { r1 = make_float2(1.f, 0.f); r2 = make_float2(0.f, 0.f); }
                if (c == q + 1) { r1 = make_float2(0.f, 0.f); r2 = make_float2(1.f, 0.f); }
                float2 n1 = cmul(w11, r1), n2 = cmul(w21, r1);
                cfma(n1, w12, r2);
                cfma(n2, w22, r2);
                if (pr & 2) nrow[q >> 1][c] = make_float4(n1.x, n1.y, n2.x, n2.y);
                __syncwarp();
                asm volatile("bar.arrive %0, 128;" ::"r"(3 + (q >> 1)) : "memory");
                const float piv = fabsf(e1.x) + fabsf(e1.y);
                if (bad < 0 && !(piv > 0.f && isfinite(piv))) bad = q;
                if (bad < 0 && !(det > 0.f && isfinite(det))) bad = q + 1;
                apply(n1, n2);
                if (pr == q) {
                    a[0] = n1;
                    a[1] = n2;
                }
            }
        } else {
#pragma unroll 1
            for (int q = 4 * ow; q < 4 * ow + 4; q += 2) {
                stage(q);
                asm volatile("bar.sync %0, 128;" ::"r"(3 + (q >> 1)) : "memory");
                const float4 nn = nrow[q >> 1][c];
                apply(make_float2(nn.x, nn.y), make_float2(nn.z, nn.w));
            }
        }
    }
    // the first bad pivot of the first bad page: what follows it is not finite, and is found bad too
    if (bad >= 0 && c == 0) atomicMax(status, flow_bad_pivot(page, k0 + bad));
    P[pr][c] = a[0];
    P[pr + 1][c] = a[1];
}

__global__ void __launch_bounds__(FT, 1) factor_flow_kernel(FlowParams p) {
    extern __shared__ __align__(16) unsigned char flow_smem[];
    FlowSmem &sm = *reinterpret_cast<FlowSmem *>(flow_smem);
    const int ny = p.co.ny, n = p.n, np_ = p.n_pad;
    const int nt = np_ / G;
    const int tid = threadIdx.x;
    const bool tile_warp = tid < kFlowTileThreads;
    const int tr = tid % 16, tc = (tid / 16) % 16;
    const int I = blockIdx.x % nt, J = blockIdx.x / nt, r0 = I * G, c0 = J * G;
    const size_t page_sz = (size_t)ny * ny;
    unsigned epoch = 0;

    // Border rows/columns of every page are zero (decompBlockLU.cu:284-288).
    for (size_t idx = (size_t)blockIdx.x * FT + tid; idx < (size_t)(p.j1 - p.j0) * 4 * ny; idx += (size_t)gridDim.x * FT) {
        const size_t page = p.j0 + idx / (4 * (size_t)ny);
        const int rem = (int)(idx % (4 * (size_t)ny));
        const int which = rem / ny, k = rem % ny;
        const size_t off = which == 0 ? (size_t)ny * k
                         : which == 1 ? (size_t)(ny - 1) + (size_t)ny * k
                         : which == 2 ? (size_t)k
                                      : (size_t)k + (size_t)ny * (ny - 1);
        p.invT[page * page_sz + off] = make_float2(0.f, 0.f);
    }

    // The coefficients that the tile of T_j takes, on their way to shared
    // memory while page j - 1 is inverted.
    auto fetch_coefs = [&](int j) {
        for (int e = tid; e < 9 * G; e += FT) {
            const int which = e / G, l = e % G, jm = j - 1;
            const int g = (which < 6 ? r0 : c0) + l + 1;               // grid row / column
            if (g > n || (jm < 0 && which != 3 && which != 4 && which != 5)) continue;
            const float2 *src;
            switch (which) {
                case 0: src = &p.co.Ld[g + (size_t)ny * jm]; break;
                case 1: src = &p.co.Ll[g - 1 + (size_t)(ny - 1) * jm]; break;
                case 2: src = &p.co.Lu[g + (size_t)(ny - 1) * jm]; break;
                case 3: src = &p.co.Dd[g + (size_t)ny * j]; break;
                case 4: src = &p.co.Dl[g - 1 + (size_t)(ny - 1) * j]; break;
                case 5: src = &p.co.Du[g + (size_t)(ny - 1) * j]; break;
                case 6: src = &p.co.Ud[g + (size_t)ny * jm]; break;
                case 7: src = &p.co.Uu[g - 1 + (size_t)(ny - 1) * jm]; break;
                default: src = &p.co.Ul[g + (size_t)(ny - 1) * jm]; break;
            }
            const unsigned dst = (unsigned)__cvta_generic_to_shared(&sm.cf[which][l]);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    // This CTA's words of the panels of step k (pivot block k0 .. k0 + FB - 1),
    // and the diagonal block of step k + 1 for the pivot warps.  A tile on the
    // diagonal that holds the block itself needs nobody's panels but its own.
    float2 a[3][3];
    auto publish = [&](int k, unsigned tag) {
        const int k0 = k * FB, kd = k0 + FB;
        const bool rows = k0 >= r0 && k0 < r0 + G, cols = k0 >= c0 && k0 < c0 + G;
        const bool next = I == J && k + 1 < p.nsteps && kd >= r0 && kd < r0 + G;
        if (!rows && !cols && !next) return;
        ulonglong2 *rw = p.rowp + (size_t)k * np_ * FB, *cw = p.colp + (size_t)k * np_ * FB;
        auto &s = sm.s[k & 1];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int jj = 0; jj < 3; ++jj) {
                const int rl = tr + 16 * i, cl = tc + 16 * jj, r = r0 + rl, c = c0 + cl;
                const bool rk = r >= k0 && r < kd, ck = c >= k0 && c < kd;
                if (rk) flow_put(rw + (size_t)c * FB + (r - k0), a[i][jj], tag);
                if (ck) flow_put(cw + (size_t)(c - k0) * np_ + r, a[i][jj], tag);
                if (rows && cols) {
                    if (rk) s.Kr[cl][r - k0] = a[i][jj];
                    if (ck) s.Cc[c - k0][rl] = rk ? make_float2(0.f, 0.f) : a[i][jj];
                }
                if (next && r >= kd && r < kd + FB && c >= kd && c < kd + FB) sm.D[(k + 1) & 1][r - kd][c - kd] = a[i][jj];
            }
    };
    // The pivot warps' part of step k: the inverse of the (updated) diagonal
    // block d into P and out to the other CTAs.
    const int pl = tid - kFlowTileThreads, pr = 2 * (pl >> 4), pc = pl & 15;     // rows pr, pr + 1, column pc
    auto pivot = [&](float2 (&d)[2], int k, unsigned tag, int page) {
        invert_block_pairs(d, pr, pc, sm.nrow, sm.S, sm.P[k & 1], p.status, page, k * FB);
        ulonglong2 *pw = p.pivp + (size_t)k * FB * FB + (size_t)pr * FB + pc;
        flow_put(pw, d[0], tag);
        flow_put(pw + FB, d[1], tag);
    };

    fetch_coefs(p.j0);
    for (int j = p.j0; j < p.j1; ++j) {
        const unsigned tag0 = 1u + (unsigned)(j - p.j0) * (unsigned)p.nsteps;
        // ---- prologue: the tile of T_j (identity padding) --------------------
        if (j > 0) {
            const float2 *X = p.invT + (size_t)(j - 1) * page_sz;
            for (int e = tid; e < (G + 2) * (G + 2); e += FT) {
                const int rr = e % (G + 2), cc = e / (G + 2);
                const int R = r0 + rr, C = c0 + cc;              // grid indices of invT_{j-1}
                sm.Xs[cc][rr] = (R < ny && C < ny) ? __ldcg(X + R + (size_t)ny * C) : make_float2(0.f, 0.f);
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        if (tile_warp) {
#pragma unroll
            for (int i = 0; i < 3; ++i) {
#pragma unroll
                for (int jj = 0; jj < 3; ++jj) {
                    const int rl = tr + 16 * i, cl = tc + 16 * jj;
                    const int r = r0 + rl, c = c0 + cl;
                    float2 v;
                    if (r >= n || c >= n) {
                        v = make_float2(r == c ? 1.f : 0.f, 0.f);
                    } else {
                        v = r == c ? sm.cf[3][rl] : r == c + 1 ? sm.cf[4][rl] : r + 1 == c ? sm.cf[5][rl]
                                                                                          : make_float2(0.f, 0.f);
                        if (j > 0) {
                            const float2 udc = sm.cf[6][cl], uuc = sm.cf[7][cl], ulc = sm.cf[8][cl];
                            float2 right[3];
#pragma unroll
                            for (int d = 0; d < 3; ++d) {        // grid rows R-1, R, R+1
                                float2 acc = cmul(sm.Xs[cl + 1][rl + d], udc);
                                cfma(acc, sm.Xs[cl][rl + d], uuc);
                                cfma(acc, sm.Xs[cl + 2][rl + d], ulc);
                                right[d] = acc;
                            }
                            float2 lr = cmul(sm.cf[0][rl], right[1]);
                            cfma(lr, sm.cf[1][rl], right[0]);
                            cfma(lr, sm.cf[2][rl], right[2]);
                            v = csub(v, lr);
                        }
                    }
                    a[i][jj] = v;
                    if (I == 0 && J == 0 && r < FB && c < FB) sm.D[0][r][c] = v;
                }
            }
        }
        __syncthreads();                          // the panels of step 0 overwrite the halo
        if (tile_warp) publish(0, tag0);
        if (j + 1 < p.j1) fetch_coefs(j + 1);
        if (!tile_warp && blockIdx.x == 0) {
            float2 d[2] = {sm.D[0][pr][pc], sm.D[0][pr + 1][pc]};
            pivot(d, 0, tag0, j);
        }

        // ---- blocked Gauss-Jordan inverse ------------------------------------
        for (int k = 0; k < p.nsteps; ++k) {
            const unsigned tag = tag0 + (unsigned)k;
            const int k0 = k * FB, par = k & 1, dk = k0 / G;
            auto &s = sm.s[par];
            bool ok = true;
            if (!(I == J && I == dk)) {
                if (tile_warp) {
                    constexpr int PER = FB * G / kFlowTileThreads;
                    const ulonglong2 *rw = p.rowp + ((size_t)k * np_ + c0) * FB;
                    const ulonglong2 *cw = p.colp + (size_t)k * np_ * FB + r0;
                    ok = flow_take<PER>(
                        p, tag, 5001, [&](int m) { return rw + tid + m * kFlowTileThreads; },
                        [&](int m, float2 v) {
                            const int e = tid + m * kFlowTileThreads;
                            s.Kr[e / FB][e % FB] = v;
                        });
                    ok = ok && flow_take<PER>(
                        p, tag, 5002,
                        [&](int m) {
                            const int e = tid + m * kFlowTileThreads;
                            return cw + (size_t)(e / G) * np_ + e % G;
                        },
                        [&](int m, float2 v) {
                            const int e = tid + m * kFlowTileThreads, r = r0 + e % G;
                            s.Cc[e / G][e % G] = (r >= k0 && r < k0 + FB) ? make_float2(0.f, 0.f) : v;
                        });
                } else {
                    const ulonglong2 *pw = p.pivp + (size_t)k * FB * FB;
                    ok = flow_take<FB * FB / kPivotThreads>(
                        p, tag, 5003, [&](int m) { return pw + pl + m * kPivotThreads; },
                        [&](int m, float2 v) {
                            const int e = pl + m * kPivotThreads;
                            sm.P[par][e / FB][e % FB] = v;
                        });
                }
            }
            if (__syncthreads_or(!ok)) {
                asm volatile("cp.async.wait_all;" ::: "memory");           // the next page's coefficients
                return;
            }
            // row panel slice R[u][cl] = (P A[K, .])_{u, c0+cl}; R = P on the columns of K.  8 x 24 threads, 2 x 2
            // entries each: shared memory delivers 128 bytes per clock to the registers, broadcast or not, which
            // bounds narrower splits; fewer threads with more entries are bound by the issue of their few warps
            if (tid < 192) {
                const int ub = tid % 8, cb = tid / 8;
                float2 acc[2][2];
#pragma unroll
                for (int i = 0; i < 2; ++i) acc[i][0] = acc[i][1] = make_float2(0.f, 0.f);
#pragma unroll 4
                for (int v = 0; v < FB; v += 2) {
                    float4 pv[2], kv[2];
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        pv[i] = *reinterpret_cast<const float4 *>(&sm.P[par][ub + 8 * i][v]);
                        kv[i] = *reinterpret_cast<const float4 *>(&s.Kr[cb + 24 * i][v]);
                    }
#pragma unroll
                    for (int i = 0; i < 2; ++i)
#pragma unroll
                        for (int m = 0; m < 2; ++m) cfma(acc[i][m], make_float2(pv[i].x, pv[i].y), make_float2(kv[m].x, kv[m].y));
#pragma unroll
                    for (int i = 0; i < 2; ++i)
#pragma unroll
                        for (int m = 0; m < 2; ++m) cfma(acc[i][m], make_float2(pv[i].z, pv[i].w), make_float2(kv[m].z, kv[m].w));
                }
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    const int cl = cb + 24 * m, c = c0 + cl;
                    const bool ck = c >= k0 && c < k0 + FB;
#pragma unroll
                    for (int i = 0; i < 2; ++i) s.Rr[ub + 8 * i][cl] = ck ? sm.P[par][ub + 8 * i][c - k0] : acc[i][m];
                }
            }
            __syncthreads();
            const int kn = k0 + FB;
            const bool next = k + 1 < p.nsteps && I == J && kn >= r0 && kn < r0 + G;
            if (tile_warp) {
                // the page's chain goes through the next diagonal block: its update first, and its inverse too
                // where the step after next leaves this tile (its panels are not on the chain then)
                if (next) asm volatile("bar.sync 2, 384;" ::: "memory");
                float2 dot[3][3];
#pragma unroll
                for (int i = 0; i < 3; ++i)
#pragma unroll
                    for (int jj = 0; jj < 3; ++jj) dot[i][jj] = make_float2(0.f, 0.f);
#pragma unroll 4
                for (int u = 0; u < FB; ++u) {
                    float2 cv[3], rv[3];
#pragma unroll
                    for (int i = 0; i < 3; ++i) cv[i] = s.Cc[u][tr + 16 * i];
#pragma unroll
                    for (int jj = 0; jj < 3; ++jj) rv[jj] = s.Rr[u][tc + 16 * jj];
#pragma unroll
                    for (int i = 0; i < 3; ++i)
#pragma unroll
                        for (int jj = 0; jj < 3; ++jj) cfma(dot[i][jj], cv[i], rv[jj]);
                }
#pragma unroll
                for (int i = 0; i < 3; ++i)
#pragma unroll
                    for (int jj = 0; jj < 3; ++jj) {
                        const int r = r0 + tr + 16 * i, cl = tc + 16 * jj, c = c0 + cl;
                        const bool rk = r >= k0 && r < kn, ck = c >= k0 && c < kn;
                        const float2 v = rk ? s.Rr[r - k0][cl] : ck ? make_float2(0.f, 0.f) : a[i][jj];
                        a[i][jj] = csub(v, dot[i][jj]);
                    }
                if (k + 1 < p.nsteps) publish(k + 1, tag + 1u);
            } else if (next) {
                // the next diagonal block (outside the rows and columns of K): its update, then its inverse
                const int off = kn - r0;
                float2 d[2], dot[2];
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    d[m] = sm.D[par ^ 1][pr + m][pc];
                    dot[m] = make_float2(0.f, 0.f);
                }
#pragma unroll 8
                for (int u = 0; u < FB; ++u) {
                    const float2 rv = s.Rr[u][off + pc];
                    const float4 cv = *reinterpret_cast<const float4 *>(&s.Cc[u][off + pr]);
                    cfma(dot[0], make_float2(cv.x, cv.y), rv);
                    cfma(dot[1], make_float2(cv.z, cv.w), rv);
                }
#pragma unroll
                for (int m = 0; m < 2; ++m) d[m] = csub(d[m], dot[m]);
                const bool leaving = kn + FB >= r0 + G;
                if (!leaving) asm volatile("bar.arrive 2, 384;" ::: "memory");
                pivot(d, k + 1, tag + 1u, j);
                if (leaving) asm volatile("bar.arrive 2, 384;" ::: "memory");
            }
        }
        if (tile_warp) {
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int jj = 0; jj < 3; ++jj) {
                    const int r = r0 + tr + 16 * i, c = c0 + tc + 16 * jj;
                    if (r < n && c < n) p.invT[(size_t)j * page_sz + (size_t)(r + 1) + (size_t)ny * (c + 1)] = a[i][jj];
                }
        }
        if (!grid_barrier(p.counter, p.err, gridDim.x, epoch, p.timeout_ns, 5004)) {
            asm volatile("cp.async.wait_all;" ::: "memory");
            return;
        }
    }
}

size_t factor_scratch_bytes(int ny) { return factor_scratch_bytes_for(ny); }

void factor_launch(const Coefs<float2> &co, float2 *invT, void *scratch, size_t scratch_bytes,
                   cudaStream_t stream, double timeout_s, int *host_status, int j0, int j1, int max_ctas) {
    const int ny = co.ny;
    const int n = ny - 2;
    const int np_ = (int)factor_pad(ny);
    if (scratch_bytes < factor_scratch_bytes(ny)) fail(WUST_ERR_RUNTIME, "factor scratch too small");
    int dev = 0, sms = 0, per_sm = 0;
    WUST_CUDA(cudaGetDevice(&dev));
    WUST_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int nt = np_ / G;
    int grid = sms;                          // one CTA per SM
    if (max_ctas > 0 && grid > max_ctas) grid = max_ctas;
    const int first = j0, last = j1 < 0 ? co.nx : j1;
    if (first < 0 || first >= last || last > co.nx) fail(WUST_ERR_RUNTIME, "factor page range [%d, %d) invalid", j0, j1);
    const unsigned long long timeout_ns = (unsigned long long)(timeout_s * 1e9);
    int *tail = nullptr;
    // One tile per CTA: the dataflow kernel (552 pages of 552^2 in 73 ms
    // against 169, 64 of 64^2 in 1.4 against 3.5).  Larger pages, or a grid
    // capped below the tiles, take the kernel whose CTAs walk over several
    // tiles between grid barriers.
    if (nt <= kFlowMaxTiles && nt * nt <= grid) {
        FlowParams p;
        p.co = co;
        p.invT = invT;
        p.nsteps = ceil_div(n, FB);          // the padding beyond n is the identity and stays so
        p.rowp = (ulonglong2 *)scratch;
        p.colp = p.rowp + (size_t)p.nsteps * np_ * FB;
        p.pivp = p.colp + (size_t)p.nsteps * np_ * FB;
        ulonglong2 *end = p.pivp + (size_t)p.nsteps * FB * FB;
        tail = (int *)end;
        p.counter = (unsigned *)tail;
        p.err = tail + 1;
        p.status = (unsigned *)(tail + 4);
        p.n = n;
        p.n_pad = np_;
        p.j0 = first;
        p.j1 = last;
        p.timeout_ns = timeout_ns;
        // tags of this launch start at 1: whatever the scratch held is cleared
        WUST_CUDA(cudaMemsetAsync(scratch, 0, (size_t)((uint8_t *)(tail + 8) - (uint8_t *)scratch), stream));
        WUST_CUDA(cudaFuncSetAttribute(factor_flow_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kFlowSmemBytes));
        WUST_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, factor_flow_kernel, FT, kFlowSmemBytes));
        if (per_sm < 1) fail(WUST_ERR_CUDA, "factor kernel cannot be resident");
        void *args[] = {&p};
        WUST_CUDA(cudaLaunchCooperativeKernel((void *)factor_flow_kernel, dim3(nt * nt), dim3(FT), args, kFlowSmemBytes,
                                              stream));
    } else {
        FactorParams p;
        p.co = co;
        p.invT = invT;
        p.ws0 = (float2 *)scratch;
        p.ws1 = p.ws0 + (size_t)np_ * np_;
        tail = (int *)(p.ws1 + (size_t)np_ * np_);
        p.counter = (unsigned *)tail;
        p.err = tail + 1;
        p.status = tail + 2;
        p.n = n;
        p.n_pad = np_;
        p.j0 = first;
        p.j1 = last;
        p.timeout_ns = timeout_ns;
        WUST_CUDA(cudaMemsetAsync(tail, 0, 8 * sizeof(int), stream));
        // Set on every launch: the attribute belongs to the current device's
        // context, which a caller may switch or reset between calls.
        WUST_CUDA(cudaFuncSetAttribute(factor_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFactorSmemBytes));
        WUST_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, factor_kernel, GT, kFactorSmemBytes));
        if (per_sm < 1) fail(WUST_ERR_CUDA, "factor kernel cannot be resident");
        if (grid > nt * nt) grid = nt * nt;
        void *args[] = {&p};
        WUST_CUDA(cudaLaunchCooperativeKernel((void *)factor_kernel, dim3(grid), dim3(GT), args, kFactorSmemBytes, stream));
    }
    WUST_LAUNCH_CHECK();
    ++g_kernel_launches;
    if (host_status) {
        int st[8];
        WUST_CUDA(cudaMemcpyAsync(st, tail, sizeof(st), cudaMemcpyDeviceToHost, stream));
        WUST_CUDA(cudaStreamSynchronize(stream));
        host_status[0] = st[2];
        host_status[1] = st[3];
        if (st[4]) {                         // the dataflow kernel's
            const unsigned at = 0xffffffffu - (unsigned)st[4];
            host_status[0] = (int)(at / kFlowPivots) + 1;
            host_status[1] = (int)(at % kFlowPivots);
        }
        host_status[2] = st[1];
    }
}

// Self-test of the bounded wait: one CTA waits at a barrier sized for
// gridDim.x + 1 CTAs, which can never fill, and must give up after timeout_ns.
__global__ void barrier_timeout_probe(unsigned *counter, int *err, unsigned long long timeout_ns, int *passed) {
    unsigned epoch = 0;
    const bool ok = grid_barrier(counter, err, gridDim.x + 1, epoch, timeout_ns, 77);
    if (threadIdx.x == 0) passed[blockIdx.x] = ok ? 1 : 0;
}

int barrier_selftest(double timeout_s, int *site_out) {
    int *buf = nullptr;
    WUST_CUDA(cudaMalloc(&buf, 4 * sizeof(int)));
    WUST_CUDA(cudaMemset(buf, 0, 4 * sizeof(int)));
    barrier_timeout_probe<<<1, 32>>>((unsigned *)buf, buf + 1, (unsigned long long)(timeout_s * 1e9), buf + 2);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    int host[4] = {0, 0, -1, 0};
    if (e == cudaSuccess) cudaMemcpy(host, buf, sizeof(host), cudaMemcpyDeviceToHost);
    cudaFree(buf);
    if (e != cudaSuccess) fail(WUST_ERR_CUDA, "barrier self-test: %s", cudaGetErrorString(e));
    *site_out = host[1];
    return host[2];
}

}  // namespace wust
