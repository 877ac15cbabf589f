// Chunked tensor-core sweeps: the column recurrence of each substitution of
// applyBlockLU (Runtime/solver/applyBlockLU.cu:433-467) cut into C chunks of
// columns that run concurrently.
//
// Step by step, every substitution is an affine recurrence on one column
// state c (ny x S):  c_i = Lambda_i c_{i-1} + g_i,  Lambda_i = -+ invT_j W_i
// (W_i the tridiagonal coupling block of the step, g_i the source or the
// already-solved column).  Cutting the nx - 1 steps of a substitution into C
// chunks of consecutive steps:
//   pass 1    every chunk runs its steps from c = 0, chunk 0 from its true
//             incoming state (it also writes its columns of u): end states z_c;
//   boundary  s_0 = z_0,  s_c = z_c + Lambda_c s_{c-1}  for c = 1 .. C-2,
//             Lambda_c the chunk's composed propagator (formed once per
//             factorization by running the chunk on the identity);
//   pass 2    chunks 1 .. C-1 rerun from s_{c-1} and write their columns.
// The serial depth drops from nx - 1 steps to about 2 (nx - 1) / C + C.
//
// A group of mt CTAs (one per 64-row complex M tile, one CTA per SM) runs a
// chunk.  Each step is one full-K complex GEMM per CTA,
//     C (64 rows x N) = A (64 rows x n) B (n x N),  N <= 256 sources,
// real-split with re/im interleaved along K exactly as in tcsweep.cu; A (the
// packed invT page) and B (the packed right-hand side) stream through a
// bulk-copy ring of 2 to 5 stages (ck_ring) into kind::tf32 MMAs of N columns,
// the accumulator sits in tensor memory.  After the MMAs each CTA writes its rows of the new
// state (re and im planes, rows fastest) and of u, meets its group on a
// counter barrier, evaluates the next step's stencil for its rows (the
// neighbour rows come from L2) into the packed B chunks, and meets the group
// again.  The A chunks of the next step are copied while that happens.
// Groups never wait on each other.  Every device wait is bounded and reports
// its site through *err.
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "kernels.cuh"
#include "tc.cuh"
#include "tcstep.cuh"

namespace wust {

constexpr int kCkThreads = 512;
constexpr int kCkWarps = kCkThreads / 32;
constexpr int kCkRingChunks = 4, kCkMaxStages = 5;               // room of the ring: K chunks of kCkMaxN sources
constexpr int kCopyTid = 96, kCopyBTid = 128;                    // the ring's copy threads, of A and of B (lanes 0)
constexpr int kCkMaxN = 256;                                     // sources per launch (MMA N)
constexpr int kCkRowsPerChunk = 16;                              // complex rows per K chunk (TF32)
constexpr int kCkRowsPerChunk16 = 32;                            // complex rows per K chunk (BF16)
constexpr int kCkMaxChunks = 148;
constexpr size_t kCkBSlot = (size_t)kCkMaxN * tc::kChunkBytes;   // 32 KB
constexpr size_t kCkSmemRing = (size_t)kCkRingChunks * (tc::kAChunk + kCkBSlot);
constexpr size_t kCkSmemHalo = 2 * kCkMaxN * sizeof(float2);
constexpr size_t kCkSmemW = 3 * 64 * sizeof(float2);
constexpr size_t kCkSmem = kCkSmemRing + kCkSmemHalo + kCkSmemW + 256;
static_assert(kCkSmem <= 232448, "shared memory of one CTA");

// The ring of a launch of N sources: as many stages as the shared memory holds,
// and K chunks per stage so that a stage's products take about as long as its
// share of the waits, commits and copies: a 16-row chunk of 256 sources is 512
// cycles of MMAs, of 128 sources 256, of 16 (the boundary chain) 192.
// Measured with 4 / 2 / 1 chunks per stage against 1: 288^2 Hessian product
// 26.9 against 28.5 ms, 437 x 401 solve 16.6 against 17.9; two at N = 256 (two
// stages left in the ring): 552^2 gradient 70.5 against 68.3.
struct CkRing { int per_stage, stages; };
constexpr CkRing ck_ring(int N) {
    const int per = N <= 64 ? 4 : N <= 128 ? 2 : 1;
    return CkRing{per, (int)(kCkSmemRing / (per * (tc::kAChunk + (size_t)N * tc::kChunkBytes)))};
}
constexpr bool ck_rings_hold() {
    for (int N = 8; N <= kCkMaxN; N += 8) {
        const CkRing r = ck_ring(N);
        // the B stages hold the staged state between a step's MMAs and the next step's copies
        if (r.stages < 2 || r.stages > kCkMaxStages ||
            (size_t)r.stages * r.per_stage * tc::kChunkBytes < 64 * sizeof(float2))
            return false;
    }
    return true;
}
static_assert(ck_rings_hold(), "a ring of two stages at least, whose B stages hold the staged state");

__host__ __device__ constexpr int ceil_div8(int x) { return (x + 7) / 8 * 8; }

using tc::chunk_off;
using tc::to_tf32;

// Launch kinds and the kind of work of one group.
enum CkPass { CK_FIRST = 0, CK_SECOND = 1, CK_PROP = 2, CK_BOUNDARY = 3 };
enum CkKind { K_EXACT = 0, K_LOCAL = 1, K_PROP = 2, K_BOUND = 3 };
// Where the incoming state of a chunk comes from.
enum CkIn { IN_ZERO = 0, IN_PLANES = 1, IN_UCOL = 2, IN_IDENT = 3 };
// What produce makes of the staged state.
enum CkProduce { P_STENCIL = 0, P_IDENT = 1, P_TURN = 2 };

size_t tc_chunk_state_floats(int ny) { return (size_t)2 * kCkMaxN * ny; }

TcChunkGeom tc_chunk_geom(int ny, int nx, int max_ctas, int chunks) {
    TcChunkGeom g{};
    g.n = ny - 2;
    g.mt = ceil_div(g.n, 64);
    g.kc = ceil_div(g.n, kCkRowsPerChunk);
    g.kc16 = ceil_div(g.n, kCkRowsPerChunk16);
    const int steps = nx - 1;
    if (steps < 1 || g.n < 1) fail(WUST_ERR_INVALID_INPUT, "chunked sweep needs Nx >= 2 and Ny >= 3");
    if (g.mt > max_ctas)
        fail(WUST_ERR_INVALID_INPUT, "chunked sweep needs %d co-resident CTAs (device holds %d)", g.mt, max_ctas);
    // about sqrt(2 steps) chunks balance the two passes against the boundary
    // chain; every chunk keeps at least 2 steps (the mirrored H^H backward
    // cuts then leave no chunk empty)
    int C = chunks > 0 ? chunks : (int)std::lround(std::sqrt(2.0 * steps));
    C = std::max(1, std::min({C, max_ctas / g.mt, steps / 2, kCkMaxChunks}));
    g.C = C;
    g.page_bytes = (size_t)g.mt * g.kc * tc::kAChunk;
    g.page_bytes16 = (size_t)g.mt * g.kc16 * tc::kAChunk;
    g.lpack_bytes = C >= 3 ? (size_t)4 * C * g.page_bytes : 0;
    g.lpack16_bytes = C >= 3 ? (size_t)4 * C * g.page_bytes16 : 0;
    g.b_bytes = (size_t)C * g.kc * kCkBSlot;
    g.state_bytes = (size_t)C * tc_chunk_state_floats(ny) * sizeof(float);
    g.edge_bytes = (size_t)C * g.mt * 2 * kCkMaxN * sizeof(float2);
    g.sync_words = C;
    return g;
}

// Optional phase timer (SM cycles of CTA 0, summed over steps, per launch
// kind), built only into profiling builds of the library.
#ifdef WUST_CHUNK_PROFILE
__device__ unsigned long long g_chunk_prof[4][8];
#define CPROF(k)                                                                                  \
    do {                                                                                          \
        if (blockIdx.x == 0 && threadIdx.x == 0) {                                                \
            const long long t_ = clock64();                                                       \
            g_chunk_prof[p.pass][k] += (unsigned long long)(t_ - prof_t);                         \
            prof_t = t_;                                                                          \
        }                                                                                         \
    } while (0)
extern "C" int wust_chunk_profile_read(unsigned long long *out) {
    return (int)cudaMemcpyFromSymbol(out, g_chunk_prof, sizeof(g_chunk_prof));
}
extern "C" int wust_chunk_profile_reset() {
    unsigned long long z[32] = {};
    return (int)cudaMemcpyToSymbol(g_chunk_prof, z, sizeof(z));
}
#else
#define CPROF(k) ((void)0)
#endif

struct ChunkParams {
    const uint8_t *apack;     // packed pages of the solve (invT or invT^H): [page][mt][kc] chunks
    const uint8_t *lpack;     // boundary launches: packed -Lambda_c pages, [chunk][mt][kc]
    size_t page_bytes;
    Coefs<float2> co;
    SrcView src;
    float2 *u;                // [ny, nx, S] (global source index)
    uint8_t *bglob;           // [group][kc] chunks of N x 128 bytes
    float *zst;               // [chunk] states: re plane [kCkMaxN][ny], im plane [kCkMaxN][ny]
    float *sb;                // [chunk] boundary states s_c (c >= 1), same layout
    float2 *edges;            // [group][mt][2][kCkMaxN]: first and last own row of each CTA's state
    unsigned *group_ctr;      // [group]
    int *err;
    int ny, nx, n, mt, kc, N;
    int s0, s_end;            // global sources [s0, s_end) of this launch
    int half;                 // 0: forward substitution (steps 0 .. nx-2), 1: backward
    int stages, per_stage;    // of the operand ring; K chunks per stage
    int pass, C;
    int bounds[kCkMaxChunks + 1];   // first step (within the half) of each chunk
    unsigned long long timeout_ns;
};

// Where the staged state holds row r of source s: pairs of rows, permuted
// within eight so that a pair of 8 sources lies in 8 different bank groups.
__device__ __forceinline__ int cs_at(int s, int r) { return s * 64 + (r ^ ((s & 7) << 1)); }

// BF: BF16 operands (kind::f16 MMAs, 32 complex rows per K chunk) for the
// correction solves of the refinement; TF32 otherwise.
template <bool ADJ, bool BF>
__global__ void __launch_bounds__(kCkThreads, 1) tc_chunk_kernel(const __grid_constant__ ChunkParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const int stages = p.stages, G = p.per_stage, kg = (p.kc + G - 1) / G;
    uint8_t *sA = smem;                                          // [stage] G chunks of 16 KB
    uint8_t *sB = smem + (size_t)stages * G * tc::kAChunk;       // [stage] G chunks of N x 128 bytes
    // Between a step's MMAs and the next step's B copies the B stages hold the
    // state of this CTA's 64 rows: cs[cs_at(s, row)] (complex).
    float2 *cs = reinterpret_cast<float2 *>(sB);
    float2 *halo = reinterpret_cast<float2 *>(smem + kCkSmemRing);  // [2][kCkMaxN]: rows 64t-1 and 64t+64
    float2 *wts = halo + 2 * kCkMaxN;                                // [3][64] stencil weights of own rows
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + kCkSmemRing + kCkSmemHalo + kCkSmemW);
    uint64_t *empty = full + kCkMaxStages;
    uint64_t *done = empty + kCkMaxStages;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(done + 1);
    int *s_ok = reinterpret_cast<int *>(tmem_slot + 1);
    uint32_t *s_ring = reinterpret_cast<uint32_t *>(s_ok + 1);   // [0] A, [1] B copies issued

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = blockIdx.x / p.mt, t = blockIdx.x % p.mt;
    const int ny = p.ny, nx = p.nx, n = p.n, kc = p.kc, N = p.N;
    const size_t plane = (size_t)ny * nx;
    const size_t sfl = (size_t)2 * kCkMaxN * ny;                 // floats per state
    const size_t bbytes = (size_t)N * tc::kChunkBytes;
    uint8_t *bg = p.bglob + (size_t)g * kc * bbytes;
    unsigned *ctr = p.group_ctr + g;
    const int row0 = 64 * t;                                     // first complex interior row of this CTA
    // the boundary chain splits the launch's sources over its groups: group g
    // takes sources [so, so + N) of the launch (every other pass: so = 0)
    const int so = p.pass == CK_BOUNDARY ? g * N : 0;

    // this group's chunk, kind and steps
    int chunk, kind, t0, nsteps;
    if (p.pass == CK_BOUNDARY) {
        chunk = 0; kind = K_BOUND; t0 = 1; nsteps = p.C - 2;
    } else {
        chunk = (p.pass == CK_FIRST ? 0 : 1) + g;
        kind = p.pass == CK_PROP ? K_PROP : (p.pass == CK_SECOND || chunk == 0) ? K_EXACT : K_LOCAL;
        t0 = p.bounds[chunk];
        nsteps = p.bounds[chunk + 1] - t0;
    }
    // state planes of the boundary sequence: s_0 = z_0 (the end state of
    // chunk 0), s_c in sb.  H^H solves carry B states between chunks (the
    // first B of the next chunk), kept in sb from the start.
    auto bstate = [&](int c) -> float * { return (c == 0 && !ADJ) ? p.zst : p.sb + (size_t)c * sfl; };

    auto col_of = [&](int k, bool &fwd) -> int {
        if (kind == K_BOUND) { fwd = false; return 0; }
        return step_col(p.half * (nx - 1) + t0 + k, nx, fwd);
    };
    auto apage = [&](int k) -> const uint8_t * {
        if (kind == K_BOUND) return p.lpack + (size_t)(t0 + k) * p.page_bytes;
        bool f;
        const int j = col_of(k, f);
        return p.apack + (size_t)((ADJ && f) ? j - 1 : j) * p.page_bytes;
    };
    // incoming state value at grid row y (0 .. ny-1; 0 outside), local source s
    // (0 for the padding sources beyond s_end: the caller's fields hold only
    // s_end sources)
    auto cval = [&](int in, const float *pl, int y, int s) -> float2 {
        if (y < 0 || y >= ny || p.s0 + so + s >= p.s_end) return f2(0.f, 0.f);
        if (in == IN_PLANES)
            return f2(__ldcg(pl + (size_t)(so + s) * ny + y), __ldcg(pl + (size_t)(kCkMaxN + so + s) * ny + y));
        if (in == IN_UCOL) return __ldcg(p.u + plane * (p.s0 + so + s) + (size_t)ny * (nx - 1) + y);
        if (in == IN_IDENT) return f2((y >= 1 && y <= n && y - 1 == p.s0 + so + s) ? 1.f : 0.f, 0.f);
        return f2(0.f, 0.f);
    };
    // staged state at complex interior row yp (row0 - 1 .. row0 + 64)
    auto cs_get = [&](int yp, int s) -> float2 {
        const int l = yp - row0;
        if (l >= 0 && l < 64) return cs[cs_at(s, l)];
        if (l == -1) return halo[s];
        if (l == 64) return halo[kCkMaxN + s];
        return f2(0.f, 0.f);
    };
    // own rows and halo rows of an incoming state -> shared memory
    auto stage_in = [&](int in, const float *pl) {
        __syncthreads();
        for (int it0 = tid; it0 < 64 * N; it0 += 4 * kCkThreads) {
            float2 v[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int it = it0 + q * kCkThreads;
                v[q] = it < 64 * N ? cval(in, pl, row0 + (it & 63) + 1, it >> 6) : f2(0.f, 0.f);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int it = it0 + q * kCkThreads;
                if (it < 64 * N) cs[cs_at(it >> 6, it & 63)] = v[q];
            }
        }
        for (int it = tid; it < 2 * N; it += kCkThreads) {
            const int e = it / N, s = it % N;
            halo[e * kCkMaxN + s] = cval(in, pl, e == 0 ? row0 : row0 + 65, s);
        }
    };
    // halo rows: the last row of the CTA above and the first row of the CTA
    // below (zero at the grid's edges)
    float2 *my_edges = p.edges + ((size_t)g * p.mt + t) * 2 * kCkMaxN;
    auto stage_halo = [&]() {
        __syncthreads();
        for (int it = tid; it < 2 * N; it += kCkThreads) {
            const int e = it / N, s = it % N;
            float2 v = f2(0.f, 0.f);
            if (e == 0 && t > 0) v = __ldcg(my_edges - 2 * kCkMaxN + kCkMaxN + s);
            if (e == 1 && t < p.mt - 1) v = __ldcg(my_edges + 2 * kCkMaxN + s);
            halo[e * kCkMaxN + s] = v;
        }
    };

    // stencil weights of own row row0 + r for step (fwd1, j1) -> wts
    auto fill_weights = [&](int r, bool ident, bool fwd1, int j1) {
        const int yp = row0 + r, y = yp + 1;
        float2 wc = f2(0.f, 0.f), wm = wc, wp = wc;
        if (yp < n) {
            if (ident) wc = f2(-1.f, 0.f);
            else step_weights<ADJ>(p.co, fwd1, j1, y, wc, wm, wp);
        }
        wts[r] = wc;
        wts[64 + r] = wm;
        wts[128 + r] = wp;
    };

    // B of step k for this CTA's rows from the staged state:
    //   P_STENCIL  B = base - stencil(state), into the packed chunks, or as
    //              FP32 planes into `out` (a chunk's outgoing B state);
    //   P_IDENT    B = state (an incoming B state, or a boundary step);
    //   P_TURN     the turn of the H^H solve: u(:, nx-1) = SRC_{nx-1} -
    //              U_{nx-2}^H c on every row, no B.
    // Exact H^H forward steps also write B into u(:, j-1) (stencil mode:
    // with its border rows).
    auto produce = [&](int k, int mode, float *out, bool wts_ready) {
        bool fwd1 = true;
        int j1 = nx;
        if (mode != P_TURN) j1 = col_of(k, fwd1);
        const bool pack = mode != P_TURN && !out;
        const bool ident = mode == P_IDENT;
        const bool wu = kind == K_EXACT && ADJ && fwd1 && !out;
        const bool has_base = (kind == K_EXACT || kind == K_LOCAL) && !ident;
        __syncthreads();
        if (!wts_ready && tid < 64) fill_weights(tid, ident, fwd1, j1);
        __syncthreads();
        if (wu && !ident) {
            // border rows 0 and ny-1 of u(:, j1-1) (no B entry)
            for (int it = tid; it < 2 * N; it += kCkThreads) {
                const int e = it / N, s = it % N, gs = p.s0 + so + s;
                if ((e == 0 && t != 0) || (e == 1 && t != p.mt - 1) || gs >= p.s_end) continue;
                const int y = e == 0 ? 0 : ny - 1, yp = y - 1;
                float2 wc, wm, wp;
                step_weights<ADJ>(p.co, fwd1, j1, y, wc, wm, wp);
                float2 acc = cmul(wc, cs_get(yp, s));
                cfma(acc, wm, cs_get(yp - 1, s));
                cfma(acc, wp, cs_get(yp + 1, s));
                p.u[plane * gs + (size_t)ny * (j1 - 1) + y] =
                    csub(step_base<ADJ>(p.src, p.u, ny, nx, fwd1, j1, y, gs), acc);
            }
            __syncthreads();                               // below, the results replace the staged state
        }
        // base of the step (step_base), what does not depend on the source taken out of the loop
        const float2 *bcol = nullptr;
        bool point = false, scatter = false;
        int col_at = 0;
        if (has_base && fwd1 && (!ADJ || j1 >= 2)) {
            const int jb = ADJ ? j1 - 1 : j1;
            col_at = row0 + 1 + ny * jb;
            if (p.src.mode == SRC_DENSE) bcol = p.src.dense + (size_t)ny * jb;
            point = p.src.mode == SRC_POINT;
            scatter = p.src.mode == SRC_SCATTER;
        } else if (has_base && ADJ && !fwd1) {
            bcol = p.u + (size_t)ny * j1;
        }
        const bool fields = bcol || wu || out;      // columns of fields are read or written
        // Where columns of fields are involved, a first pass forms B in place of
        // the staged state, rows in lanes, so that each access to a field is a
        // run of 32 rows.  The second packs it (and, without fields, forms it):
        // a lane takes one 16-byte unit of one source, a warp 4 units of 8
        // sources, 512 bytes of a packed chunk in a row, straight from registers.
        // Loops stay rolled: a step runs all of its code once, and straight-line
        // code for 8 sources was bound by instruction fetch.  Per step of 16
        // sources 2.5 -> 0.8 us, of 64 (half of the steps with fields) 3.5 -> 2.8,
        // of 192 without fields 5.2 -> 4.6; of 256 with fields 8.6 -> 9.0.
        constexpr int RPC = BF ? kCkRowsPerChunk16 : kCkRowsPerChunk;
        constexpr int RPU = RPC / 8, NI = 16 / RPU;                   // rows of a 16-byte unit; items of 8 sources
        if (fields) {
            const int yl = row0 + lane + 1;                           // rows of this lane: yl and yl + 32
            int at[2] = {col_at + lane, col_at + lane + 32};
            if (scatter)
                for (int h = 0; h < 2; ++h) at[h] = yl + 32 * h <= n ? p.src.at[at[h]] : -1;
            float2 wc[2], wm[2], wp[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                wc[h] = wts[lane + 32 * h];
                wm[h] = wts[64 + lane + 32 * h];
                wp[h] = wts[128 + lane + 32 * h];
            }
#pragma unroll 1
            for (int s0 = 4 * warp; s0 < N; s0 += 4 * kCkWarps) {
                float2 v[4][2];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int gs = p.s0 + so + s0 + q;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        v[q][h] = f2(0.f, 0.f);
                        if (gs >= p.s_end) continue;
                        if (bcol) {
                            if (yl + 32 * h <= n) v[q][h] = __ldcg(bcol + plane * gs + yl + 32 * h);
                        } else if (point) {
                            v[q][h].x = p.src.lin[gs] == at[h] ? 1.f : 0.f;
                        } else if (scatter && at[h] >= 0) {
                            v[q][h] = p.src.vals[at[h] + (size_t)p.src.n_slots * gs];
                        }
                    }
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int s = s0 + q, gs = p.s0 + so + s;
                    float2 c[2][3];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int r = lane + 32 * h;
                        c[h][0] = r == 0 ? halo[s] : cs[cs_at(s, r - 1)];
                        c[h][1] = cs[cs_at(s, r)];
                        c[h][2] = r == 63 ? halo[kCkMaxN + s] : cs[cs_at(s, r + 1)];
                    }
                    __syncwarp();
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        float2 acc = cmul(wc[h], c[h][1]);
                        cfma(acc, wm[h], c[h][0]);
                        cfma(acc, wp[h], c[h][2]);
                        const bool on = gs < p.s_end && yl + 32 * h <= n;
                        const float2 b = on ? csub(v[q][h], acc) : f2(0.f, 0.f);
                        if (on && wu) p.u[plane * gs + (size_t)ny * (j1 - 1) + yl + 32 * h] = b;
                        if (on && out) {
                            __stcg(out + (size_t)(so + s) * ny + yl + 32 * h, b.x);
                            __stcg(out + (size_t)(kCkMaxN + so + s) * ny + yl + 32 * h, b.y);
                        }
                        cs[cs_at(s, lane + 32 * h)] = b;
                    }
                }
            }
            if (!pack) return;
            __syncthreads();
        }
#pragma unroll 1
        for (int it = warp; it < N / 8 * NI; it += kCkWarps) {
            const int unit = (it % NI) * 4 + (lane >> 3), r = unit * RPU, s = it / NI * 8 + (lane & 7);
            const int gs = p.s0 + so + s;
            float2 v[RPU], c[RPU + 2];
#pragma unroll
            for (int h = 0; h < RPU; h += 2) {
                const float4 c2 = *reinterpret_cast<const float4 *>(cs + cs_at(s, r + h));
                c[h + 1] = f2(c2.x, c2.y);
                c[h + 2] = f2(c2.z, c2.w);
            }
            if (fields) {
#pragma unroll
                for (int h = 0; h < RPU; ++h) v[h] = c[h + 1];
            } else {
                c[0] = r == 0 ? halo[s] : cs[cs_at(s, r - 1)];
                c[RPU + 1] = r + RPU == 64 ? halo[kCkMaxN + s] : cs[cs_at(s, r + RPU)];
                const int src_row = point && gs < p.s_end ? p.src.lin[gs] - col_at : -1;
#pragma unroll
                for (int h = 0; h < RPU; ++h) {
                    float2 acc = cmul(wts[r + h], c[h + 1]), base = f2(0.f, 0.f);
                    cfma(acc, wts[64 + r + h], c[h]);
                    cfma(acc, wts[128 + r + h], c[h + 2]);
                    const bool on = gs < p.s_end && row0 + r + h < n;
                    if (src_row == r + h) base.x = 1.f;
                    if (scatter && on) {
                        const int k1 = p.src.at[col_at + r + h];
                        if (k1 >= 0) base = p.src.vals[k1 + (size_t)p.src.n_slots * gs];
                    }
                    v[h] = on ? csub(base, acc) : f2(0.f, 0.f);
                }
            }
            const int at = row0 / RPU + unit;                         // unit of the group's B
            if (at >= 8 * kc) continue;
            float4 q;
            if constexpr (BF) {
                uint32_t w[4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    w[i] = (uint32_t)tc::to_bf16_bits(v[i].x) | ((uint32_t)tc::to_bf16_bits(v[i].y) << 16);
                q = make_float4(__uint_as_float(w[0]), __uint_as_float(w[1]), __uint_as_float(w[2]), __uint_as_float(w[3]));
            } else {
                q = make_float4(to_tf32(v[0].x), to_tf32(v[0].y), to_tf32(v[1].x), to_tf32(v[1].y));
            }
            *reinterpret_cast<float4 *>(bg + (size_t)(at >> 3) * bbytes + (size_t)(s >> 3) * 1024 + (at & 7) * 128 + (s & 7) * 16) = q;
        }
    };

    if (tid == 0) {
        for (int q = 0; q < stages; ++q) {
            tc::mbar_init(&full[q], 2);       // A copy + B copy
            tc::mbar_init(&empty[q], 1);      // MMAs of the stage retired
        }
        tc::mbar_init(done, 1);
        tc::mbar_fence_init();
    }
    const uint32_t tcols = N <= 32 ? 32u : N <= 64 ? 64u : N <= 128 ? 128u : 256u;
    if (warp == 0) tc::tmem_alloc(tmem_slot, tcols);
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = *tmem_slot;

    // Accumulator (TMEM) -> staged state, own rows (rows beyond the grid 0).
    auto drain_tmem = [&]() {
        const int l = 32 * (warp & 3) + lane;
        const int part = l >> 6;                       // TMEM lanes 0-63: real parts, 64-127: imaginary
        const int row = l & 63;
        const bool row_ok = row0 + row < n;
        const int hc = ceil_div8(N / (kCkWarps / 4)), c0 = (warp >> 2) * hc;
        float *csf = reinterpret_cast<float *>(cs);
        const uint32_t tl = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
        int cb = 0;
        for (; cb + 32 <= hc && c0 + cb + 32 <= N; cb += 32) {
            float v[32];
            tc::tmem_ld32(tl + (uint32_t)(c0 + cb), v);
#pragma unroll
            for (int q = 0; q < 32; ++q) csf[cs_at(c0 + cb + q, row) * 2 + part] = row_ok ? v[q] : 0.f;
        }
        for (; cb < hc && c0 + cb < N; cb += 8) {
            float v[8];
            tc::tmem_ld8(tl + (uint32_t)(c0 + cb), v);
#pragma unroll
            for (int q = 0; q < 8; ++q) csf[cs_at(c0 + cb + q, row) * 2 + part] = row_ok ? v[q] : 0.f;
        }
    };
    // The state after step k: subtracting steps take old - value; write the
    // finished columns of u, and the state's edge rows (every row on the
    // chunk's last step) to the planes curp.
    auto finish = [&](int k, float *curp, bool last) {
        bool fwd = false;
        const int j = col_of(k, fwd);
        const bool sub = kind == K_BOUND || (!ADJ && !fwd);
        const bool wu = kind == K_EXACT && (!ADJ || !fwd);
        const float *oldp = kind == K_BOUND ? (ADJ ? p.sb : p.zst) + (size_t)(t0 + k) * sfl : nullptr;
        const bool old_u = sub && kind != K_BOUND && kind != K_PROP;
        const int y0 = row0 + lane + 1, y1 = y0 + 32;
        const bool v0 = y0 <= n, v1 = y1 <= n;
        __syncthreads();
        for (int sb0 = warp; sb0 < N; sb0 += 4 * kCkWarps) {
            float2 o[4][2];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int s = sb0 + kCkWarps * q, gs = p.s0 + so + s;
                o[q][0] = o[q][1] = f2(0.f, 0.f);
                if (s < N && gs < p.s_end) {
                    if (old_u) {
                        const float2 *uc = p.u + plane * gs + (size_t)ny * j;
                        if (v0) o[q][0] = __ldcs(uc + y0);
                        if (v1) o[q][1] = __ldcs(uc + y1);
                    } else if (kind == K_BOUND) {
                        const float *ore = oldp + (size_t)(so + s) * ny, *oim = oldp + (size_t)(kCkMaxN + so + s) * ny;
                        if (v0) o[q][0] = f2(__ldcg(ore + y0), __ldcg(oim + y0));
                        if (v1) o[q][1] = f2(__ldcg(ore + y1), __ldcg(oim + y1));
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int s = sb0 + kCkWarps * q, gs = p.s0 + so + s;
                if (s >= N) break;                                   // warp-uniform
                float2 *e0 = cs + cs_at(s, lane), *e1 = cs + cs_at(s, lane + 32);
                float2 c0 = *e0, c1 = *e1;
                if (sub) {
                    c0 = v0 ? csub(o[q][0], c0) : f2(0.f, 0.f);
                    c1 = v1 ? csub(o[q][1], c1) : f2(0.f, 0.f);
                    *e0 = c0;
                    *e1 = c1;
                }
                if (gs >= p.s_end) continue;
                if (wu) {                 // u streams through L2 (evict first), as the old column it replaces
                    float2 *uc = p.u + plane * gs + (size_t)ny * j;
                    if (v0) __stcs(uc + y0, c0);
                    if (v1) __stcs(uc + y1, c1);
                }
                if (last) {
                    float *re = curp + (size_t)(so + s) * ny, *im = curp + (size_t)(kCkMaxN + so + s) * ny;
                    if (v0) { __stcg(re + y0, c0.x); __stcg(im + y0, c0.y); }
                    if (v1) { __stcg(re + y1, c1.x); __stcg(im + y1, c1.y); }
                }
            }
        }
        // edge rows of the warp's sources
        __syncwarp();
        for (int it = lane; it < 2 * kCkMaxN / kCkWarps; it += 32) {
            const int s = warp + kCkWarps * (it >> 1), e = it & 1;
            if (s < N && p.s0 + so + s < p.s_end && (e == 0 || row0 + 63 < n))
                __stcg(my_edges + e * kCkMaxN + s, cs[cs_at(s, 63 * e)]);
        }
        if (kind == K_EXACT && ADJ && !fwd && t == 0) {
            // H^H backward: border rows of u(:, j) are zero
            for (int s = tid; s < N; s += kCkThreads) {
                const int gs = p.s0 + so + s;
                if (gs >= p.s_end) continue;
                p.u[plane * gs + (size_t)ny * j] = f2(0.f, 0.f);
                p.u[plane * gs + (size_t)ny * j + ny - 1] = f2(0.f, 0.f);
            }
        }
    };

    // Warps 1-7, while the MMAs run: pull into L2 the field columns that the
    // coming finish (old column of a subtracting step) and produce (base of
    // the next step) will read, own rows of every source.
    auto prefetch_cols = [&](int k) {
        const float2 *cols[2] = {nullptr, nullptr};
        bool fwd;
        const int j = col_of(k, fwd);
        if ((kind == K_EXACT || kind == K_LOCAL) && !ADJ && !fwd) cols[0] = p.u + (size_t)ny * j;
        if ((kind == K_EXACT || kind == K_LOCAL) && k + 1 < nsteps) {
            bool f1;
            const int j1 = col_of(k + 1, f1);
            if (ADJ && !f1) cols[1] = p.u + (size_t)ny * j1;
            else if (p.src.mode == SRC_DENSE && (!ADJ || j1 >= 2) && f1)
                cols[1] = p.src.dense + (size_t)ny * (ADJ ? j1 - 1 : j1);
        }
        const int y_first = row0 + 1, y_last = min(row0 + 64, n);
        for (int c = 0; c < 2; ++c) {
            if (!cols[c]) continue;
            for (int it = tid - 32; it < N * 5; it += kCkThreads - 32) {
                const int s = it / 5, q = it % 5, gs = p.s0 + so + s;
                if (gs >= p.s_end) continue;
                const char *first = reinterpret_cast<const char *>(cols[c] + plane * gs + y_first);
                const char *last = reinterpret_cast<const char *>(cols[c] + plane * gs + y_last);
                const uintptr_t line = ((uintptr_t)first >> 7) + (uintptr_t)q;
                if (line > ((uintptr_t)last >> 7)) continue;
                const char *a = q == 0 ? first : reinterpret_cast<const char *>(line << 7);
                tc::prefetch_l2(a);
            }
        }
    };

    // ---- bulk-copy ring; chunk ci = k * kc + q of step k --------------------
    // Three threads drive it: the copy threads (kCopyTid for A, kCopyBTid for
    // B) refill each stage as soon as the MMAs that read it have completed,
    // and thread 0 issues each chunk's MMAs as soon as its copies have landed,
    // so none waits on another's latency.  Chunk ci's stage is slot ci %
    // stages, used for the (ci / stages)-th time; each thread counts its slots
    // and phases along.  Up to N = 128 the ring is bound by what these threads
    // do per stage rather than by bytes or products.  With divisions by kc and
    // the ring's length per chunk, and the timer read in each wait, a step's
    // ring took 13.3 us at 552^2 (256 sources, TF32 and BF16 steps averaged),
    // 9.9 at 437 x 401 (97) and 6.6 at 288^2 (64), and 12.0, 9.1 and 6.0 in the
    // boundary chain (16); now 11.0, 6.3 and 3.7, and 5.8, 4.6 and 3.4.  An L2
    // prefetch of the next step's pages while this one's results are finished:
    // TF32 steps 4 % slower.
    int c_slot = 0, c_q = 0, a_k = 0;                            // a copy thread's next chunk; thread 0: the next MMAs
    uint32_t c_next = 0, c_phase = 0;
    const uint8_t *a_src = nullptr;
    // the page stream passes through L2 once; the packed B is read by every
    // CTA of the group and should stay
    const uint64_t policy = tid == kCopyTid && kind != K_BOUND ? tc::policy_evict_first() : tc::policy_evict_last();
    auto advance = [&]() {
        ++c_next;
        if (++c_slot == stages) { c_slot = 0; c_phase ^= 1u; }
    };
    // the next chunk of a copy thread may go into its stage
    auto stage_free = [&]() { return c_next < (uint32_t)stages || tc::mbar_wait(&empty[c_slot], c_phase ^ 1u, p.timeout_ns); };
    // A: stages up to `end`
    auto copies_a = [&](uint32_t end) {
        while (c_next < end) {
            if (!stage_free()) {
                atomicCAS(p.err, 0, SITE_COPY);
                return;
            }
            if (c_q == 0) a_src = apage(a_k++) + (size_t)t * kc * tc::kAChunk;
            const uint32_t bytes = (uint32_t)min(G, kc - c_q) * (uint32_t)tc::kAChunk;
            tc::mbar_expect_tx(&full[c_slot], bytes);
            tc::bulk_g2s_hint(sA + c_slot * (G * (uint32_t)tc::kAChunk), a_src, bytes, &full[c_slot], policy);
            a_src += bytes;
            c_q += G;
            if (c_q >= kc) c_q = 0;
            advance();
        }
    };
    // B: every stage of a step
    auto copies_b = [&]() {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the copies land where the state was staged
        const uint8_t *src = bg;
        for (int q = 0; q < kc; q += G) {
            if (!stage_free()) {
                atomicCAS(p.err, 0, SITE_COPY);
                return;
            }
            const uint32_t bytes = (uint32_t)min(G, kc - q) * (uint32_t)bbytes;
            tc::mbar_expect_tx(&full[c_slot], bytes);
            tc::bulk_g2s_hint(sB + c_slot * (G * (uint32_t)bbytes), src, bytes, &full[c_slot], policy);
            src += bytes;
            advance();
        }
    };

    unsigned epoch = 0;
    bool ok = nsteps > 0;
    if (ok) {
        if (tid == kCopyTid) copies_a((uint32_t)min(stages, kg));      // the first A chunks of step 0
        int in0 = IN_ZERO, mode0 = P_STENCIL;
        const float *pl0 = nullptr;
        if (kind == K_EXACT && chunk > 0) {
            in0 = IN_PLANES;
            pl0 = bstate(chunk - 1);
            if (ADJ) mode0 = P_IDENT;                      // the incoming state is this chunk's first B
        } else if (kind == K_EXACT && p.half == 1) {
            in0 = IN_UCOL;
        } else if (kind == K_PROP) {
            in0 = IN_IDENT;
        } else if (kind == K_BOUND) {
            in0 = IN_PLANES;
            pl0 = bstate(0);
            mode0 = P_IDENT;
        } else if (kind == K_LOCAL && ADJ) {
            mode0 = P_IDENT;                               // first B = 0
        }
        stage_in(in0, pl0);
        produce(0, mode0, nullptr, false);
        epoch += (unsigned)p.mt;
        ok = counter_sync(ctr, epoch, p.err, s_ok, p.timeout_ns, SITE_B);
    }
    float *cur = kind == K_BOUND ? nullptr : p.zst + (size_t)chunk * sfl;
    constexpr int kMmaPerChunk = tc::kChunkBytes / 32;
    const uint32_t idesc = tc::instr_desc<!BF>(tc::kTileRows, N);
    const uint64_t desc_a = tc::smem_desc(sA), desc_b = tc::smem_desc(sB);

#ifdef WUST_CHUNK_PROFILE
    long long prof_t = clock64();
    if (blockIdx.x == 0 && tid == 0) g_chunk_prof[p.pass][7] += (unsigned long long)nsteps;
#endif
    for (int k = 0; k < nsteps && ok; ++k) {
        CPROF(6);
        // this step's chunks, and the next one's first A chunks as stages free up
        if (tid == kCopyTid)
            copies_a(min((uint32_t)min(k + 2, nsteps) * (uint32_t)kg, (uint32_t)(k + 1) * (uint32_t)kg + (uint32_t)stages));
        if (tid == kCopyBTid) copies_b();
        if (tid == 0) {
            bool good = true;
            auto chunk_mmas = [&](uint32_t da, uint32_t db, bool first) {
#pragma unroll
                for (int kk = 0; kk < kMmaPerChunk; ++kk)
                    tc::mma<!BF>(tmem, tc::desc_at(da + kk * 16, desc_a), tc::desc_at(db + kk * 16, desc_b), idesc,
                                 first && kk == 0 ? 0u : 1u);
            };
            const uint32_t step_a = G * (uint32_t)(tc::kAChunk / 16), step_b = G * (uint32_t)(bbytes / 16);
            uint32_t da = (uint32_t)desc_a + c_slot * step_a, db = (uint32_t)desc_b + c_slot * step_b;
            for (int q = 0; q < kc; q += G) {
                if (!tc::mbar_wait(&full[c_slot], c_phase, p.timeout_ns)) { good = false; break; }
                tc::fence_after();
                chunk_mmas(da, db, q == 0);
                if (G > 1)
                    for (int i = 1; i < min(G, kc - q); ++i)
                        chunk_mmas(da + i * (uint32_t)(tc::kAChunk / 16), db + i * (uint32_t)(bbytes / 16), false);
                tc::commit(&empty[c_slot]);
                advance();
                da = c_slot ? da + step_a : (uint32_t)desc_a;
                db = c_slot ? db + step_b : (uint32_t)desc_b;
            }
            tc::commit(done);
            if (!good) atomicCAS(p.err, 0, SITE_COPY);
        }
        if (warp >= 1 && tid != kCopyTid && tid != kCopyBTid) prefetch_cols(k);
        if (warp == 1 || warp == 2) {
            const bool next_b = k + 1 < nsteps || (ADJ && p.pass == CK_FIRST && chunk + 1 < p.C);
            if (next_b) {
                bool f1 = false;
                const int j1 = col_of(k + 1, f1);
                fill_weights(tid - 32, kind == K_BOUND, f1, j1);
            }
        }
        CPROF(0);
        if (!tc::mbar_wait(done, (uint32_t)(k & 1), p.timeout_ns)) atomicCAS(p.err, 0, SITE_MMA);
        tc::fence_after();
        if (tid == 0) *s_ok = (*(volatile int *)p.err == 0);
        __syncthreads();
        if (!*s_ok) {
            ok = false;
            break;
        }
        float *curp = kind == K_BOUND ? bstate(t0 + k) : cur;
        CPROF(1);
        drain_tmem();
        tc::fence_before();
        finish(k, curp, kind == K_BOUND || k + 1 == nsteps);
        CPROF(2);
        epoch += (unsigned)p.mt;
        if (!counter_sync(ctr, epoch, p.err, s_ok, p.timeout_ns, SITE_GROUP)) {
            ok = false;
            break;
        }
        tc::fence_after();
        CPROF(3);
        if (k + 1 < nsteps) {
            stage_halo();
            CPROF(5);
            produce(k + 1, kind == K_BOUND ? P_IDENT : P_STENCIL, nullptr, true);
            CPROF(4);
            epoch += (unsigned)p.mt;
            if (!counter_sync(ctr, epoch, p.err, s_ok, p.timeout_ns, SITE_B)) {
                ok = false;
                break;
            }
        } else if (kind == K_EXACT && ADJ && p.half == 0 && t0 + k == nx - 2) {
            stage_halo();
            produce(k, P_TURN, nullptr, false);
        } else if (ADJ && p.pass == CK_FIRST && chunk + 1 < p.C) {
            // outgoing B state of the chunk: the first B of the next chunk
            stage_halo();
            produce(k + 1, P_STENCIL, bstate(chunk), true);
        }
    }

    // copies issued but never waited for (a failure, in which one of the two
    // may have stopped short): stand in for those that will not come, then let
    // the others land (bounded)
    if (tid == kCopyTid) s_ring[0] = c_next;
    if (tid == kCopyBTid) s_ring[1] = c_next;
    __syncthreads();
    if (tid == 0) {
        for (; c_next < max(s_ring[0], s_ring[1]); advance()) {
            for (int h = 0; h < 2; ++h)
                if (c_next >= s_ring[h]) tc::mbar_arrive(&full[c_slot]);
            tc::mbar_wait(&full[c_slot], c_phase, p.timeout_ns);
        }
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    if (warp == 0) tc::tmem_dealloc(tmem, tcols);
}

// -Lambda_c (columns [s0, s_end) of the propagators of chunks 1 .. C-2, in
// the state planes) -> packed [Ar -Ai; Ai Ar] A pages of the boundary steps
// (page c), and the rows [s0, s_end) of -Lambda_c^H -> the pages C-1-c of the
// H^H boundary steps.  BF: BF16 pages (32 complex columns per K chunk).
template <bool BF>
__global__ void pack_lambda_kernel(const float *zst, size_t sfl, int ny, int n, int mt, int kc, size_t page_bytes,
                                   int s0, int s_end, int C, uint8_t *lpack, uint8_t *lpack_h) {
    constexpr int RPC = BF ? kCkRowsPerChunk16 : kCkRowsPerChunk;   // complex columns per chunk
    constexpr int CPU = RPC / 8;                                      // complex columns per 16-byte unit
    const int i_s = threadIdx.x;                     // stacked row 0..127
    const int Q = blockIdx.x;                        // K chunk
    const int m = blockIdx.y;                        // M tile
    const int c = 1 + blockIdx.z;                    // chunk
    const int i = m * 64 + (i_s & 63);
    const bool imrow = i_s >= 64;
    const float *pl = zst + (size_t)c * sfl;
    auto store = [&](uint8_t *dst, int u, const float (&v)[2 * CPU]) {
        if (BF) {
            uint32_t w[CPU];
#pragma unroll
            for (int h = 0; h < CPU; ++h)
                w[h] = (uint32_t)tc::to_bf16_bits(v[2 * h]) | ((uint32_t)tc::to_bf16_bits(v[2 * h + 1]) << 16);
            *reinterpret_cast<uint4 *>(dst + tc::chunk_off16(i_s, 8 * u)) = make_uint4(w[0], w[1], w[2 % CPU], w[3 % CPU]);
        } else {
            *reinterpret_cast<float4 *>(dst + chunk_off(i_s, 4 * u)) =
                make_float4(to_tf32(v[0]), to_tf32(v[1]), to_tf32(v[2 % (2 * CPU)]), to_tf32(v[3 % (2 * CPU)]));
        }
    };
    // direct: A(i, k) = -Lambda(i, k) for K columns k in [s0, s_end)
    if ((Q * RPC < s_end || s_end >= n) && (Q + 1) * RPC > s0) {
        uint8_t *dst = lpack + (size_t)c * page_bytes + ((size_t)m * kc + Q) * tc::kAChunk;
#pragma unroll 2
        for (int u = 0; u < 8; ++u) {
            const int kk = Q * RPC + CPU * u;          // K columns kk .. kk+CPU-1 (the last tile also zeroes the padding)
            if (!(kk + CPU - 1 >= s0 && (kk < s_end || s_end >= n))) continue;
            float v[2 * CPU];
#pragma unroll
            for (int h = 0; h < CPU; ++h) {
                const int k = kk + h;
                float2 a = make_float2(0.f, 0.f);
                if (i < n && k >= s0 && k < s_end) {
                    const int sc = k - s0;
                    a = make_float2(-pl[(size_t)sc * ny + i + 1], -pl[(size_t)(kCkMaxN + sc) * ny + i + 1]);
                }
                v[2 * h] = imrow ? a.y : a.x;
                v[2 * h + 1] = imrow ? a.x : -a.y;
            }
            store(dst, u, v);
        }
    }
    // conjugate transpose: A(i, k) = -conj(Lambda(k, i)) for rows i in [s0, s_end)
    if (m * 64 >= s0 && m * 64 < s_end) {
        uint8_t *dst = lpack_h + (size_t)(C - 1 - c) * page_bytes + ((size_t)m * kc + Q) * tc::kAChunk;
#pragma unroll 2
        for (int u = 0; u < 8; ++u) {
            float v[2 * CPU];
#pragma unroll
            for (int h = 0; h < CPU; ++h) {
                const int k = Q * RPC + CPU * u + h;
                float2 a = make_float2(0.f, 0.f);
                if (i < n && i < s_end && k < n) {
                    const int sc = i - s0;
                    a = make_float2(-pl[(size_t)sc * ny + k + 1], pl[(size_t)(kCkMaxN + sc) * ny + k + 1]);
                }
                v[2 * h] = imrow ? a.y : a.x;
                v[2 * h + 1] = imrow ? a.x : -a.y;
            }
            store(dst, u, v);
        }
    }
}

// invT pages -> BF16 packed [Ar -Ai; Ai Ar] operands of invT_j and invT_j^H
// (32 complex columns per K chunk).  One thread per (row of the 128-row tile,
// chunk, M tile, page).
__global__ void pack_invT16_kernel(const float2 *__restrict__ invT, int ny, int n, int mt, int kc, size_t page_bytes,
                                   uint8_t *afwd, uint8_t *aadj) {
    const int i_s = threadIdx.x;
    const int c = blockIdx.x, m = blockIdx.y, j = blockIdx.z;
    const int i = m * 64 + (i_s & 63);
    const bool imrow = i_s >= 64;
    const size_t off = (size_t)j * page_bytes + ((size_t)m * kc + c) * tc::kAChunk;
    const float2 *page = invT + (size_t)j * ny * ny;
#pragma unroll 2
    for (int u = 0; u < 8; ++u) {
        uint32_t wf[4], wa[4];
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const int k = c * kCkRowsPerChunk16 + 4 * u + h;
            float2 af = make_float2(0.f, 0.f), aa = af;
            if (i < n && k < n) {
                af = page[(size_t)(i + 1) + (size_t)ny * (k + 1)];
                const float2 at = page[(size_t)(k + 1) + (size_t)ny * (i + 1)];
                aa = make_float2(at.x, -at.y);
            }
            const float f0 = imrow ? af.y : af.x, f1 = imrow ? af.x : -af.y;
            const float a0 = imrow ? aa.y : aa.x, a1 = imrow ? aa.x : -aa.y;
            wf[h] = (uint32_t)tc::to_bf16_bits(f0) | ((uint32_t)tc::to_bf16_bits(f1) << 16);
            wa[h] = (uint32_t)tc::to_bf16_bits(a0) | ((uint32_t)tc::to_bf16_bits(a1) << 16);
        }
        *reinterpret_cast<uint4 *>(afwd + off + tc::chunk_off16(i_s, 8 * u)) = make_uint4(wf[0], wf[1], wf[2], wf[3]);
        *reinterpret_cast<uint4 *>(aadj + off + tc::chunk_off16(i_s, 8 * u)) = make_uint4(wa[0], wa[1], wa[2], wa[3]);
    }
}

// Both packings in one pass: each thread reads the 32 complex values of its
// row in a BF16 K chunk and their transposes once, and writes the BF16 chunk
// and the two TF32 chunks (16 complex columns each) it covers, for invT_j
// and invT_j^H.  Same layouts as pack_invT_kernel and pack_invT16_kernel.
__global__ void pack_invT_both_kernel(const float2 *__restrict__ invT, int ny, int n, int mt, int kc, int kc16,
                                      size_t page_bytes16, uint8_t *afwd, uint8_t *aadj, uint8_t *afwd16,
                                      uint8_t *aadj16) {
    const int i_s = threadIdx.x;
    const int c16 = blockIdx.x, m = blockIdx.y, j = blockIdx.z;
    const int i = m * 64 + (i_s & 63);
    const bool imrow = i_s >= 64;
    const size_t off16 = (size_t)j * page_bytes16 + ((size_t)m * kc16 + c16) * tc::kAChunk;
    const float2 *page = invT + (size_t)j * ny * ny;
#pragma unroll 2
    for (int u = 0; u < 8; ++u) {                   // complex columns 4u .. 4u + 3 of the BF16 chunk
        uint32_t wf[4], wa[4];
        float vf[8], va[8];
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const int k = c16 * kCkRowsPerChunk16 + 4 * u + h;
            float2 af = make_float2(0.f, 0.f), aa = af;
            if (i < n && k < n) {
                af = page[(size_t)(i + 1) + (size_t)ny * (k + 1)];                  // invT(i, k)
                const float2 at = page[(size_t)(k + 1) + (size_t)ny * (i + 1)];     // invT(k, i)
                aa = make_float2(at.x, -at.y);                                      // invT^H(i, k)
            }
            const float f0 = imrow ? af.y : af.x, f1 = imrow ? af.x : -af.y;
            const float a0 = imrow ? aa.y : aa.x, a1 = imrow ? aa.x : -aa.y;
            wf[h] = (uint32_t)tc::to_bf16_bits(f0) | ((uint32_t)tc::to_bf16_bits(f1) << 16);
            wa[h] = (uint32_t)tc::to_bf16_bits(a0) | ((uint32_t)tc::to_bf16_bits(a1) << 16);
            vf[2 * h] = tc::to_tf32(f0);
            vf[2 * h + 1] = tc::to_tf32(f1);
            va[2 * h] = tc::to_tf32(a0);
            va[2 * h + 1] = tc::to_tf32(a1);
        }
        *reinterpret_cast<uint4 *>(afwd16 + off16 + tc::chunk_off16(i_s, 8 * u)) = make_uint4(wf[0], wf[1], wf[2], wf[3]);
        *reinterpret_cast<uint4 *>(aadj16 + off16 + tc::chunk_off16(i_s, 8 * u)) = make_uint4(wa[0], wa[1], wa[2], wa[3]);
        const int c = 2 * c16 + u / 4;               // TF32 chunk of these columns
        if (c < kc) {
            const size_t off = (((size_t)j * mt + m) * kc + c) * tc::kAChunk;
            const int ke = 8 * (u % 4);
            *reinterpret_cast<float4 *>(afwd + off + tc::chunk_off(i_s, ke)) = make_float4(vf[0], vf[1], vf[2], vf[3]);
            *reinterpret_cast<float4 *>(afwd + off + tc::chunk_off(i_s, ke + 4)) = make_float4(vf[4], vf[5], vf[6], vf[7]);
            *reinterpret_cast<float4 *>(aadj + off + tc::chunk_off(i_s, ke)) = make_float4(va[0], va[1], va[2], va[3]);
            *reinterpret_cast<float4 *>(aadj + off + tc::chunk_off(i_s, ke + 4)) = make_float4(va[4], va[5], va[6], va[7]);
        }
    }
}

void tc_pack_invT_both(const float2 *invT, int ny, int nx, const TcChunkGeom &g, uint8_t *afwd, uint8_t *aadj,
                       uint8_t *afwd16, uint8_t *aadj16, cudaStream_t st) {
    const dim3 grid(g.kc16, g.mt, nx);
    pack_invT_both_kernel<<<grid, 128, 0, st>>>(invT, ny, g.n, g.mt, g.kc, g.kc16, g.page_bytes16, afwd, aadj, afwd16,
                                                aadj16);
    ++g_kernel_launches;
    WUST_LAUNCH_CHECK();
}

void tc_pack_invT16(const float2 *invT, int ny, int nx, const TcChunkGeom &g, uint8_t *afwd16, uint8_t *aadj16,
                    cudaStream_t st) {
    const dim3 grid(g.kc16, g.mt, nx);
    pack_invT16_kernel<<<grid, 128, 0, st>>>(invT, ny, g.n, g.mt, g.kc16, g.page_bytes16, afwd16, aadj16);
    ++g_kernel_launches;
    WUST_LAUNCH_CHECK();
}

static void ck_configure() {
    // called before every launch: the attribute lives in the current
    // device's context, which a caller may switch or reset between calls
    WUST_CUDA(cudaFuncSetAttribute(tc_chunk_kernel<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCkSmem));
    WUST_CUDA(cudaFuncSetAttribute(tc_chunk_kernel<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCkSmem));
    WUST_CUDA(cudaFuncSetAttribute(tc_chunk_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCkSmem));
    WUST_CUDA(cudaFuncSetAttribute(tc_chunk_kernel<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCkSmem));
}

int tc_chunk_max_ctas() {
    ck_configure();
    int dev = 0, sms = 0, per_sm = 0;
    WUST_CUDA(cudaGetDevice(&dev));
    WUST_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    WUST_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, tc_chunk_kernel<false, false>, kCkThreads, kCkSmem));
    return sms * per_sm;
}

static ChunkParams base_params(const Coefs<float2> &co, const TcChunkGeom &g, const TcChunkBuffers &b) {
    ChunkParams p{};
    p.page_bytes = g.page_bytes;
    p.co = co;
    p.bglob = b.bglob;
    p.zst = b.zst;
    p.sb = b.sb;
    p.edges = b.edges;
    p.group_ctr = b.sync;
    p.err = b.err;
    p.ny = co.ny;
    p.nx = co.nx;
    p.n = g.n;
    p.mt = g.mt;
    p.kc = g.kc;
    p.C = g.C;
    p.timeout_ns = 1000000000ull;
    return p;
}

// Chunk bounds (first step within the half) of one substitution.  The
// forward substitutions cut the columns at F[c] = c (nx-1) / C; the backward
// ones mirror the cuts so that the composed propagators of the H^H
// substitutions (which carry B states) are the conjugate transposes of those
// of the H substitutions: H backward chunk C-1-c covers the pages of the H^H
// forward chunk c, H^H backward chunk C-1-c the columns of H forward chunk c.
static void set_bounds(ChunkParams &p, int C, bool adjoint, int half) {
    const int steps = p.nx - 1;
    auto F = [&](int c) { return (int)((long long)c * steps / C); };
    for (int c = 0; c <= C; ++c) {
        if (half == 0) p.bounds[c] = F(c);
        else if (!adjoint) p.bounds[c] = steps - F(C - c);
        else p.bounds[c] = (c == 0 || c == C) ? (c == 0 ? 0 : steps) : steps - 1 - F(C - c);
    }
}

static void ck_launch(ChunkParams &p, bool adjoint, bool bf16, int pass, int groups, cudaStream_t st) {
    if (groups <= 0) return;
    p.pass = pass;
    const CkRing ring = ck_ring(p.N);
    p.per_stage = ring.per_stage;
    p.stages = ring.stages;
    WUST_CUDA(cudaMemsetAsync(p.group_ctr, 0, sizeof(unsigned) * groups, st));
    void *args[] = {&p};
    const dim3 grid(groups * p.mt), block(kCkThreads);
    void *fn = adjoint ? (bf16 ? (void *)tc_chunk_kernel<true, true> : (void *)tc_chunk_kernel<true, false>)
                       : (bf16 ? (void *)tc_chunk_kernel<false, true> : (void *)tc_chunk_kernel<false, false>);
    WUST_CUDA(cudaLaunchCooperativeKernel(fn, grid, block, args, kCkSmem, st));
    ++g_kernel_launches;
}

static uint8_t *lpack_of(const TcChunkGeom &g, uint8_t *lpack, bool adjoint, int half, size_t page_bytes) {
    return lpack + (size_t)((adjoint ? 2 : 0) + half) * g.C * page_bytes;
}

void tc_chunk_prepare(const Coefs<float2> &co, const uint8_t *afwd, const uint8_t *aadj, const TcChunkGeom &g,
                      const TcChunkBuffers &b, cudaStream_t st) {
    (void)aadj;
    ck_configure();
    if (g.C < 3) return;
    ChunkParams p = base_params(co, g, b);
    const size_t sfl = tc_chunk_state_floats(co.ny);
    p.apack = afwd;
    for (int half = 0; half < 2; ++half) {
        p.half = half;
        set_bounds(p, g.C, false, half);
        uint8_t *lp = lpack_of(g, b.lpack, false, half, g.page_bytes);
        uint8_t *lph = lpack_of(g, b.lpack, true, 1 - half, g.page_bytes);
        for (int s0 = 0, N = 0; s0 < g.n; s0 += N) {
            // source tiles of whole 64-row M tiles (the transposed pack fills M tiles)
            N = std::min(kCkMaxN, ceil_div(g.n - s0, 64) * 64);
            p.s0 = s0;
            p.s_end = std::min(g.n, s0 + N);
            p.N = N;
            ck_launch(p, false, false, CK_PROP, g.C - 2, st);
            const dim3 grid(g.kc, g.mt, g.C - 2);
            pack_lambda_kernel<false><<<grid, 128, 0, st>>>(b.zst, sfl, co.ny, g.n, g.mt, g.kc, g.page_bytes, s0,
                                                            p.s_end, g.C, lp, lph);
            ++g_kernel_launches;
            if (b.lpack16) {
                const dim3 grid16(g.kc16, g.mt, g.C - 2);
                pack_lambda_kernel<true><<<grid16, 128, 0, st>>>(
                    b.zst, sfl, co.ny, g.n, g.mt, g.kc16, g.page_bytes16, s0, p.s_end, g.C,
                    lpack_of(g, b.lpack16, false, half, g.page_bytes16), lpack_of(g, b.lpack16, true, 1 - half, g.page_bytes16));
                ++g_kernel_launches;
            }
        }
    }
    WUST_LAUNCH_CHECK();
}

void tc_chunk_solve(const Coefs<float2> &co, const uint8_t *afwd, const uint8_t *aadj, const TcChunkGeom &g,
                    const TcChunkBuffers &b, const SrcView &src, int S, bool adjoint, float2 *u, bool bf16,
                    cudaStream_t st) {
    ck_configure();
    const int ny = co.ny, nx = co.nx;
    WUST_CUDA(cudaMemsetAsync(u, 0, sizeof(float2) * (size_t)ny * nx * S, st));
    ChunkParams p = base_params(co, g, b);
    p.apack = adjoint ? aadj : afwd;
    if (bf16) {
        p.kc = g.kc16;
        p.page_bytes = g.page_bytes16;
    }
    p.src = src;
    p.u = u;
    for (int s0 = 0; s0 < S; s0 += kCkMaxN) {
        p.s0 = s0;
        p.s_end = std::min(S, s0 + kCkMaxN);
        p.N = ceil_div(p.s_end - s0, 16) * 16;
        for (int half = 0; half < 2; ++half) {
            p.half = half;
            set_bounds(p, g.C, adjoint, half);
            p.lpack = bf16 ? lpack_of(g, b.lpack16, adjoint, half, g.page_bytes16)
                           : lpack_of(g, b.lpack, adjoint, half, g.page_bytes);
            ck_launch(p, adjoint, bf16, CK_FIRST, g.C, st);
            if (g.C >= 3) {
                // the chain of C - 2 dense steps on up to C groups, each
                // carrying a 16-multiple slice of the sources (one group
                // would leave all but mt SMs idle for the whole chain)
                const int N = p.N;
                const int per = ceil_div(ceil_div(N, g.C), 16) * 16;
                p.N = per;
                ck_launch(p, adjoint, bf16, CK_BOUNDARY, ceil_div(N, per), st);
                p.N = N;
            }
            if (g.C >= 2) ck_launch(p, adjoint, bf16, CK_SECOND, g.C - 1, st);
        }
    }
    WUST_LAUNCH_CHECK();
}

}  // namespace wust
