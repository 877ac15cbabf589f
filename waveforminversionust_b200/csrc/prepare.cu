// The DTFT of the RF preparation, Runtime/matlab/wust_prepare.m:30-37:
//     Y(tx, rx, k) = single( sum_t exp(-2 pi i f_k t) dt * rf(t, rx, tx) )
// over the sample times t of the record, FP64 phases and accumulation, with
// the traces of inactive channels taken as zero (the reference zeroes them
// before the product, so non-finite samples there do not matter).
//
// It is one real x complex GEMM, Y^T (traces x nf) = RF^T (traces x nt) K^T,
// bound by its FP64 multiply-adds (64 per clock and SM on this part, scalar
// or through the FP64 matrix instruction; the RF stream would take a third of
// their time at 16 frequencies).  Two kernels:
//   * evenly spaced samples (dtft_fold_kernel): folded about the middle of
//     the record, x(+m) + x(-m) meets the cosines and x(+m) - x(-m) the
//     sines of omega times the distance from the middle, which halves the
//     multiply-adds; a rotation by the middle's phase ends it;
//   * any other times (dtft_kernel): a block takes 64 traces, stages 32-sample
//     slabs of them and of the phase matrix K (nf x nt) in shared memory, and
//     every thread accumulates 2 traces x 4 frequencies in complex double.
//     Frequencies beyond 32 are done in further passes over the traces.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "kernels.cuh"

namespace wust {

constexpr int kDtTraces = 64;      // traces per block
constexpr int kDtSamples = 32;     // samples per slab
constexpr int kDtFreqs = 32;       // frequencies per pass
constexpr int kDtThreads = 256;    // 32 trace pairs x 8 frequency quads

// K(k, t) = exp(-2 pi i f_k t) * dt, arguments formed as ((-2 pi) f_k) t
__global__ void dtft_phase_kernel(const double *time_s, const double *freq, int nt, int nf, double dt, double2 *K) {
    const size_t total = (size_t)nf * nt;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int k = (int)(i / nt), t = (int)(i % nt);
        const double arg = (-2.0 * M_PI * freq[k]) * time_s[t];
        double s, c;
        sincos(arg, &s, &c);
        K[i] = make_double2(c * dt, s * dt);
    }
}

template <typename T>
__global__ void __launch_bounds__(kDtThreads) dtft_kernel(const T *rf, const uint8_t *active, const double2 *K, int nt,
                                                         int nf, int n_rx, int n_tx, float2 *Y, int *bad) {
    __shared__ double sp[kDtSamples][kDtTraces + 1];        // rf(t, trace)
    __shared__ double2 sk[kDtSamples][kDtFreqs];            // K(k, t)
    const int n_tr = n_rx * n_tx;
    const int tr0 = blockIdx.x * kDtTraces;
    const int k0 = blockIdx.y * kDtFreqs;
    const int tid = threadIdx.x;
    const int tp = tid & 31, fq = tid >> 5;                // traces 2 tp, 2 tp + 1; frequencies 4 fq .. 4 fq + 3
    double2 acc[2][4];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = make_double2(0.0, 0.0);
    int nonfinite = 0;
    for (int t0 = 0; t0 < nt; t0 += kDtSamples) {
        // rf slab: 64 traces x 32 samples, samples fastest (coalesced)
        for (int e = tid; e < kDtTraces * kDtSamples; e += kDtThreads) {
            const int ts = e % kDtSamples, tr = e / kDtSamples;
            const int t = t0 + ts, g = tr0 + tr;
            double v = 0.0;
            if (t < nt && g < n_tr && active[(g / n_rx) + (size_t)n_tx * (g % n_rx)]) {
                v = (double)rf[(size_t)t + (size_t)nt * g];
                if (!isfinite(v)) {
                    nonfinite = 1;
                    v = 0.0;
                }
            }
            sp[ts][tr] = v;
        }
        for (int e = tid; e < kDtFreqs * kDtSamples; e += kDtThreads) {
            const int ts = e % kDtSamples, kk = e / kDtSamples;
            const int t = t0 + ts, k = k0 + kk;
            sk[ts][kk] = (t < nt && k < nf) ? K[(size_t)k * nt + t] : make_double2(0.0, 0.0);
        }
        __syncthreads();
#pragma unroll 4
        for (int ts = 0; ts < kDtSamples; ++ts) {
            const double p0 = sp[ts][2 * tp], p1 = sp[ts][2 * tp + 1];
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const double2 kv = sk[ts][4 * fq + b];
                acc[0][b].x += kv.x * p0;
                acc[0][b].y += kv.y * p0;
                acc[1][b].x += kv.x * p1;
                acc[1][b].y += kv.y * p1;
            }
        }
        __syncthreads();
    }
    if (nonfinite) atomicExch(bad, 1);
    // Y(tx, rx, k), tx fastest; trace g = rx + n_rx tx
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        const int g = tr0 + 2 * tp + a;
        if (g >= n_tr) continue;
        const int rx = g % n_rx, tx = g / n_rx;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int k = k0 + 4 * fq + b;
            if (k < nf)
                Y[tx + (size_t)n_tx * (rx + (size_t)n_rx * k)] = make_float2((float)acc[a][b].x, (float)acc[a][b].y);
        }
    }
}

// ---------------------------------------------------------------------------
// Evenly spaced samples.  Sample pair m = 0 .. P-1 (P = ceil(nt / 2)) lies at
// distance d_m from the record's middle on both sides (an odd record's middle
// sample is paired with itself at weight 1/2); pairs go in blocks of 16.
//     Y = r_k (sum_m (x+ + x-) cos(2 pi f_k d_m) - i sum_m (x+ - x-) sin(2 pi f_k d_m)),
//     r_k = dt exp(-2 pi i f_k t_mid).
// Both sums are products of m8n8k4 FP64 matrix instructions: 8 traces x 4
// pairs times 4 pairs x 8 frequencies.  A thread's four pairs of a block are
// consecutive samples (one 16-byte load on each side), so the page of K that
// instruction j takes is pairs j, 4 + j, 8 + j, 12 + j of the block; the
// table of cosines and sines is laid out in that order, 32 lanes of a B
// fragment side by side.  A CTA stages the table in shared memory, eight
// blocks at a time; KW of its eight warps split the pairs of the same traces
// where there are too few traces to fill the GPU, and their sums are added in
// a fixed order.  Rows run along the transmitters, whose outputs are
// neighbours.
// 2048 x 256 x 256 samples in float32, 16 frequencies: 211 us, 55 % of the FP64 rate
// (the plain product
// on CUDA cores: 2144 us).
// ---------------------------------------------------------------------------
constexpr int kFoldWarps = 8, kFoldThreads = 32 * kFoldWarps;
constexpr int kFoldBlocks = 8;                            // blocks of 16 pairs per stage
constexpr int kFragDoubles = 4 * 2 * 32;                  // fragments of a block and 8 frequencies: 4 j, cos and sin
constexpr int kFoldMaxNb = 5;                             // frequency octets per pass
constexpr int kFoldParams = 256;                          // frequencies per table launch

struct FoldFreqs {
    double f[kFoldParams];
};

// table[block][octet][j][cos, sin][lane] and rot[k] for frequencies k0 .. k0 + nk - 1 (k0 a multiple of 8)
__global__ void dtft_table_kernel(const __grid_constant__ FoldFreqs fr, int k0, int nk, int nb_all, int blocks, int pairs,
                                  double half, double h, double t_mid, double dt, double *table, double2 *rot, int *bad) {
    if (blockIdx.x == 0 && threadIdx.x == 0 && k0 == 0) *bad = 0;
    const int octs = (nk + 7) / 8;
    const size_t total = (size_t)blocks * octs * 4 * 32;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int lane = (int)(i % 32), j = (int)(i / 32 % 4), o = (int)(i / 128 % octs), b = (int)(i / 128 / octs);
        const int m = 16 * b + 4 * (lane & 3) + j, k = 8 * o + (lane >> 2);
        double s = 0.0, c = 0.0;
        if (m < pairs && k < nk) {
            sincos(2.0 * M_PI * fr.f[k] * ((m + half) * h), &s, &c);
            if (half == 0.0 && m == 0) c = 0.5;           // the middle sample, paired with itself
        }
        double *dst = table + (((size_t)b * nb_all + k0 / 8 + o) * 4 + j) * 64 + lane;
        dst[0] = c;
        dst[32] = s;
    }
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nk; k += gridDim.x * blockDim.x) {
        double s, c;
        sincos((-2.0 * M_PI * fr.f[k]) * t_mid, &s, &c);
        rot[k0 + k] = make_double2(c * dt, s * dt);
    }
}

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};" : "+d"(c[0]), "+d"(c[1]) : "d"(a), "d"(b));
}

// four samples from p (16-byte loads where VEC)
template <typename T, bool VEC>
__device__ __forceinline__ void load4(T (&v)[4], const T *p) {
    if constexpr (VEC && sizeof(T) == 4) {
        const float4 q = __ldcs(reinterpret_cast<const float4 *>(p));
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    } else if constexpr (VEC) {
        const double2 q = __ldcs(reinterpret_cast<const double2 *>(p)), r = __ldcs(reinterpret_cast<const double2 *>(p) + 1);
        v[0] = q.x; v[1] = q.y; v[2] = r.x; v[3] = r.y;
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = p[i];
    }
}

struct FoldParams {
    const void *rf;
    const uint8_t *active;
    const double *table;
    const double2 *rot;
    float2 *Y;
    int *bad;
    int nt, pairs, blocks, nf, nb_all, nb0, n_rx, n_tx, kw;
};

template <typename T, int NB, int MT, bool VEC>
__global__ void __launch_bounds__(kFoldThreads, NB <= 2 ? 2 : 1) dtft_fold_kernel(FoldParams p) {
    extern __shared__ __align__(16) double fold_sm[];     // two stages [block][octet of the pass][j][cos, sin][lane]
    constexpr int kBlk = NB * kFragDoubles, kStage = kFoldBlocks * kBlk;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int kpart = warp % p.kw, groups = kFoldWarps / p.kw, n_tr = p.n_rx * p.n_tx;
    const int row0 = ((int)blockIdx.x * groups + warp / p.kw) * MT * 8;      // rows tx + n_tx rx
    const int nb0 = p.nb0 + (int)blockIdx.y * NB;
    auto stage = [&](int s) {
        const int b0 = s * kFoldBlocks;
        if (b0 < p.blocks) {
            double *dst = fold_sm + (s & 1) * kStage;
            const int nb_n = min(NB, p.nb_all - nb0), n16 = min(kFoldBlocks, p.blocks - b0) * nb_n * (kFragDoubles / 2);
            for (int e = tid; e < n16; e += kFoldThreads) {
                const int b = e / (nb_n * (kFragDoubles / 2)), r = e % (nb_n * (kFragDoubles / 2));
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                                 (unsigned)__cvta_generic_to_shared(dst + (size_t)b * kBlk + 2 * r)),
                             "l"(p.table + ((size_t)(b0 + b) * p.nb_all + nb0) * kFragDoubles + 2 * r) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // a thread's samples: of row lane / 4, pairs 16 b + 4 (lane % 4) .. + 3
    const int q4 = 4 * (lane & 3), plus0 = p.nt / 2, minus0 = (p.nt - 1) / 2;
    const T *x[MT];
#pragma unroll
    for (int t = 0; t < MT; ++t) {
        const int row = min(row0 + 8 * t + (lane >> 2), n_tr - 1);
        x[t] = static_cast<const T *>(p.rf) + (size_t)p.nt * ((size_t)(row / p.n_tx) + (size_t)p.n_rx * (row % p.n_tx));
    }
    T xp[2][MT][4], xm[2][MT][4];
    auto fetch = [&](int b, T (&vp)[MT][4], T (&vm)[MT][4]) {
        // beyond the last pair any samples do: the table is zero there
        const int m = 16 * b + q4;
        if (VEC) {
            const int mc = m + 3 < p.pairs ? m : 0;
#pragma unroll
            for (int t = 0; t < MT; ++t) {
                load4<T, VEC>(vp[t], x[t] + plus0 + mc);
                load4<T, VEC>(vm[t], x[t] + minus0 - mc - 3);
            }
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int mc = min(m + i, p.pairs - 1);
#pragma unroll
                for (int t = 0; t < MT; ++t) {
                    vp[t][i] = x[t][plus0 + mc];
                    vm[t][3 - i] = x[t][minus0 - mc];
                }
            }
        }
    };
    double ac[MT][NB][2], as[MT][NB][2];
#pragma unroll
    for (int t = 0; t < MT; ++t)
#pragma unroll
        for (int o = 0; o < NB; ++o) ac[t][o][0] = ac[t][o][1] = as[t][o][0] = as[t][o][1] = 0.0;
    unsigned worst[MT];                                   // exponent bits of the largest magnitude seen
#pragma unroll
    for (int t = 0; t < MT; ++t) worst[t] = 0;
    auto bits = [](T v) -> unsigned {
        if constexpr (sizeof(T) == 4) return __float_as_uint((float)v) & 0x7f800000u;
        else return (unsigned)(__double2hiint((double)v)) & 0x7ff00000u;
    };
    auto block = [&](const double *B, const T (&vp)[MT][4], const T (&vm)[MT][4]) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            double s[MT], d[MT];
#pragma unroll
            for (int t = 0; t < MT; ++t) {
                const double a = (double)vp[t][j], b = (double)vm[t][3 - j];
                s[t] = a + b;
                d[t] = a - b;
                worst[t] = max(worst[t], max(bits(vp[t][j]), bits(vm[t][j])));
            }
#pragma unroll
            for (int o = 0; o < NB; ++o) {
                const double bc = B[(o * 4 + j) * 64 + lane], bs = B[(o * 4 + j) * 64 + 32 + lane];
#pragma unroll
                for (int t = 0; t < MT; ++t) {
                    dmma(ac[t][o], s[t], bc);
                    dmma(as[t][o], d[t], bs);
                }
            }
        }
    };
    const int stages = (p.blocks + kFoldBlocks - 1) / kFoldBlocks;
    stage(0);
    int b = kpart, buf = 0;                               // this warp's blocks: kpart, kpart + kw, ...
    if (b < p.blocks) fetch(b, xp[0], xm[0]);
    if (b + p.kw < p.blocks) fetch(b + p.kw, xp[1], xm[1]);
    for (int s = 0; s < stages; ++s) {
        stage(s + 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        const double *S = fold_sm + (s & 1) * kStage;
        const int end = min((s + 1) * kFoldBlocks, p.blocks);
        for (; b < end; b += p.kw) {
            const double *B = S + (size_t)(b - s * kFoldBlocks) * kBlk;
            if (buf == 0) {
                block(B, xp[0], xm[0]);
                if (b + 2 * p.kw < p.blocks) fetch(b + 2 * p.kw, xp[0], xm[0]);
            } else {
                block(B, xp[1], xm[1]);
                if (b + 2 * p.kw < p.blocks) fetch(b + 2 * p.kw, xp[1], xm[1]);
            }
            buf ^= 1;
        }
        __syncthreads();                                  // the stage is read
    }
    if (p.kw > 1) {                                       // the parts of a group, added in order by the first
        double *mine = fold_sm + (size_t)warp * (MT * NB * 4 * 32) + lane;
#pragma unroll
        for (int t = 0; t < MT; ++t)
#pragma unroll
            for (int o = 0; o < NB; ++o)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    mine[((t * NB + o) * 4 + e) * 32] = ac[t][o][e];
                    mine[((t * NB + o) * 4 + 2 + e) * 32] = as[t][o][e];
                }
        __syncthreads();
        if (kpart == 0)
            for (int w = 1; w < p.kw; ++w) {
                const double *other = mine + (size_t)w * (MT * NB * 4 * 32);
#pragma unroll
                for (int t = 0; t < MT; ++t)
#pragma unroll
                    for (int o = 0; o < NB; ++o)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            ac[t][o][e] += other[((t * NB + o) * 4 + e) * 32];
                            as[t][o][e] += other[((t * NB + o) * 4 + 2 + e) * 32];
                        }
            }
    }
#pragma unroll
    for (int t = 0; t < MT; ++t) {
        const int row = row0 + 8 * t + (lane >> 2);
        if (row >= n_tr) continue;
        const bool on = p.active[row] != 0;
        if (on && worst[t] >= (sizeof(T) == 4 ? 0x7f800000u : 0x7ff00000u)) atomicExch(p.bad, 1);
        if (kpart != 0) continue;
        // accumulator columns 2 (lane % 4) and + 1 of every octet
#pragma unroll
        for (int o = 0; o < NB; ++o)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int k = 8 * (nb0 + o) + 2 * (lane & 3) + e;
                if (k >= p.nf) continue;
                const double2 z = zmul(p.rot[k], make_double2(ac[t][o][e], -as[t][o][e]));
                p.Y[row + (size_t)n_tr * k] = on ? make_float2((float)z.x, (float)z.y) : make_float2(0.f, 0.f);
            }
    }
}

// Whether the samples are evenly spaced to rounding: within 1e-11 of a step
// (the phase of a frequency below Nyquist is then off by less than 1e-10).
// Times more than some 45,000 steps from zero are not, by their own rounding in
// 64 bits: such a record takes the general kernel.
static bool evenly_spaced(const double *t, int nt, double &h) {
    h = (t[nt - 1] - t[0]) / (nt - 1);
    for (int i = 0; i < nt; ++i)
        if (!(std::fabs(t[i] - (t[0] + i * h)) <= 1e-11 * h)) return false;
    return true;
}

static int fold_blocks(int nt) { return ((nt + 1) / 2 + 15) / 16; }

// table (fold) or times, frequencies and K (plain), rot, the flag
size_t dtft_workspace_bytes(int nt, int nf) {
    const size_t nb = (nf + 7) / 8;
    const size_t fold = sizeof(double) * (size_t)fold_blocks(nt) * nb * kFragDoubles + sizeof(double2) * nb * 8;
    const size_t plain = sizeof(double) * ((size_t)nt + nf + 1) + sizeof(double2) * (size_t)nt * nf;
    return 256 + std::max(fold, plain);
}

template <typename T, int NB, int MT>
static void fold_launch(const FoldParams &p, bool vec, dim3 grid, cudaStream_t st) {
    constexpr size_t smem = sizeof(double) * 2 * kFoldBlocks * NB * kFragDoubles;
    auto go = [&](auto kernel) {
        WUST_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        kernel<<<grid, kFoldThreads, smem, st>>>(p);
    };
    if (vec) go(dtft_fold_kernel<T, NB, MT, true>);
    else go(dtft_fold_kernel<T, NB, MT, false>);
}
template <typename T>
static void fold_launch(const FoldParams &p, int nb, int mt, bool vec, dim3 grid, cudaStream_t st) {
    switch (nb * 2 + mt) {
        case 3: return fold_launch<T, 1, 1>(p, vec, grid, st);
        case 4: return fold_launch<T, 1, 2>(p, vec, grid, st);
        case 5: return fold_launch<T, 2, 1>(p, vec, grid, st);
        case 6: return fold_launch<T, 2, 2>(p, vec, grid, st);
        case 7: return fold_launch<T, 3, 1>(p, vec, grid, st);
        case 8: return fold_launch<T, 3, 2>(p, vec, grid, st);
        case 9: return fold_launch<T, 4, 1>(p, vec, grid, st);
        case 10: return fold_launch<T, 4, 2>(p, vec, grid, st);
        case 11: return fold_launch<T, 5, 1>(p, vec, grid, st);
        default: return fold_launch<T, 5, 2>(p, vec, grid, st);
    }
}

static void dtft_fold(const double *time_s, const double *freq, int nt, int nf, double h, double dt, const void *rf,
                      bool rf_double, int n_rx, int n_tx, const uint8_t *active, uint8_t *ws, float2 *Y, int *bad,
                      cudaStream_t st) {
    FoldParams p;
    p.rf = rf;
    p.active = active;
    p.Y = Y;
    p.bad = bad;
    p.nt = nt;
    p.pairs = (nt + 1) / 2;
    p.blocks = fold_blocks(nt);
    p.nf = nf;
    p.nb_all = ceil_div(nf, 8);
    p.nb0 = 0;
    p.n_rx = n_rx;
    p.n_tx = n_tx;
    double *table = reinterpret_cast<double *>(ws);
    double2 *rot = reinterpret_cast<double2 *>(table + (size_t)p.blocks * p.nb_all * kFragDoubles);
    p.table = table;
    p.rot = rot;
    const double half = nt % 2 ? 0.0 : 0.5, t_mid = time_s[0] + 0.5 * (nt - 1) * h;
    for (int k0 = 0; k0 < nf; k0 += kFoldParams) {
        FoldFreqs fr;
        const int nk = std::min(kFoldParams, nf - k0);
        for (int k = 0; k < kFoldParams; ++k) fr.f[k] = k < nk ? freq[k0 + k] : 0.0;
        const size_t total = (size_t)p.blocks * ceil_div(nk, 8) * 128;
        dtft_table_kernel<<<(int)std::min<size_t>((total + 127) / 128, 4096), 128, 0, st>>>(
            fr, k0, nk, p.nb_all, p.blocks, p.pairs, half, h, t_mid, dt, table, rot, bad);
        ++g_kernel_launches;
        WUST_LAUNCH_CHECK();
    }
    // the octets in passes over the traces, as evenly as they go
    const int passes = ceil_div(p.nb_all, kFoldMaxNb), nb = ceil_div(p.nb_all, passes);
    // 16-byte loads on both sides of the middle
    const bool vec = nt % 8 == 0 && (reinterpret_cast<uintptr_t>(rf) & 15) == 0;
    // warps on traces of their own (16 each) while that gives every SM two CTAs; then they split the pairs, then 8 each
    const int n_tr = n_rx * n_tx;
    int mt = 2, kw = 1;
    while (kw < kFoldWarps && ceil_div(n_tr, 8 * mt * (kFoldWarps / kw)) < 2 * 148) kw *= 2;
    if (kw == kFoldWarps && ceil_div(n_tr, 8 * mt) < 2 * 148) mt = 1;
    p.kw = kw;
    const dim3 grid(ceil_div(n_tr, 8 * mt * (kFoldWarps / kw)), passes);
    if (rf_double) fold_launch<double>(p, nb, mt, vec, grid, st);
    else fold_launch<float>(p, nb, mt, vec, grid, st);
    ++g_kernel_launches;
    WUST_LAUNCH_CHECK();
}

void dtft_launch(const double *time_s, const double *freq, int nt, int nf, double dt, const void *rf, bool rf_double,
                 int n_rx, int n_tx, const uint8_t *active, void *workspace, float2 *Y, int **bad_out, cudaStream_t st) {
    // the flag first, then the tables on 256 bytes
    int *bad = static_cast<int *>(workspace);
    uint8_t *ws = static_cast<uint8_t *>(workspace) + 256;
    *bad_out = bad;
    double h = 0.0;
    if (evenly_spaced(time_s, nt, h)) {
        dtft_fold(time_s, freq, nt, nf, h, dt, rf, rf_double, n_rx, n_tx, active, ws, Y, bad, st);
        return;
    }
    double *t_d = reinterpret_cast<double *>(ws), *f_d = t_d + nt;
    double2 *K = reinterpret_cast<double2 *>(f_d + nf + ((nt + nf) & 1));
    WUST_CUDA(cudaMemcpyAsync(t_d, time_s, sizeof(double) * nt, cudaMemcpyHostToDevice, st));
    WUST_CUDA(cudaMemcpyAsync(f_d, freq, sizeof(double) * nf, cudaMemcpyHostToDevice, st));
    WUST_CUDA(cudaMemsetAsync(bad, 0, sizeof(int), st));
    const size_t nk = (size_t)nf * nt;
    dtft_phase_kernel<<<(int)std::min<size_t>((nk + 255) / 256, 4096), 256, 0, st>>>(t_d, f_d, nt, nf, dt, K);
    ++g_kernel_launches;
    WUST_LAUNCH_CHECK();
    const dim3 grid(ceil_div((long long)n_rx * n_tx, kDtTraces), ceil_div(nf, kDtFreqs));
    if (rf_double)
        dtft_kernel<double><<<grid, kDtThreads, 0, st>>>(static_cast<const double *>(rf), active, K, nt, nf, n_rx,
                                                         n_tx, Y, bad);
    else
        dtft_kernel<float><<<grid, kDtThreads, 0, st>>>(static_cast<const float *>(rf), active, K, nt, nf, n_rx, n_tx,
                                                        Y, bad);
    ++g_kernel_launches;
    WUST_LAUNCH_CHECK();
}

}  // namespace wust
