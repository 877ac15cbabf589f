// RF simulation of Runtime/matlab/wust_simulate.m: the 2-D first-order
// k-space pseudospectral method of k-Wave (linear acoustics, scalar density,
// no absorption, Dirichlet pressure source, pressure sensors, PML outside
// the grid) for every transmitter of a record, batched on one GPU.
//
// The reference runs k-Wave's kspaceFirstOrder2D once per transmitter, or
// the vendored native solver (Runtime/third_party/kspaceFirstOrder-CUDA) over
// the batch.  Here all transmitters of a batch share one set of coefficient
// arrays and march together: the fields of S transmitters are S planes (x, y),
// and each time step is
//     P   = F(p)
//     G   = kappa D+ P / N     (y and x derivative)
//     g   = F^-1(G)
//     u   = pml_sg (pml_sg u - dt / rho0 g)
//     U   = F(u)
//     U  *= kappa D- / N
//     du  = F^-1(U)
//     rho = pml (pml rho - dt rho0 du); Dirichlet source; p = c^2 (rho_y +
//           rho_x); sensors recorded
// with the constants of the vendored solver (kappa = sinc(c_ref dt |k| / 2),
// D+- = i k exp(+-i k d / 2) on k-Wave's wavenumber vectors, PML factors
// exp(-dt / 2 * 2 * c_ref / d * (distance / pml)^4)).  Own transforms, fused
// with what stands between them; library transforms, one kernel between each
// two and the step in a CUDA graph where a length has a large prime.
// Optional FIR decimation of the records (downsampleKWaveChannelData.m:
// MATLAB resample(x, 1, q, 24, 8.6)) runs on the device at the end.
#include <cooperative_groups.h>
#include <cufft.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "kernels.cuh"
#include "simfft.cuh"

namespace wust {

namespace {

constexpr int kSimThreads = 256;

#define WUST_CUFFT(call)                                                                      \
    do {                                                                                      \
        cufftResult r_ = (call);                                                              \
        if (r_ != CUFFT_SUCCESS) ::wust::fail(WUST_ERR_CUDA, "%s failed (cuFFT %d)", #call, (int)r_); \
    } while (0)

struct SimGeom {
    int Ny, Nx;          // expanded grid
    int Nyh;             // Ny / 2 + 1 (R2C along y)
    int S;               // transmitters in the batch
    size_t plane, cplane;
};

struct SimCoefs {
    const float *kappa;          // [Nx][Nyh]
    const float2 *dyp, *dyn;     // [Nyh] i k_y exp(+-i k_y dy / 2)
    const float2 *dxp, *dxn;     // [Nx]
    const float *pmly, *pmly_sg; // [Ny]
    const float *pmlx, *pmlx_sg; // [Nx]
    const float *c2;             // [Nx][Ny]
    float inv_n;                 // 1 / (Ny Nx): cuFFT's inverse is unnormalised
    float dt_rho0, dt_over_rho0;
};

// k-Wave's wavenumber of index i of an axis of n points (ifftshifted
// -n/2 .. n/2-1 for even n, -(n-1)/2 .. (n-1)/2 for odd n).
double kwave_k(int i, int n, double d) {
    const int m = i <= (n - 1) / 2 ? i : i - n;
    return 2.0 * M_PI * m / (n * d);
}

double pml_value(int i, int n, int pml, double d, double dt, double c_ref, bool staggered) {
    const double a = -0.5 * dt * 2.0 * c_ref / d, sh = staggered ? 0.5 : 0.0;
    if (i < pml) return std::exp(a * std::pow((i + sh - pml) / (double)(-pml), 4));
    if (i >= n - pml) return std::exp(a * std::pow((i - (n - pml) + sh + 1.0) / pml, 4));
    return 1.0;
}

// G[0..S) = kappa D+_y P / N,  G[S..2S) = kappa D+_x P / N
__global__ void sim_grad_kernel(SimGeom g, SimCoefs k, const float2 *__restrict__ P, float2 *__restrict__ G) {
    const size_t total = (size_t)g.S * g.cplane;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const size_t e = i % g.cplane;
        const int iy = (int)(e % g.Nyh), ix = (int)(e / g.Nyh);
        const float kap = k.kappa[e] * k.inv_n;
        const float2 v = make_float2(P[i].x * kap, P[i].y * kap);
        G[i] = cmul(v, k.dyp[iy]);
        G[i + (size_t)g.S * g.cplane] = cmul(v, k.dxp[ix]);
    }
}

// u_y, u_x from the pressure gradient (two planes of g per transmitter)
__global__ void sim_velocity_kernel(SimGeom g, SimCoefs k, const float *__restrict__ grad, float *__restrict__ u) {
    const size_t half = (size_t)g.S * g.plane;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < half; i += (size_t)gridDim.x * blockDim.x) {
        const size_t e = i % g.plane;
        const int iy = (int)(e % g.Ny), ix = (int)(e / g.Ny);
        const float py = k.pmly_sg[iy], px = k.pmlx_sg[ix];
        u[i] = py * (py * u[i] - k.dt_over_rho0 * grad[i]);
        u[i + half] = px * (px * u[i + half] - k.dt_over_rho0 * grad[i + half]);
    }
}

// U_y *= kappa D-_y / N, U_x *= kappa D-_x / N (in place)
__global__ void sim_div_kernel(SimGeom g, SimCoefs k, float2 *__restrict__ U) {
    const size_t half = (size_t)g.S * g.cplane;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < half; i += (size_t)gridDim.x * blockDim.x) {
        const size_t e = i % g.cplane;
        const int iy = (int)(e % g.Nyh), ix = (int)(e / g.Nyh);
        const float kap = k.kappa[e] * k.inv_n;
        const float2 a = U[i], b = U[i + half];
        U[i] = cmul(make_float2(a.x * kap, a.y * kap), k.dyn[iy]);
        U[i + half] = cmul(make_float2(b.x * kap, b.y * kap), k.dxn[ix]);
    }
}

// split densities, Dirichlet source, pressure, sensors; the time index is
// read from *tstep (advanced by sim_tick_kernel after the step)
__global__ void sim_density_kernel(SimGeom g, SimCoefs k, const float *__restrict__ du, float *__restrict__ rho,
                                   float *__restrict__ p, const int *__restrict__ src_at, const float *__restrict__ src,
                                   const int *__restrict__ rx_slot, int n_rx, int nt, const int *__restrict__ tstep,
                                   float *__restrict__ record) {
    const int t = *tstep;
    const size_t half = (size_t)g.S * g.plane;
    const float sv = t < nt ? src[t] : 0.f;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < half; i += (size_t)gridDim.x * blockDim.x) {
        const size_t e = i % g.plane;
        const int s = (int)(i / g.plane);
        const int iy = (int)(e % g.Ny), ix = (int)(e / g.Ny);
        const float py = k.pmly[iy], px = k.pmlx[ix];
        float ry = py * (py * rho[i] - k.dt_rho0 * du[i]);
        float rx = px * (px * rho[i + half] - k.dt_rho0 * du[i + half]);
        const float c2 = k.c2[e];
        if ((int)e == src_at[s]) ry = rx = sv / (2.f * c2);
        rho[i] = ry;
        rho[i + half] = rx;
        const float pv = c2 * (ry + rx);
        p[i] = pv;
        const int r = rx_slot[e];
        if (r >= 0 && t < nt) record[((size_t)s * n_rx + r) * nt + t] = pv;
    }
}

__global__ void sim_tick_kernel(int *tstep) { *tstep += 1; }

// y[m] = sum_j h[j] x[m q + M - j] over each record (x zero outside)
__global__ void sim_decimate_kernel(const float *__restrict__ in, int nt, int n_tr, const float *__restrict__ h, int L,
                                    int q, int ly, float *__restrict__ out) {
    const size_t total = (size_t)n_tr * ly;
    const int M = (L - 1) / 2;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int m = (int)(i % ly);
        const size_t tr = i / ly;
        const float *x = in + tr * nt;
        double acc = 0.0;
        const int c = m * q + M;
        const int j0 = std::max(0, c - (nt - 1)), j1 = std::min(L - 1, c);
        for (int j = j0; j <= j1; ++j) acc += (double)h[j] * (double)x[c - j];
        out[i] = (float)acc;
    }
}

// ---------------------------------------------------------------------------
// Fused steps.  Grids whose fields fit a cluster's shared memory march there,
// all steps in one launch (fused_resident_kernel, below).  Larger ones take
// four kernels a step, each a tile of lines in shared memory from its first
// transform to its last:
//   x kernel 1   P -> forward along x, kappa D+_y and kappa D+_x, inverse
//                along x -> the two gradient spectra (along y)
//   y kernel 1   inverse along y (both gradients as one complex line, their
//                spectra are Hermitian), velocities updated, forward along y
//                -> the two velocity spectra
//   x kernel 2   forward along x, kappa D-, inverse along x, in place
//   y kernel 2   inverse along y, densities, source, pressure, sensors,
//                forward along y (two pressure lines as one) -> P
// A step reads and writes 22 planes per transmitter (the transforms of a
// library each pass over their planes two or three times more, and the
// pointwise kernels between them over all of them again: 50).  What bounds a
// tile is the latency of its phases (loads, stages, barriers: 0.41 to 0.46 of
// the issue slots at 288^2 x 64; 30 % of the memory's rate at 552^2), hence the
// three tiles an SM and the loads in batches.  Microseconds per step, library
// transforms -> here:
//   552^2, 64 transmitters         1126 -> 870
//   288^2, 64                       343 -> 274
//   1024 x 800, 4                   218 -> 172
//   266 x 259 (19, 37), 10           97 -> 87
// and no plans, allocations or graph to set up on each call: 1 ms in place of
// 5 to 60 (900 ms at 541 x 537).
// ---------------------------------------------------------------------------
struct FusedGeom {
    int Ny, Nx, Nyh, P;            // P: Nyh rounded up to 8
    int S, XB;                     // transmitters of the batch; blocks of kXT rows x
    size_t spec, cells;            // entries of a spectrum, of a pair of fields
    float inv_n, dt_rho0, dt_over_rho0;
};
struct FusedTables {
    const float *kappa;            // times 1 / (Ny Nx); [tile of KT columns ky][position of kx][KT]
    const float2 *dyp, *dyn;       // [P] i k_y exp(+-i k_y dy / 2)
    const float2 *dxp, *dxn;       // [position of kx]
    const float *pmly, *pmly_sg;   // [position of y]
    const float *pmlx, *pmlx_sg;   // [x], to whole blocks
    const float *c2;               // by cell
    const float2 *twx, *twy;       // roots of unity
};
struct FusedFields {
    const int *src_at;             // per transmitter: its cell
    const float *src;              // source samples
    const int2 *rx;                // receivers (place, slot), those of block xb from rx_row[xb] to rx_row[xb + 1]
    const int *rx_row;
    float *record;                 // [s][slot][nt]
    int n_rx, nt;
};
constexpr int kXT = 8;             // x rows per y tile
// Three tiles an SM (80 registers): at 552^2 and 64 transmitters 0.87 ms a step
// against 0.92 with two (128 registers) and 0.96 with four (64, spilling);
// loads eight at a time: 0.87 against 0.89 with four.
constexpr int kFusedThreads = 256, kTileBlocks = 3, kBatch = 8;

__global__ void fused_tables_kernel(FusedGeom g, int KT, double dy, double dx, double c_ref, double dt, const short *order,
                                    float *kappa, float2 *dyp, float2 *dyn, float2 *dxp, float2 *dxn, float2 *twx, float2 *twy) {
    const int n = blockDim.x * gridDim.x, t0 = blockIdx.x * blockDim.x + threadIdx.x;
    auto wave = [](int i, int n, double d) { return 2.0 * M_PI * (i <= (n - 1) / 2 ? i : i - n) / (n * d); };
    for (int e = t0; e < g.Nx * g.P; e += n) {
        const int row = e / KT, iy = row / g.Nx * KT + e % KT;
        float v = 0.f;
        if (iy < g.Nyh) {
            const double kx = wave(order[row % g.Nx], g.Nx, dx), ky = wave(iy, g.Ny, dy);
            const double arg = 0.5 * c_ref * dt * sqrt(kx * kx + ky * ky);
            v = (float)(arg == 0.0 ? 1.0 : sin(arg) / arg) * g.inv_n;
        }
        kappa[e] = v;
    }
    for (int i = t0; i < g.Nx; i += n) {
        const double k = wave(order[i], g.Nx, dx);
        dxp[i] = make_float2((float)(-k * sin(k * dx / 2)), (float)(k * cos(k * dx / 2)));
        dxn[i] = make_float2((float)(k * sin(k * dx / 2)), (float)(k * cos(k * dx / 2)));
        twx[i] = make_float2((float)cospi(2.0 * i / g.Nx), (float)-sinpi(2.0 * i / g.Nx));
    }
    for (int i = t0; i < g.P; i += n) {
        const double k = i < g.Nyh ? wave(i, g.Ny, dy) : 0.0;
        dyp[i] = make_float2((float)(-k * sin(k * dy / 2)), (float)(k * cos(k * dy / 2)));
        dyn[i] = make_float2((float)(k * sin(k * dy / 2)), (float)(k * cos(k * dy / 2)));
    }
    for (int i = t0; i < g.Ny; i += n) twy[i] = make_float2((float)cospi(2.0 * i / g.Ny), (float)-sinpi(2.0 * i / g.Ny));
}

// The thread's share of `total` items, U at a time: all loads of a batch are
// in flight before the first is used.  (One at a time, a tile spent most of
// its life in the latency of its 9 to 18 rounds of loads.)
template <int U, typename Load, typename Use>
__device__ __forceinline__ void in_batches(int total, Load load, Use use) {
    using V = decltype(load(0));
    for (int e0 = threadIdx.x; e0 < total; e0 += U * blockDim.x) {
        V v[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (e0 + u * blockDim.x < total) v[u] = load(e0 + u * blockDim.x);
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (e0 + u * blockDim.x < total) use(e0 + u * blockDim.x, v[u]);
    }
}
__device__ __forceinline__ float *fft_floats(int at) { return reinterpret_cast<float *>(sim::fft_sm) + at; }

// An inverse transform is a forward one between exchanges of real and imaginary part.
__device__ __forceinline__ float2 swapped(float2 v) { return make_float2(v.y, v.x); }
__device__ __forceinline__ float2 scaled(float2 v, float s) { return make_float2(v.x * s, v.y * s); }
// Two real lines travel as one complex line Z = A + i B.  Entries y and Ny - y
// of the exchanged Z from entry y of the (Hermitian) spectra A and B, and back.
__device__ __forceinline__ float2 merged(float2 a, float2 b) { return make_float2(a.y + b.x, a.x - b.y); }
__device__ __forceinline__ float2 merged_mirror(float2 a, float2 b) { return make_float2(b.x - a.y, a.x + b.y); }
__device__ __forceinline__ float2 split_a(float2 z, float2 m) { return make_float2(0.5f * (z.x + m.x), 0.5f * (z.y - m.y)); }
__device__ __forceinline__ float2 split_b(float2 z, float2 m) { return make_float2(0.5f * (z.y + m.y), 0.5f * (m.x - z.x)); }

// The entry (x, ky) of a spectrum: blocks of kXT rows x, [ky][x] in each, so
// that a y tile is one run and an x tile's pieces are whole sectors.
constexpr int tile_pad(int n) { return (n + 15) / 16 * 16; }

// FIRST: one plane in, two out; otherwise two planes in place.
template <bool FIRST, int LK>
__global__ void __launch_bounds__(kFusedThreads, kTileBlocks)
fused_x_kernel(FusedGeom g, FusedTables k, const __grid_constant__ sim::FftPlan f, const float2 *__restrict__ in, float2 *out) {
    constexpr int KT = 1 << LK;
    const int k0 = blockIdx.x * KT, N = g.Nx, za = tile_pad(N), zb = za + N * KT;
    float2 *A = sim::fft_sm + za, *B = sim::fft_sm + zb;
    const size_t at = (size_t)blockIdx.y * g.spec + (size_t)k0 * kXT, half = (size_t)g.S * g.spec;
    sim::keep_plan(0, f);
    in_batches<4>(N, [&](int i) { return k.twx[i]; }, [&](int i, float2 v) { sim::fft_sm[i] = v; });
    // lanes: 4 rows x, then the columns
    const int items = (N + 3) / 4 * 4 * KT;
    auto x_of = [](int e) { return (e >> (2 + LK)) * 4 + (e & 3); };
    auto c_of = [](int e) { return (e >> 2) & (KT - 1); };
    auto spec_at = [&](int x, int c) { return at + ((size_t)(x >> 3) * g.P + c) * kXT + (x & 7); };
    in_batches<kBatch>(items, [&](int e) {
        const int x = x_of(e);
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (x < N) {
            const size_t i = spec_at(x, c_of(e));
            const float2 a = FIRST ? in[i] : out[i];
            v.x = a.x;
            v.y = a.y;
            if (!FIRST) {
                const float2 b = out[i + half];
                v.z = b.x;
                v.w = b.y;
            }
        }
        return v;
    }, [&](int e, float4 v) {
        const int i = x_of(e) * KT + c_of(e);
        if (x_of(e) >= N) return;
        A[i] = make_float2(v.x, v.y);
        if (!FIRST) B[i] = make_float2(v.z, v.w);
    });
    __syncthreads();
    sim::fft_lines<false>(za, sim::TileLines<LK>{FIRST ? 1 : 2, N * KT}, 0, 0);
    struct Row { float kap; float2 dx; };
    const float2 dy = (FIRST ? k.dyp : k.dyn)[k0 + (threadIdx.x & (KT - 1))];   // a thread's items share the column
    const float *kappa = k.kappa + (size_t)blockIdx.x * N * KT;
    in_batches<kBatch>(N * KT, [&](int e) { return Row{kappa[e], (FIRST ? k.dxp : k.dxn)[e >> LK]}; }, [&](int e, Row r) {
        const float2 a = scaled(A[e], r.kap), b = FIRST ? a : scaled(B[e], r.kap);
        A[e] = swapped(cmul(a, dy));
        B[e] = swapped(cmul(b, r.dx));
    });
    __syncthreads();
    sim::fft_lines<true>(za, sim::TileLines<LK>{2, N * KT}, 0, 0);
    for (int e = threadIdx.x; e < items; e += kFusedThreads) {
        const int x = x_of(e), c = c_of(e);
        if (x >= N) continue;
        const size_t i = spec_at(x, c);
        out[i] = swapped(A[x * KT + c]);
        out[i + half] = swapped(B[x * KT + c]);
    }
}

// VELOCITY: gradients -> velocities -> their spectra, in place in spec (two
// planes).  Otherwise: divergence (two planes of spec) -> densities,
// pressure -> its spectrum in p_spec.  The fields (y part, x part) are kept
// in the order of the tile in shared memory, transform's order included.
template <bool VELOCITY>
__global__ void __launch_bounds__(kFusedThreads, kTileBlocks)
fused_y_kernel(FusedGeom g, FusedTables k, const __grid_constant__ sim::FftPlan f, FusedFields q, float2 *fields, float2 *spec,
               float2 *p_spec, int t) {
    const int N = g.Ny, xb = blockIdx.x, s = blockIdx.y, tid = threadIdx.x, z0 = tile_pad(N), l = tid & (kXT - 1);
    float2 *z = sim::fft_sm + z0;                                          // [y or ky][kXT]
    const size_t half = (size_t)g.S * g.spec, at = (size_t)s * g.spec + (size_t)xb * g.P * kXT;
    const int spec_items = g.Nyh * kXT;
    sim::keep_plan(0, f);
    in_batches<4>(N, [&](int i) { return k.twy[i]; }, [&](int i, float2 v) { sim::fft_sm[i] = v; });
    in_batches<kBatch>(spec_items, [&](int e) {
        const float2 a = spec[at + e], b = spec[at + half + e];
        return make_float4(a.x, a.y, b.x, b.y);
    }, [&](int e, float4 v) {
        const int y = e / kXT;
        const float2 a = make_float2(v.x, v.y), b = make_float2(v.z, v.w);
        const bool self = y == 0 || 2 * y == N;                            // real there
        z[e] = self ? make_float2(b.x, a.x) : merged(a, b);
        if (!self) z[(N - y) * kXT + l] = merged_mirror(a, b);
    });
    __syncthreads();
    sim::fft_lines<false>(z0, sim::TileLines<3>{1, 0}, 0, 0);
    const int src = VELOCITY ? 0 : q.src_at[s], cell0 = xb * N * kXT;
    const float sv = VELOCITY ? 0.f : q.src[t], px = (VELOCITY ? k.pmlx_sg : k.pmlx)[xb * kXT + l];
    const float scale = VELOCITY ? g.dt_over_rho0 : g.dt_rho0;
    float2 *state = fields + (size_t)s * g.cells + cell0;
    struct Point { float2 v; float py, c2; };
    in_batches<kBatch>(N * kXT, [&](int e) {
        return Point{state[e], (VELOCITY ? k.pmly_sg : k.pmly)[e / kXT], VELOCITY ? 0.f : k.c2[cell0 + e]};
    }, [&](int e, Point p) {
        const float2 d = z[e];                                             // exchanged: y part in .y
        float2 v = make_float2(p.py * (p.py * p.v.x - scale * d.y), px * (px * p.v.y - scale * d.x));
        if (!VELOCITY && cell0 + e == src) v.x = v.y = sv / (2.f * p.c2);
        state[e] = v;
        z[e] = VELOCITY ? v : make_float2(p.c2 * (v.x + v.y), 0.f);
    });
    __syncthreads();
    if (!VELOCITY) {
        for (int r = q.rx_row[xb] + tid; r < q.rx_row[xb + 1]; r += kFusedThreads) {
            const int2 place = q.rx[r];
            q.record[((size_t)s * q.n_rx + place.y) * q.nt + t] = z[place.x].x;
        }
        // pressure lines l and l + 4 as one complex line, packed to four lines
        const int w0 = z0 + N * kXT;
        float2 *w = sim::fft_sm + w0;
        for (int e = tid; e < N * (kXT / 2); e += kFusedThreads) {
            const int i = e + (e & ~(kXT / 2 - 1));
            w[e] = make_float2(z[i].x, z[i + kXT / 2].x);
        }
        __syncthreads();
        sim::fft_lines<true>(w0, sim::TileLines<2>{1, 0}, 0, 0);
        float2 *p = p_spec + at;
        for (int e = tid; e < spec_items; e += kFusedThreads) {
            const int y = e / kXT, h = kXT / 2, c = l & (h - 1);
            const float2 a = w[y * h + c], b = w[(y ? N - y : 0) * h + c];
            p[e] = l < h ? split_a(a, b) : split_b(a, b);
        }
        return;
    }
    sim::fft_lines<true>(z0, sim::TileLines<3>{1, 0}, 0, 0);
    for (int e = tid; e < spec_items; e += kFusedThreads) {
        const int y = e / kXT;
        const float2 a = z[e], b = z[(y ? N - y : 0) * kXT + l];
        spec[at + e] = split_a(a, b);
        spec[at + half + e] = split_b(a, b);
    }
}

// Grids whose fields fit the shared memory of a cluster: it takes all steps of
// its transmitter in one launch, with no global memory but the records.  A
// block holds XR rows x for what goes along y and CK columns ky for what goes
// along x; the passes hand each other their values through distributed shared
// memory, a cluster barrier between them (four a step).  Bound by instructions
// where a block has 2000 points or more, by the latency of some 35 phases
// below.  Microseconds per step, library transforms (14 launches) -> here:
//   20 x 20, 2 transmitters          24 -> 9
//   43 x 47 (both prime), 3          31 -> 15
//   62 x 79 (31, 79), 5              44 -> 22
//   128 x 128, 4                     31 -> 21
//   180 x 200, 3                     36 -> 32
// One block for all of a transmitter took 31 at 43 x 47 and 76 at 62 x 79.
struct ResidentShape {
    int C, XR, CK, threads;        // blocks of the cluster; rows, columns and threads of a block
    int ldr, ldc, H;               // pitch of a row, of the columns (A, then B); rows of pressure pairs
    int twy, dxp, dxn, dyp, dyn, u, r, rows, cols, floats;       // places in shared memory (float2)
    size_t bytes;
};
inline ResidentShape resident_shape(int Ny, int Nx, int C) {
    ResidentShape m{};
    const int Nyh = Ny / 2 + 1;
    m.C = C;
    m.XR = (Nx + C - 1) / C;
    m.CK = (Nyh + C - 1) / C;
    m.threads = m.XR * Ny <= 512 ? 256 : 512;                              // 43 x 47: 15.4 against 16.4 us a step; 62 x 79: 23.8 against 22.4
    m.ldr = Ny | 1;                                                        // odd: no bank conflicts down a column
    m.ldc = 2 * m.CK;
    m.H = (m.XR + 1) / 2;
    m.twy = Nx;
    m.dxp = m.twy + Ny;
    m.dxn = m.dxp + Nx;
    m.dyp = m.dxn + Nx;
    m.dyn = m.dyp + m.CK;
    m.u = m.dyn + m.CK;
    m.r = m.u + m.XR * Ny;
    m.rows = m.r + m.XR * Ny;
    m.cols = m.rows + m.XR * m.ldr;
    m.floats = 2 * (m.cols + Nx * m.ldc);                                  // c2, kappa, pml: in floats
    m.bytes = (size_t)4 * m.floats + (size_t)4 * ((size_t)m.XR * Ny + (size_t)Nx * m.CK + 2 * Ny + 2 * m.XR);
    return m;
}
__global__ void __launch_bounds__(512)
fused_resident_kernel(FusedGeom g, FusedTables k, const __grid_constant__ ResidentShape m, const __grid_constant__ sim::FftPlan fx,
                      const __grid_constant__ sim::FftPlan fy, FusedFields q) {
    namespace cg = cooperative_groups;
    const cg::cluster_group cluster = cg::this_cluster();
    const int Ny = g.Ny, Nx = g.Nx, Nyh = g.Nyh, tid = threadIdx.x, nt = blockDim.x;
    const int rank = (int)cluster.block_rank(), s = blockIdx.x / m.C, XR = m.XR, CK = m.CK, ldr = m.ldr, ldc = m.ldc, H = m.H;
    const int x0 = rank * XR, k0 = rank * CK, n = XR * Ny, nc = Nx * CK, nh = XR * Nyh;
    float2 *const u = sim::fft_sm + m.u, *const r = sim::fft_sm + m.r, *const rows = sim::fft_sm + m.rows,
                 *const cols = sim::fft_sm + m.cols;
    float *const c2 = fft_floats(m.floats), *const kappa = c2 + n, *const pmly = kappa + nc, *const pmly_sg = pmly + Ny,
                *const pmlx = pmly_sg + Ny, *const pmlx_sg = pmlx + XR;
    const float inv_y = 1.f / Ny, inv_h = 1.f / Nyh, inv_k = 1.f / CK, inv_x = 1.f / XR;
    sim::keep_plan(0, fx);
    sim::keep_plan(1, fy);
    for (int e = tid; e < n; e += nt) {
        u[e] = r[e] = make_float2(0.f, 0.f);
        c2[e] = x0 * Ny + e < Nx * Ny ? k.c2[x0 * Ny + e] : 0.f;
    }
    for (int e = tid; e < XR * ldr; e += nt) rows[e] = make_float2(0.f, 0.f);
    for (int e = tid; e < Nx * ldc; e += nt) cols[e] = make_float2(0.f, 0.f);
    for (int e = tid; e < nc; e += nt) {
        const int i = sim::fast_div(e, inv_k), y = k0 + e - i * CK;
        kappa[e] = y < Nyh ? k.kappa[i * g.P + y] : 0.f;
    }
    for (int i = tid; i < Ny; i += nt) {
        sim::fft_sm[m.twy + i] = k.twy[i];
        pmly[i] = k.pmly[i];
        pmly_sg[i] = k.pmly_sg[i];
    }
    for (int i = tid; i < Nx; i += nt) {
        sim::fft_sm[i] = k.twx[i];
        sim::fft_sm[m.dxp + i] = k.dxp[i];
        sim::fft_sm[m.dxn + i] = k.dxn[i];
    }
    for (int i = tid; i < XR; i += nt) {
        pmlx[i] = x0 + i < Nx ? k.pmlx[x0 + i] : 0.f;
        pmlx_sg[i] = x0 + i < Nx ? k.pmlx_sg[x0 + i] : 0.f;
    }
    for (int i = tid; i < CK; i += nt) {
        const bool on = k0 + i < Nyh;
        sim::fft_sm[m.dyp + i] = on ? k.dyp[k0 + i] : make_float2(0.f, 0.f);
        sim::fft_sm[m.dyn + i] = on ? k.dyn[k0 + i] : make_float2(0.f, 0.f);
    }
    const int src = q.src_at[s] - x0 * Ny, rx0 = q.rx_row[rank], rx1 = q.rx_row[rank + 1];
    const sim::GridLines one{CK, 1, ldc, 1.f / CK}, both{2 * CK, 1, ldc, 0.5f / CK}, whole{XR, ldr, 1, 1.f / XR},
        pairs{H, ldr, 1, 1.f / H};
    // columns of both spectra -> rows of complex lines
    auto to_rows = [&] {
        for (int e = tid; e < nc; e += nt) {
            const int x = sim::fast_div(e, inv_k), c = e - x * CK, y = k0 + c;
            if (y >= Nyh) continue;
            const int owner = sim::fast_div(x, inv_x);
            float2 *const row = cluster.map_shared_rank(rows, owner) + (x - owner * XR) * ldr;
            const bool self = y == 0 || 2 * y == Ny;
            const float2 a = swapped(cols[x * ldc + c]), b = swapped(cols[x * ldc + CK + c]);
            row[y] = self ? make_float2(b.x, a.x) : merged(a, b);
            if (!self) row[Ny - y] = merged_mirror(a, b);
        }
        cluster.sync();
    };
    cluster.sync();
    for (int t = 0; t < q.nt; ++t) {
        // pressure spectrum -> gradients
        sim::fft_lines<false>(m.cols, one, 0, 0);
        for (int e = tid; e < nc; e += nt) {
            const int i = sim::fast_div(e, inv_k), c = e - i * CK;
            float2 *const a = cols + i * ldc + c;
            const float2 v = scaled(*a, kappa[e]);
            a[0] = swapped(cmul(v, sim::fft_sm[m.dyp + c]));
            a[CK] = swapped(cmul(v, sim::fft_sm[m.dxp + i]));
        }
        __syncthreads();
        sim::fft_lines<true>(m.cols, both, 0, 0);
        to_rows();
        sim::fft_lines<false>(m.rows, whole, 1, m.twy);
        for (int e = tid; e < n; e += nt) {
            const int x = sim::fast_div(e, inv_y), i = e - x * Ny;
            const float2 d = rows[x * ldr + i], v = u[e];
            const float py = pmly_sg[i], px = pmlx_sg[x];
            rows[x * ldr + i] = u[e] =
                make_float2(py * (py * v.x - g.dt_over_rho0 * d.y), px * (px * v.y - g.dt_over_rho0 * d.x));
        }
        __syncthreads();
        // velocities -> divergence
        sim::fft_lines<true>(m.rows, whole, 1, m.twy);
        for (int e = tid; e < nh; e += nt) {
            const int x = sim::fast_div(e, inv_h), y = e - x * Nyh;
            if (x0 + x >= Nx) continue;
            const float2 a = rows[x * ldr + y], b = rows[x * ldr + (y ? Ny - y : 0)];
            const int owner = sim::fast_div(y, inv_k);
            float2 *const to = cluster.map_shared_rank(cols, owner) + (x0 + x) * ldc + y - owner * CK;
            to[0] = split_a(a, b);
            to[CK] = split_b(a, b);
        }
        cluster.sync();
        sim::fft_lines<false>(m.cols, both, 0, 0);
        for (int e = tid; e < nc; e += nt) {
            const int i = sim::fast_div(e, inv_k), c = e - i * CK;
            float2 *const a = cols + i * ldc + c;
            a[0] = swapped(cmul(scaled(a[0], kappa[e]), sim::fft_sm[m.dyn + c]));
            a[CK] = swapped(cmul(scaled(a[CK], kappa[e]), sim::fft_sm[m.dxn + i]));
        }
        __syncthreads();
        sim::fft_lines<true>(m.cols, both, 0, 0);
        to_rows();
        sim::fft_lines<false>(m.rows, whole, 1, m.twy);
        // densities, source, pressure: rows x and x + H, one complex row afterwards
        const float sv = q.src[t];
        for (int e = tid; e < H * Ny; e += nt) {
            const int x = sim::fast_div(e, inv_y), i = e - x * Ny;
            const float py = pmly[i];
            auto pressure = [&](int x) {
                const int c = x * Ny + i;
                const float2 d = rows[x * ldr + i], v = r[c];
                const float px = pmlx[x];
                float2 w = make_float2(py * (py * v.x - g.dt_rho0 * d.y), px * (px * v.y - g.dt_rho0 * d.x));
                if (c == src) w.x = w.y = sv / (2.f * c2[c]);
                r[c] = w;
                return c2[c] * (w.x + w.y);
            };
            const float p = pressure(x);
            rows[x * ldr + i] = make_float2(p, x + H < XR ? pressure(x + H) : 0.f);
        }
        __syncthreads();
        for (int i = rx0 + tid; i < rx1; i += nt) {
            const int2 place = q.rx[i];
            q.record[((size_t)s * q.n_rx + place.y) * q.nt + t] = fft_floats(2 * m.rows)[place.x];
        }
        __syncthreads();
        sim::fft_lines<true>(m.rows, pairs, 1, m.twy);
        for (int e = tid; e < H * Nyh; e += nt) {
            const int x = sim::fast_div(e, inv_h), y = e - x * Nyh;
            const float2 a = rows[x * ldr + y], b = rows[x * ldr + (y ? Ny - y : 0)];
            const int owner = sim::fast_div(y, inv_k);
            float2 *const to = cluster.map_shared_rank(cols, owner) + (x0 + x) * ldc + y - owner * CK;
            if (x0 + x < Nx) to[0] = split_a(a, b);
            if (x + H < XR && x0 + x + H < Nx) to[H * ldc] = split_b(a, b);
        }
        cluster.sync();
    }
}

int sim_grid(size_t n) { return (int)std::min<size_t>((n + kSimThreads - 1) / kSimThreads, 148 * 16); }

}  // namespace

// Taps of MATLAB resample(., 1, q, half_length, beta): the least-squares
// ideal low-pass (the truncated sinc, cut-off pi / q), Kaiser window, unit DC
// gain.
static std::vector<float> decimation_taps(int q, int half_length, double beta) {
    const int L = 2 * half_length * q + 1, M = half_length * q;
    auto bessel_i0 = [](double x) {
        double sum = 1.0, term = 1.0;
        for (int k = 1; k < 200; ++k) {
            term *= (x / (2.0 * k)) * (x / (2.0 * k));
            sum += term;
            if (term < 1e-17 * sum) break;
        }
        return sum;
    };
    std::vector<double> h(L);
    double total = 0.0;
    for (int j = 0; j < L; ++j) {
        const double k = j - M, arg = M_PI * k / q;
        const double sinc = k == 0 ? 1.0 : std::sin(arg) / arg;
        const double r = 2.0 * j / (L - 1) - 1.0;
        const double w = bessel_i0(beta * std::sqrt(std::max(0.0, 1.0 - r * r))) / bessel_i0(beta);
        h[j] = sinc / q * w;
        total += h[j];
    }
    std::vector<float> hf(L);
    for (int j = 0; j < L; ++j) hf[j] = (float)(h[j] / total);
    return hf;
}

// ---- the fused steps: workspace layout and host side ---------------------------
constexpr size_t kFusedSmem = 226 * 1024;        // dynamic; the plans take another 0.7 KB
struct FusedLayout {
    FusedGeom g;
    int KT;                        // ky columns per x tile
    bool resident;
    ResidentShape shape;
    size_t kappa, dyp, dyn, dxp, dxn, pml, c2, twx, twy, order, src_at, src, rx, rx_row, taps, host_end, fields, specs, record, total;
    size_t smem_x, smem_v, smem_p;
};
static FusedLayout fused_layout(int ny, int nx, int pml, int ntx, int nrx, int nt, int q, int tx_batch) {
    FusedLayout L{};
    FusedGeom &g = L.g;
    g.Ny = ny + 2 * pml;
    g.Nx = nx + 2 * pml;
    g.Nyh = g.Ny / 2 + 1;
    g.P = (g.Nyh + 7) / 8 * 8;
    g.S = std::max(1, std::min(tx_batch > 0 ? tx_batch : ntx, ntx));
    g.XB = (g.Nx + kXT - 1) / kXT;
    g.spec = (size_t)g.XB * kXT * g.P;
    g.cells = (size_t)g.XB * kXT * g.Ny;
    // the widest cluster that leaves every transmitter its own, or else the narrowest that holds the fields
    if ((long long)g.Nx * g.Ny <= 1 << 17)
        for (int C = 8; C >= 1; C /= 2) {
            const ResidentShape m = resident_shape(g.Ny, g.Nx, C);
            if (m.bytes > kFusedSmem) break;
            L.resident = true;
            L.shape = m;
            if (C * g.S <= 120) break;
        }
    // 64-byte pieces of the spectra where two such tiles fit an SM
    auto tile = [](int n, int lines) { return sizeof(float2) * ((size_t)tile_pad(n) + (size_t)n * lines); };
    L.KT = tile(g.Nx, 16) <= 112 * 1024 ? 8 : 4;
    L.smem_x = tile(g.Nx, 2 * L.KT);
    L.smem_v = tile(g.Ny, kXT);
    L.smem_p = tile(g.Ny, kXT + kXT / 2);
    size_t at = 0;
    auto put = [&](size_t bytes) {
        const size_t r = at;
        at += (bytes + 255) / 256 * 256;
        return r;
    };
    L.kappa = put((size_t)g.Nx * g.P * 4);
    L.dyp = put(g.P * 8);
    L.dyn = put(g.P * 8);
    L.dxp = put(g.Nx * 8);
    L.dxn = put(g.Nx * 8);
    L.twx = put(g.Nx * 8);
    L.twy = put(g.Ny * 8);
    L.c2 = put(g.cells * 4);                     // from here to host_end: copied from the host
    L.pml = put((size_t)2 * (g.Ny + g.XB * kXT) * 4);
    L.order = put((size_t)g.Nx * 2);
    L.src_at = put((size_t)ntx * 4);
    L.src = put((size_t)nt * 4);
    L.rx = put((size_t)nrx * 8);
    L.rx_row = put((size_t)(std::max(g.XB, 8) + 1) * 4);
    L.taps = put((size_t)(48 * q + 1) * 4);
    L.host_end = at;
    L.fields = put(L.resident ? 0 : (size_t)2 * g.S * g.cells * 8);
    L.specs = put(L.resident ? 0 : (size_t)3 * g.S * g.spec * 8);
    L.record = put((size_t)g.S * nrx * nt * 4);
    L.total = at;
    return L;
}

// Whether the fused kernels take the grid: a tile of lines in shared memory,
// indices in 16 and 32 bits, and no prime whose direct sums cost more than the
// library's transforms.  In a cluster they are even at 113 x 109 (48 us a step
// each) and behind at 128 x 149 (50 against 43); tiles win at 266 x 259 (37: 87
// against 97) and lose at 236 x 305 with few transmitters (59, 61: 89 against 77).
static bool fused_fits(const FusedLayout &L) {
    auto largest_prime = [](int n) {
        int p = 1;
        for (int r = 2; r * r <= n; ++r)
            while (n % r == 0) {
                p = r;
                n /= r;
            }
        return std::max(p, n);
    };
    return L.smem_x <= kFusedSmem && L.smem_p <= kFusedSmem && std::max(L.g.Nx, L.g.Ny) <= 32767 &&
           L.g.cells <= 2147483647ULL && L.g.S <= 65535 &&
           std::max(largest_prime(L.g.Nx), largest_prime(L.g.Ny)) <= (L.resident ? 113 : 37);
}

static void simulate_fused(const SimulateArgs &a, const FusedLayout &L, uint8_t *ws, float *rf, cudaStream_t st) {
    FusedGeom g = L.g;
    const int ny = a.ny, nx = a.nx, P = a.pml, ntx = a.ntx, nrx = a.nrx, nt = a.nt, S = g.S;
    const int q = std::max(1, a.decimation), ly = (nt + q - 1) / q;
    g.inv_n = (float)(1.0 / ((double)g.Ny * g.Nx));
    g.dt_rho0 = (float)(a.dt * a.rho0);
    g.dt_over_rho0 = (float)(a.dt / a.rho0);
    const int largest = L.resident ? 8 : 24;
    const sim::FftPlan fx = sim::fft_plan(g.Nx, largest), fy = sim::fft_plan(g.Ny, largest);
    std::vector<int> pos(g.Ny);                  // where the y transform leaves sample y
    for (int i = 0; i < g.Ny; ++i) pos[sim::fft_index_at(fy, i)] = i;
    auto cell = [&](int ix, int iy) {
        return L.resident ? ix * g.Ny + pos[iy] : (ix / kXT * g.Ny + pos[iy]) * kXT + ix % kXT;
    };
    // ---- what comes from the host, in one copy --------------------------------
    std::vector<uint8_t> host(L.host_end - L.c2, 0);
    auto h = [&](size_t at) { return host.data() + (at - L.c2); };
    float *c2 = (float *)h(L.c2);
    for (int ix = 0; ix < g.Nx; ++ix) {          // the medium extended with its edge values
        const double *col = a.c + (size_t)ny * std::min(std::max(ix - P, 0), nx - 1);
        for (int iy = 0; iy < g.Ny; ++iy) {
            const double c = col[std::min(std::max(iy - P, 0), ny - 1)];
            c2[cell(ix, iy)] = (float)(c * c);
        }
    }
    float *pml = (float *)h(L.pml);
    const int pml_x = 2 * g.Ny, pml_xs = pml_x + g.XB * kXT;
    for (int i = 0; i < g.Ny; ++i) {
        pml[pos[i]] = (float)pml_value(i, g.Ny, P, a.dy, a.dt, a.c_ref, false);
        pml[g.Ny + pos[i]] = (float)pml_value(i, g.Ny, P, a.dy, a.dt, a.c_ref, true);
    }
    for (int i = 0; i < g.Nx; ++i) {
        pml[pml_x + i] = (float)pml_value(i, g.Nx, P, a.dx, a.dt, a.c_ref, false);
        pml[pml_xs + i] = (float)pml_value(i, g.Nx, P, a.dx, a.dt, a.c_ref, true);
    }
    short *order = (short *)h(L.order);
    for (int i = 0; i < g.Nx; ++i) order[i] = (short)sim::fft_index_at(fx, i);
    auto padded = [&](int lin1) { return cell((lin1 - 1) / ny + P, (lin1 - 1) % ny + P); };
    int *src_at = (int *)h(L.src_at);
    for (int s = 0; s < ntx; ++s) src_at[s] = padded(a.tx_index[s]);
    float *src = (float *)h(L.src);
    for (int i = 0; i < nt; ++i) src[i] = (float)a.source[i];
    int2 *rx = (int2 *)h(L.rx);
    int *rx_row = (int *)h(L.rx_row);
    for (int r = 0; r < nrx; ++r) rx[r] = make_int2(padded(a.rx_index[r]), r);
    std::sort(rx, rx + nrx, [](int2 u, int2 v) { return u.x < v.x; });
    const int rows_each = L.resident ? L.shape.XR : kXT;
    for (int b = 0, r = 0; b <= (L.resident ? L.shape.C : g.XB); ++b) {
        for (; r < nrx && rx[r].x < (long long)b * rows_each * g.Ny; ++r) {
            rx[r].x -= (b - 1) * rows_each * g.Ny;
            if (L.resident) {                    // floats of the block's rows: x and x + H share one
                const ResidentShape &m = L.shape;
                const int x = rx[r].x / g.Ny, i = rx[r].x % g.Ny;
                rx[r].x = 2 * ((x < m.H ? x : x - m.H) * m.ldr + i) + (x >= m.H);
            }
        }
        rx_row[b] = r;
    }
    if (q > 1) {
        const std::vector<float> taps = decimation_taps(q, 24, 8.6);
        std::copy(taps.begin(), taps.end(), (float *)h(L.taps));
    }
    WUST_CUDA(cudaMemcpyAsync(ws + L.c2, host.data(), host.size(), cudaMemcpyHostToDevice, st));
    FusedTables k{};
    k.kappa = (float *)(ws + L.kappa);
    k.dyp = (float2 *)(ws + L.dyp);
    k.dyn = (float2 *)(ws + L.dyn);
    k.dxp = (float2 *)(ws + L.dxp);
    k.dxn = (float2 *)(ws + L.dxn);
    k.twx = (float2 *)(ws + L.twx);
    k.twy = (float2 *)(ws + L.twy);
    k.c2 = (float *)(ws + L.c2);
    k.pmly = (float *)(ws + L.pml);
    k.pmly_sg = k.pmly + g.Ny;
    k.pmlx = k.pmly + pml_x;
    k.pmlx_sg = k.pmly + pml_xs;
    fused_tables_kernel<<<std::min(ceil_div((long long)g.Nx * g.P, 256), 2 * 148), 256, 0, st>>>(
        g, L.resident ? g.P : L.KT, a.dy, a.dx, a.c_ref, a.dt, (const short *)(ws + L.order), (float *)(ws + L.kappa),
        (float2 *)(ws + L.dyp), (float2 *)(ws + L.dyn), (float2 *)(ws + L.dxp), (float2 *)(ws + L.dxn), (float2 *)(ws + L.twx),
        (float2 *)(ws + L.twy));
    ++g_kernel_launches;
    WUST_LAUNCH_CHECK();
    // to the limit, not to this grid's need: the attribute belongs to the
    // function, and another thread may be launching it at another size
    auto grow = [](const void *kernel) {
        WUST_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFusedSmem));
    };
    auto x_first = L.KT == 8 ? fused_x_kernel<true, 3> : fused_x_kernel<true, 2>;
    auto x_second = L.KT == 8 ? fused_x_kernel<false, 3> : fused_x_kernel<false, 2>;
    if (L.resident) {
        grow((const void *)fused_resident_kernel);
    } else {
        grow((const void *)x_first);
        grow((const void *)x_second);
        grow((const void *)fused_y_kernel<true>);
        grow((const void *)fused_y_kernel<false>);
    }
    float *record = (float *)(ws + L.record);
    float2 *u = (float2 *)(ws + L.fields), *r = u + (size_t)S * g.cells;
    float2 *specs = (float2 *)(ws + L.specs), *p_spec = specs + (size_t)2 * S * g.spec;
    for (int s0 = 0; s0 < ntx; s0 += S) {
        const int sb = std::min(S, ntx - s0);
        const FusedFields d{(const int *)(ws + L.src_at) + s0, (const float *)(ws + L.src), (const int2 *)(ws + L.rx),
                            (const int *)(ws + L.rx_row), record, nrx, nt};
        if (L.resident) {
            cudaLaunchConfig_t config{};
            cudaLaunchAttribute in_cluster{};
            in_cluster.id = cudaLaunchAttributeClusterDimension;
            in_cluster.val.clusterDim.x = L.shape.C;
            in_cluster.val.clusterDim.y = in_cluster.val.clusterDim.z = 1;
            config.gridDim = dim3(sb * L.shape.C);
            config.blockDim = dim3(L.shape.threads);
            config.dynamicSmemBytes = L.shape.bytes;
            config.stream = st;
            config.attrs = &in_cluster;
            config.numAttrs = 1;
            WUST_CUDA(cudaLaunchKernelEx(&config, fused_resident_kernel, g, k, L.shape, fx, fy, d));
            ++g_kernel_launches;
        } else {
            WUST_CUDA(cudaMemsetAsync(u, 0, sizeof(float2) * 2 * (size_t)S * g.cells, st));
            WUST_CUDA(cudaMemsetAsync(specs, 0, sizeof(float2) * 3 * (size_t)S * g.spec, st));
            const dim3 gx(ceil_div(g.Nyh, L.KT), sb), gy(g.XB, sb);
            for (int t = 0; t < nt; ++t) {
                x_first<<<gx, kFusedThreads, L.smem_x, st>>>(g, k, fx, p_spec, specs);
                fused_y_kernel<true><<<gy, kFusedThreads, L.smem_v, st>>>(g, k, fy, d, u, specs, nullptr, t);
                x_second<<<gx, kFusedThreads, L.smem_x, st>>>(g, k, fx, nullptr, specs);
                fused_y_kernel<false><<<gy, kFusedThreads, L.smem_p, st>>>(g, k, fy, d, r, specs, p_spec, t);
            }
            g_kernel_launches += 4LL * nt;
        }
        WUST_LAUNCH_CHECK();
        // records [s][r][t] -> rf [t][r][tx] column-major, i.e. memory [tx][r][t]
        float *dst = rf + (size_t)s0 * nrx * ly;
        if (q == 1) {
            WUST_CUDA(cudaMemcpyAsync(dst, record, (size_t)sb * nrx * nt * 4, cudaMemcpyDeviceToDevice, st));
        } else {
            const size_t n_out = (size_t)sb * nrx * ly;
            sim_decimate_kernel<<<sim_grid(n_out), kSimThreads, 0, st>>>(record, nt, sb * nrx, (const float *)(ws + L.taps),
                                                                          48 * q + 1, q, ly, dst);
            ++g_kernel_launches;
            WUST_LAUNCH_CHECK();
        }
    }
    WUST_CUDA(cudaStreamSynchronize(st));
}

size_t simulate_workspace_bytes(int ny, int nx, int pml, int ntx, int nrx, int nt, int decimation, int tx_batch) {
    const FusedLayout L = fused_layout(ny, nx, pml, ntx, nrx, nt, std::max(1, decimation), tx_batch);
    return fused_fits(L) ? L.total : 0;
}

static void simulate_library(const SimulateArgs &a, float *rf, cudaStream_t caller);

void simulate_rf(const SimulateArgs &a, void *workspace, float *rf, cudaStream_t st) {
    const FusedLayout L = fused_layout(a.ny, a.nx, a.pml, a.ntx, a.nrx, a.nt, std::max(1, a.decimation), a.tx_batch);
    if (!fused_fits(L)) {
        simulate_library(a, rf, st);
        return;
    }
    CallMemory mem(st);
    simulate_fused(a, L, static_cast<uint8_t *>(mem.take(workspace, L.total)), rf, st);
    mem.done = true;
}

// Grids beyond the fused kernels (fused_fits): library transforms.
static void simulate_library(const SimulateArgs &a, float *rf, cudaStream_t caller) {
    // the work runs on a stream of its own, ordered after the caller's stream
    // (which may be the legacy default stream, where a graph cannot be
    // captured); the call returns when it is done
    struct StreamGuard {
        cudaStream_t s = nullptr;
        cudaEvent_t e = nullptr;
        ~StreamGuard() {
            if (s) {
                cudaStreamSynchronize(s);
                cudaStreamDestroy(s);
            }
            if (e) cudaEventDestroy(e);
        }
    } own;
    WUST_CUDA(cudaStreamCreateWithFlags(&own.s, cudaStreamNonBlocking));
    WUST_CUDA(cudaEventCreateWithFlags(&own.e, cudaEventDisableTiming));
    WUST_CUDA(cudaEventRecord(own.e, caller));
    WUST_CUDA(cudaStreamWaitEvent(own.s, own.e, 0));
    cudaStream_t st = own.s;
    const int ny = a.ny, nx = a.nx, P = a.pml;
    SimGeom g{};
    g.Ny = ny + 2 * P;
    g.Nx = nx + 2 * P;
    g.Nyh = g.Ny / 2 + 1;
    g.plane = (size_t)g.Ny * g.Nx;
    g.cplane = (size_t)g.Nyh * g.Nx;
    const int ntx = a.ntx, nrx = a.nrx, nt = a.nt;
    const int S = std::max(1, std::min(a.tx_batch > 0 ? a.tx_batch : ntx, ntx));
    g.S = S;
    const int q = std::max(1, a.decimation);
    const int ly = (nt + q - 1) / q;

    // ---- coefficients (host, FP64, stored in float) -------------------------
    std::vector<float> kappa(g.cplane), pmly(g.Ny), pmlys(g.Ny), pmlx(g.Nx), pmlxs(g.Nx), c2(g.plane);
    std::vector<float2> dyp(g.Nyh), dyn(g.Nyh), dxp(g.Nx), dxn(g.Nx);
    for (int ix = 0; ix < g.Nx; ++ix) {
        const double kx = kwave_k(ix, g.Nx, a.dx);
        for (int iy = 0; iy < g.Nyh; ++iy) {
            const double ky = kwave_k(iy, g.Ny, a.dy);
            const double arg = 0.5 * a.c_ref * a.dt * std::sqrt(kx * kx + ky * ky);
            kappa[(size_t)ix * g.Nyh + iy] = (float)(arg == 0.0 ? 1.0 : std::sin(arg) / arg);
        }
        dxp[ix] = make_float2((float)(-kx * std::sin(kx * a.dx / 2)), (float)(kx * std::cos(kx * a.dx / 2)));
        dxn[ix] = make_float2((float)(kx * std::sin(kx * a.dx / 2)), (float)(kx * std::cos(kx * a.dx / 2)));
        pmlx[ix] = (float)pml_value(ix, g.Nx, P, a.dx, a.dt, a.c_ref, false);
        pmlxs[ix] = (float)pml_value(ix, g.Nx, P, a.dx, a.dt, a.c_ref, true);
    }
    for (int iy = 0; iy < g.Nyh; ++iy) {
        const double ky = kwave_k(iy, g.Ny, a.dy);
        dyp[iy] = make_float2((float)(-ky * std::sin(ky * a.dy / 2)), (float)(ky * std::cos(ky * a.dy / 2)));
        dyn[iy] = make_float2((float)(ky * std::sin(ky * a.dy / 2)), (float)(ky * std::cos(ky * a.dy / 2)));
    }
    for (int iy = 0; iy < g.Ny; ++iy) {
        pmly[iy] = (float)pml_value(iy, g.Ny, P, a.dy, a.dt, a.c_ref, false);
        pmlys[iy] = (float)pml_value(iy, g.Ny, P, a.dy, a.dt, a.c_ref, true);
    }
    // the medium extended with its edge values
    for (int ix = 0; ix < g.Nx; ++ix)
        for (int iy = 0; iy < g.Ny; ++iy) {
            const int sy = std::min(std::max(iy - P, 0), ny - 1), sx = std::min(std::max(ix - P, 0), nx - 1);
            const double c = a.c[sy + (size_t)ny * sx];
            c2[(size_t)ix * g.Ny + iy] = (float)(c * c);
        }
    std::vector<int> rx_slot(g.plane, -1), src_at_all(ntx);
    auto padded = [&](int lin1) {
        const int iy = (lin1 - 1) % ny, ix = (lin1 - 1) / ny;
        return (ix + P) * g.Ny + (iy + P);
    };
    for (int r = 0; r < nrx; ++r) rx_slot[padded(a.rx_index[r])] = r;
    for (int s = 0; s < ntx; ++s) src_at_all[s] = padded(a.tx_index[s]);
    std::vector<float> srcf(nt);
    for (int t = 0; t < nt; ++t) srcf[t] = (float)a.source[t];

    // ---- device buffers (one allocation) ----------------------------------
    auto al = [](size_t b) { return (b + 255) / 256 * 256; };
    const size_t b_coef = al(g.cplane * 4) + 4 * al(std::max<size_t>(g.Nyh, g.Nx) * 8) + 2 * al(g.Ny * 4) +
                          2 * al(g.Nx * 4) + al(g.plane * 4) + al(g.plane * 4) + al(ntx * 4) + al(nt * 4) + 256;
    const size_t b_fields = al((size_t)S * g.plane * 4) * 7;            // p, u (2), rho (2), g/du (2)
    const size_t b_spec = al((size_t)S * g.cplane * 8) * 3;             // P (1), G/U (2)
    const size_t b_rec = al((size_t)S * nrx * nt * 4);
    std::vector<float> taps;
    if (q > 1) taps = decimation_taps(q, 24, 8.6);
    const size_t b_taps = al(taps.size() * 4 + 4);
    uint8_t *base = nullptr;
    WUST_CUDA(cudaMallocAsync(&base, b_coef + b_fields + b_spec + b_rec + b_taps, st));
    uint8_t *q8 = base;
    auto take = [&](size_t b) { uint8_t *r = q8; q8 += al(b); return r; };
    SimCoefs k{};
    float *d_kappa = (float *)take(g.cplane * 4);
    float2 *d_dyp = (float2 *)take(std::max<size_t>(g.Nyh, g.Nx) * 8), *d_dyn = (float2 *)take(std::max<size_t>(g.Nyh, g.Nx) * 8);
    float2 *d_dxp = (float2 *)take(std::max<size_t>(g.Nyh, g.Nx) * 8), *d_dxn = (float2 *)take(std::max<size_t>(g.Nyh, g.Nx) * 8);
    float *d_pmly = (float *)take(g.Ny * 4), *d_pmlys = (float *)take(g.Ny * 4);
    float *d_pmlx = (float *)take(g.Nx * 4), *d_pmlxs = (float *)take(g.Nx * 4);
    float *d_c2 = (float *)take(g.plane * 4);
    int *d_rxslot = (int *)take(g.plane * 4);
    int *d_srcat = (int *)take(ntx * 4);
    float *d_src = (float *)take(nt * 4);
    int *d_t = (int *)take(4);
    q8 = base + b_coef;
    float *d_p = (float *)take((size_t)S * g.plane * 4);
    float *d_u = (float *)take((size_t)2 * S * g.plane * 4);
    q8 = base + b_coef + al((size_t)S * g.plane * 4) * 3;
    float *d_rho = (float *)take((size_t)2 * S * g.plane * 4);
    q8 = base + b_coef + al((size_t)S * g.plane * 4) * 5;
    float *d_g = (float *)take((size_t)2 * S * g.plane * 4);
    q8 = base + b_coef + b_fields;
    float2 *d_P = (float2 *)take((size_t)S * g.cplane * 8);
    float2 *d_G = (float2 *)take((size_t)2 * S * g.cplane * 8);
    q8 = base + b_coef + b_fields + b_spec;
    float *d_rec = (float *)take((size_t)S * nrx * nt * 4);
    q8 = base + b_coef + b_fields + b_spec + b_rec;
    float *d_taps = (float *)take(taps.size() * 4 + 4);

    WUST_CUDA(cudaMemcpyAsync(d_kappa, kappa.data(), g.cplane * 4, cudaMemcpyHostToDevice, st));
    WUST_CUDA(cudaMemcpyAsync(d_dyp, dyp.data(), g.Nyh * 8, cudaMemcpyHostToDevice, st));
    WUST_CUDA(cudaMemcpyAsync(d_dyn, dyn.data(), g.Nyh * 8, cudaMemcpyHostToDevice, st));
    WUST_CUDA(cudaMemcpyAsync(d_dxp, dxp.data(), g.Nx * 8, cudaMemcpyHostToDevice, st));
    WUST_CUDA(cudaMemcpyAsync(d_dxn, dxn.data(), g.Nx * 8, cudaMemcpyHostToDevice, st));
    WUST_CUDA(cudaMemcpyAsync(d_pmly, pmly.data(), g.Ny * 4, cudaMemcpyHostToDevice, st));
    WUST_CUDA(cudaMemcpyAsync(d_pmlys, pmlys.data(), g.Ny * 4, cudaMemcpyHostToDevice, st));
    WUST_CUDA(cudaMemcpyAsync(d_pmlx, pmlx.data(), g.Nx * 4, cudaMemcpyHostToDevice, st));
    WUST_CUDA(cudaMemcpyAsync(d_pmlxs, pmlxs.data(), g.Nx * 4, cudaMemcpyHostToDevice, st));
    WUST_CUDA(cudaMemcpyAsync(d_c2, c2.data(), g.plane * 4, cudaMemcpyHostToDevice, st));
    WUST_CUDA(cudaMemcpyAsync(d_rxslot, rx_slot.data(), g.plane * 4, cudaMemcpyHostToDevice, st));
    WUST_CUDA(cudaMemcpyAsync(d_src, srcf.data(), nt * 4, cudaMemcpyHostToDevice, st));
    if (q > 1) WUST_CUDA(cudaMemcpyAsync(d_taps, taps.data(), taps.size() * 4, cudaMemcpyHostToDevice, st));
    k.kappa = d_kappa;
    k.dyp = d_dyp; k.dyn = d_dyn; k.dxp = d_dxp; k.dxn = d_dxn;
    k.pmly = d_pmly; k.pmly_sg = d_pmlys; k.pmlx = d_pmlx; k.pmlx_sg = d_pmlxs;
    k.c2 = d_c2;
    k.inv_n = (float)(1.0 / ((double)g.Ny * g.Nx));
    k.dt_rho0 = (float)(a.dt * a.rho0);
    k.dt_over_rho0 = (float)(a.dt / a.rho0);

    // ---- FFT plans: S planes (p) and 2S planes (g, u) ----------------------
    cufftHandle fwd1 = 0, fwd2 = 0, inv2 = 0;
    int n2[2] = {g.Nx, g.Ny};
    struct PlanGuard {
        cufftHandle *h[3];
        uint8_t *mem;
        cudaStream_t st;
        ~PlanGuard() {
            for (auto p : h)
                if (*p) cufftDestroy(*p);
            if (mem) cudaFreeAsync(mem, st);
        }
    } guard{{&fwd1, &fwd2, &inv2}, base, st};
    WUST_CUFFT(cufftPlanMany(&fwd1, 2, n2, nullptr, 1, (int)g.plane, nullptr, 1, (int)g.cplane, CUFFT_R2C, S));
    WUST_CUFFT(cufftPlanMany(&fwd2, 2, n2, nullptr, 1, (int)g.plane, nullptr, 1, (int)g.cplane, CUFFT_R2C, 2 * S));
    WUST_CUFFT(cufftPlanMany(&inv2, 2, n2, nullptr, 1, (int)g.cplane, nullptr, 1, (int)g.plane, CUFFT_C2R, 2 * S));
    for (cufftHandle h : {fwd1, fwd2, inv2}) WUST_CUFFT(cufftSetStream(h, st));

    const int gp = sim_grid((size_t)S * g.plane), gc = sim_grid((size_t)S * g.cplane);
    for (int s0 = 0; s0 < ntx; s0 += S) {
        const int sb = std::min(S, ntx - s0);
        std::vector<int> src_at(S, -1);
        for (int s = 0; s < sb; ++s) src_at[s] = src_at_all[s0 + s];
        WUST_CUDA(cudaMemcpyAsync(d_srcat, src_at.data(), S * 4, cudaMemcpyHostToDevice, st));
        WUST_CUDA(cudaMemsetAsync(d_p, 0, al((size_t)S * g.plane * 4) * 7, st));   // p, u, rho, g
        WUST_CUDA(cudaMemsetAsync(d_t, 0, 4, st));
        if (q == 1) WUST_CUDA(cudaMemsetAsync(d_rec, 0, (size_t)S * nrx * nt * 4, st));
        auto step = [&]() {
            WUST_CUFFT(cufftExecR2C(fwd1, d_p, (cufftComplex *)d_P));
            sim_grad_kernel<<<gc, kSimThreads, 0, st>>>(g, k, d_P, d_G);
            WUST_CUFFT(cufftExecC2R(inv2, (cufftComplex *)d_G, d_g));
            sim_velocity_kernel<<<gp, kSimThreads, 0, st>>>(g, k, d_g, d_u);
            WUST_CUFFT(cufftExecR2C(fwd2, d_u, (cufftComplex *)d_G));
            sim_div_kernel<<<gc, kSimThreads, 0, st>>>(g, k, d_G);
            WUST_CUFFT(cufftExecC2R(inv2, (cufftComplex *)d_G, d_g));
            sim_density_kernel<<<gp, kSimThreads, 0, st>>>(g, k, d_g, d_rho, d_p, d_srcat, d_src, d_rxslot, nrx, nt,
                                                           d_t, d_rec);
            sim_tick_kernel<<<1, 1, 0, st>>>(d_t);
        };
        // one step captured as a graph and replayed; launched directly if the
        // capture is refused
        cudaGraph_t graph = nullptr;
        cudaGraphExec_t exec = nullptr;
        bool graphed = false;
        if (cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
            cudaGetLastError();
        } else {
            bool recorded = true;
            try {
                step();
            } catch (const WustError &) {
                recorded = false;
            }
            if (cudaStreamEndCapture(st, &graph) == cudaSuccess && graph && recorded &&
                cudaGraphInstantiate(&exec, graph, 0) == cudaSuccess)
                graphed = true;
            if (graph) cudaGraphDestroy(graph);
            cudaGetLastError();
        }
        for (int t = 0; t < nt; ++t) {
            if (graphed) WUST_CUDA(cudaGraphLaunch(exec, st));
            else step();
        }
        if (exec) cudaGraphExecDestroy(exec);
        g_kernel_launches += 5LL * nt;
        WUST_LAUNCH_CHECK();
        // records [s][r][t] -> rf [t][r][tx] column-major, i.e. memory [tx][r][t]
        float *dst = rf + (size_t)s0 * nrx * ly;
        if (q == 1) {
            WUST_CUDA(cudaMemcpyAsync(dst, d_rec, (size_t)sb * nrx * nt * 4, cudaMemcpyDeviceToDevice, st));
        } else {
            const size_t n_out = (size_t)sb * nrx * ly;
            sim_decimate_kernel<<<sim_grid(n_out), kSimThreads, 0, st>>>(d_rec, nt, sb * nrx, d_taps, (int)taps.size(),
                                                                          q, ly, dst);
            ++g_kernel_launches;
            WUST_LAUNCH_CHECK();
        }
    }
    WUST_CUDA(cudaStreamSynchronize(st));
}

}  // namespace wust
