// Mixed-radix FFTs of many lines in shared memory, in place: decimation in
// frequency takes natural order to digit-reversed order, decimation in time
// takes it back, so that a transform, a pointwise operation and the inverse
// transform need no reordering -- the pointwise operation's coefficients are
// laid out in the order of the positions.  Forward only: an inverse is the
// same on values with real and imaginary part exchanged.  Any length: a stage
// is one register butterfly per thread, of a radix up to 24 or of a prime up
// to 23, or a direct sum in shared memory (larger primes; all primes above 8
// where one small grid leaves few butterflies).  A stage costs a barrier, the
// shared memory's 24 bytes per point with its twiddle and some 40
// instructions per point, hence the large radices: 288 = 24 12, 552 = 24 23
// (12 2 23 took 0.96 ms a step where 24 23 takes 0.87).
#pragma once

#include <algorithm>

#include "common.cuh"

namespace wust {
namespace sim {

constexpr int kMaxStages = 12;

// A stage works on blocks of r m points; `per` butterflies a line, their
// twiddles `spacing` roots of unity apart.
struct FftStage {
    int r, m, len, spacing, per;
    float inv_m, inv_h;            // 1 / m, 1 / ((r - 1) / 2)
};
struct FftPlan {
    int n, stages;
    FftStage at[kMaxStages];
};

// Few stages, of radices up to `largest` (and primes).
inline FftPlan fft_plan(int n, int largest = 24) {
    FftPlan p{};
    p.n = n;
    int rest = n;
    auto take = [&](int r) {
        while (rest % r == 0 && p.stages < kMaxStages) {
            p.at[p.stages++].r = r;
            rest /= r;
        }
    };
    for (int r : {24, 16, 12, 10, 9, 8, 6, 5, 4, 3, 2, 7})
        if (r <= largest) take(r);
    for (int r = 3; rest > 1; r += 2) take(r);
    // an odd radix last: its butterflies are neighbours there, and an even number of rows apart they would share banks
    std::stable_partition(p.at, p.at + p.stages, [](const FftStage &s) { return s.r % 2 == 0; });
    int len = n;
    for (int i = 0; i < p.stages; ++i) {
        FftStage &s = p.at[i];
        s.len = len;
        s.m = len / s.r;
        s.spacing = n / len;
        s.per = n / s.r;
        s.inv_m = 1.0f / (float)s.m;
        s.inv_h = s.r > 2 ? 1.0f / (float)((s.r - 1) / 2) : 1.0f;
        len = s.m;
    }
    return p;
}

// The index that position i holds after the decimation in frequency.
inline int fft_index_at(const FftPlan &p, int i) {
    int f = 0, scale = 1;
    for (int s = 0; s < p.stages; ++s) {
        f += scale * (i / p.at[s].m);
        i %= p.at[s].m;
        scale *= p.at[s].r;
    }
    return f;
}

// All of a block's shared memory; lines and tables are named by their place in it, so
// that the compiler knows the address space and computes with 32 bits.
extern __shared__ __align__(128) float2 fft_sm[];

// The plans of a block, read at every stage: in shared memory (read as a
// kernel parameter through a call, a stage began with some 500 cycles of
// dependent loads and divisions).
__shared__ FftPlan fft_plans[2];
__device__ __forceinline__ void keep_plan(int which, const FftPlan &f) {
    for (int i = threadIdx.x; i < (int)(sizeof(FftPlan) / 4); i += blockDim.x)
        reinterpret_cast<int *>(&fft_plans[which])[i] = reinterpret_cast<const int *>(&f)[i];
}

// (e + 1/2) / n for 0 <= e < 2^21, inv = 1 / n
__device__ __forceinline__ int fast_div(int e, float inv) { return (int)(((float)e + 0.5f) * inv); }

// cos and sin of 2 pi j / p, j = 1 .. (p - 1) / 2, for the primes 3 .. 23
__constant__ float2 c_root[45] = {
    {-0.5f, 0.866025404f}, {0.309016994f, 0.951056516f}, {-0.809016994f, 0.587785252f}, {0.623489802f, 0.781831482f},
    {-0.222520934f, 0.974927912f}, {-0.900968868f, 0.433883739f}, {0.841253533f, 0.540640817f},
    {0.415415013f, 0.909631995f}, {-0.142314838f, 0.989821442f}, {-0.654860734f, 0.755749574f},
    {-0.959492974f, 0.281732557f}, {0.885456026f, 0.464723172f}, {0.568064747f, 0.822983866f},
    {0.12053668f, 0.992708874f}, {-0.354604887f, 0.935016243f}, {-0.748510748f, 0.663122658f},
    {-0.970941817f, 0.239315664f}, {0.932472229f, 0.361241666f}, {0.739008917f, 0.673695644f},
    {0.445738356f, 0.895163291f}, {0.0922683595f, 0.995734176f}, {-0.27366299f, 0.961825643f},
    {-0.602634636f, 0.798017227f}, {-0.850217136f, 0.526432163f}, {-0.9829731f, 0.183749518f},
    {0.945817242f, 0.324699469f}, {0.789140509f, 0.614212713f}, {0.546948158f, 0.837166478f},
    {0.245485487f, 0.969400266f}, {-0.0825793455f, 0.996584493f}, {-0.401695425f, 0.915773327f},
    {-0.677281572f, 0.735723911f}, {-0.879473751f, 0.475947393f}, {-0.986361303f, 0.16459459f},
    {0.962917287f, 0.269796771f}, {0.854419405f, 0.51958395f}, {0.682553143f, 0.730835964f},
    {0.460065038f, 0.887885218f}, {0.203456013f, 0.979084088f}, {-0.0682424134f, 0.997668769f},
    {-0.334879612f, 0.942260922f}, {-0.576680322f, 0.816969893f}, {-0.775711291f, 0.631087944f},
    {-0.917211302f, 0.39840109f}, {-0.990685946f, 0.136166649f},
};
constexpr int root_at(int p) {
    return p == 3 ? 0 : p == 5 ? 1 : p == 7 ? 3 : p == 11 ? 6 : p == 13 ? 11 : p == 17 ? 17 : p == 19 ? 25 : 34;
}

__device__ __forceinline__ float2 fadd2(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 fsub2(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 turn2(float2 a) { return make_float2(a.y, -a.x); }          // times -i

// x[k] <- sum_j x[j] exp(-2 pi i j k / R)
template <int R>
struct Dft;
template <>
struct Dft<2> {
    static __device__ __forceinline__ void run(float2 (&x)[2]) {
        const float2 t = x[0];
        x[0] = fadd2(t, x[1]);
        x[1] = fsub2(t, x[1]);
    }
};
template <>
struct Dft<4> {
    static __device__ __forceinline__ void run(float2 (&x)[4]) {
        const float2 s = fadd2(x[0], x[2]), t = fsub2(x[0], x[2]), u = fadd2(x[1], x[3]), v = turn2(fsub2(x[1], x[3]));
        x[0] = fadd2(s, u);
        x[2] = fsub2(s, u);
        x[1] = fadd2(t, v);
        x[3] = fsub2(t, v);
    }
};
template <>
struct Dft<8> {
    static __device__ __forceinline__ void run(float2 (&x)[8]) {
        float2 e[4] = {x[0], x[2], x[4], x[6]}, o[4] = {x[1], x[3], x[5], x[7]};
        Dft<4>::run(e);
        Dft<4>::run(o);
        constexpr float c = 0.70710678118654752f;
        o[1] = make_float2(c * (o[1].x + o[1].y), c * (o[1].y - o[1].x));
        o[2] = turn2(o[2]);
        o[3] = make_float2(c * (o[3].y - o[3].x), -c * (o[3].x + o[3].y));
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            x[k] = fadd2(e[k], o[k]);
            x[k + 4] = fsub2(e[k], o[k]);
        }
    }
};
template <>
struct Dft<16> {
    static __device__ __forceinline__ void run(float2 (&x)[16]) {
        constexpr float c1 = 0.92387953251128676f, s1 = 0.38268343236508977f, c2 = 0.70710678118654752f;
        float2 y[4][4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
#pragma unroll
            for (int b = 0; b < 4; ++b) y[a][b] = x[a + 4 * b];
            Dft<4>::run(y[a]);
        }
        // y[a][k] times exp(-2 pi i a k / 16)
        auto by = [](float2 v, float c, float s) { return make_float2(c * v.x + s * v.y, c * v.y - s * v.x); };
        y[1][1] = by(y[1][1], c1, s1);
        y[1][2] = by(y[1][2], c2, c2);
        y[1][3] = by(y[1][3], s1, c1);
        y[2][1] = by(y[2][1], c2, c2);
        y[2][2] = turn2(y[2][2]);
        y[2][3] = by(y[2][3], -c2, c2);
        y[3][1] = by(y[3][1], s1, c1);
        y[3][2] = by(y[3][2], -c2, c2);
        y[3][3] = by(y[3][3], -c1, -s1);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            float2 z[4] = {y[0][k], y[1][k], y[2][k], y[3][k]};
            Dft<4>::run(z);
#pragma unroll
            for (int a = 0; a < 4; ++a) x[k + 4 * a] = z[a];
        }
    }
};
template <>
struct Dft<9> {
    static __device__ __forceinline__ void run(float2 (&x)[9]);
};
// odd primes: x_j + x_{R-j} meets the cosines, x_j - x_{R-j} the sines; emit(k, value) takes the results as they come
template <int R, typename Emit>
__device__ __forceinline__ void dft_prime(float2 (&x)[R], Emit emit) {
    constexpr int H = (R - 1) / 2;
    float2 sum = x[0];
#pragma unroll
    for (int j = 1; j <= H; ++j) {
        const float2 s = fadd2(x[j], x[R - j]);
        x[R - j] = fsub2(x[j], x[R - j]);
        x[j] = s;
        sum = fadd2(sum, s);
    }
    emit(0, sum);
#pragma unroll
    for (int k = 1; k <= H; ++k) {
        float2 a = x[0], b = make_float2(0.f, 0.f);
#pragma unroll
        for (int j = 1; j <= H; ++j) {
            const int i = j * k % R, m = i <= H ? i : R - i;
            const float c = c_root[root_at(R) + m - 1].x, s = c_root[root_at(R) + m - 1].y;
            a.x = fmaf(c, x[j].x, a.x);
            a.y = fmaf(c, x[j].y, a.y);
            b.x = fmaf(i <= H ? s : -s, x[R - j].x, b.x);
            b.y = fmaf(i <= H ? s : -s, x[R - j].y, b.y);
        }
        emit(k, make_float2(a.x + b.y, a.y - b.x));          // a - i b
        emit(R - k, make_float2(a.x - b.y, a.y + b.x));
    }
}
template <int R>
struct Dft {
    static __device__ __forceinline__ void run(float2 (&x)[R]) {
        float2 y[R];
        dft_prime<R>(x, [&](int k, float2 v) { y[k] = v; });
#pragma unroll
        for (int k = 0; k < R; ++k) x[k] = y[k];
    }
};
__device__ __forceinline__ void Dft<9>::run(float2 (&x)[9]) {
    float2 y[3][3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
#pragma unroll
        for (int b = 0; b < 3; ++b) y[a][b] = x[a + 3 * b];
        Dft<3>::run(y[a]);
    }
    constexpr float c1 = 0.76604444311897804f, s1 = 0.64278760968653933f, c2 = 0.17364817766693035f, s2 = 0.98480775301220806f,
                    c4 = -0.93969262078590838f, s4 = 0.34202014332566873f;
    auto by = [](float2 v, float c, float s) { return make_float2(c * v.x + s * v.y, c * v.y - s * v.x); };
    y[1][1] = by(y[1][1], c1, s1);
    y[1][2] = by(y[1][2], c2, s2);
    y[2][1] = by(y[2][1], c2, s2);
    y[2][2] = by(y[2][2], c4, s4);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        float2 z[3] = {y[0][k], y[1][k], y[2][k]};
        Dft<3>::run(z);
#pragma unroll
        for (int a = 0; a < 3; ++a) x[k + 3 * a] = z[a];
    }
}
// coprime A B: index maps by the Chinese remainder theorem, no twiddles
constexpr int inv_mod(int a, int m) {
    for (int i = 1; i < m; ++i)
        if (a * i % m == 1) return i;
    return 0;
}
template <int A, int B>
struct DftCoprime {
    static __device__ __forceinline__ void run(float2 (&x)[A * B]) {
        constexpr int N = A * B;
        float2 y[B][A];
#pragma unroll
        for (int b = 0; b < B; ++b) {
#pragma unroll
            for (int a = 0; a < A; ++a) y[b][a] = x[(a * B + b * A) % N];
            Dft<A>::run(y[b]);
        }
#pragma unroll
        for (int a = 0; a < A; ++a) {
            float2 z[B];
#pragma unroll
            for (int b = 0; b < B; ++b) z[b] = y[b][a];
            Dft<B>::run(z);
#pragma unroll
            for (int b = 0; b < B; ++b) x[(a * B * inv_mod(B % A, A) + b * A * inv_mod(A % B, B)) % N] = z[b];
        }
    }
};
template <>
struct Dft<6> : DftCoprime<2, 3> {};
template <>
struct Dft<10> : DftCoprime<2, 5> {};
template <>
struct Dft<12> : DftCoprime<4, 3> {};
template <>
struct Dft<24> : DftCoprime<8, 3> {};

// How the lines lie: element n of line l at offset(l) + n * stride().
// A tile: `sets` planes of n rows of 2^LOG lines each.
template <int LOG>
struct TileLines {
    int sets, plane;
    __device__ __forceinline__ int count() const { return sets << LOG; }
    __device__ __forceinline__ int stride() const { return 1 << LOG; }
    __device__ __forceinline__ int offset(int l) const { return (l & ((1 << LOG) - 1)) + (l >> LOG) * plane; }
    // work item -> its line's offset and its butterfly out of `per`
    __device__ __forceinline__ void split(int it, int per, int &off, int &b) const {
        off = it & ((1 << LOG) - 1);
        b = it >> LOG;
        if (b >= per) {
            b -= per;
            off += plane;
        }
    }
};
// Rows or columns of one plane.
struct GridLines {
    int lines, between, along;     // distance of neighbouring lines, of neighbouring elements
    float inv;                     // 1 / lines
    __device__ __forceinline__ int count() const { return lines; }
    __device__ __forceinline__ int stride() const { return along; }
    __device__ __forceinline__ int offset(int l) const { return l * between; }
    __device__ __forceinline__ void split(int it, int, int &off, int &b) const {
        b = fast_div(it, inv);
        off = (it - b * lines) * between;
    }
};

// One stage of register butterflies, a work item one butterfly of one line.
template <int R, bool DIT, class Lines>
__device__ __forceinline__ void stage_small(int z, const Lines &lines, const FftStage &f, int tw) {
    const int M = f.m, spacing = f.spacing, per = f.per, items = per * lines.count(), step = M * lines.stride(), len = f.len;
    const float inv = f.inv_m;
    for (int it = threadIdx.x; it < items; it += blockDim.x) {
        int off, b;
        lines.split(it, per, off, b);
        const int blk = M == 1 ? b : fast_div(b, inv), q = b - blk * M;
        float2 *p = fft_sm + z + off + (blk * len + q) * lines.stride();
        const float2 *w = fft_sm + tw;
        const int turn = spacing * q;
        float2 x[R];
#pragma unroll
        for (int j = 0; j < R; ++j) x[j] = p[j * step];
        if (DIT && M > 1)
#pragma unroll
            for (int j = 1; j < R; ++j) x[j] = cmul(x[j], w[turn * j]);
        auto emit = [&](int k, float2 v) {
            if (!DIT && M > 1 && k) v = cmul(v, w[turn * k]);
            p[k * step] = v;
        };
        if constexpr (R > 9 && R % 2 == 1) {
            dft_prime<R>(x, emit);
        } else {
            Dft<R>::run(x);
#pragma unroll
            for (int k = 0; k < R; ++k) emit(k, x[k]);
        }
    }
}

// One stage of an odd p by direct sums.  A first pass turns the entries j
// and p - j into their sum and difference (and, in time, gives them their
// twiddles); a thread then sums KT outputs k (and their mirrors p - k) of CT
// adjacent lines of one butterfly, straight from shared memory.  Neighbouring
// threads take neighbouring lines, so that roots are read once a warp and
// lines without conflicts.  Passes over whole butterflies: nobody writes what
// another thread has yet to read.
template <int KT, int CT, bool DIT, class Lines>
__device__ __forceinline__ void stage_prime(int z, const Lines &lines, const FftStage &f, int tw) {
    const int p = f.r, M = f.m, h = (p - 1) / 2, spacing = f.spacing, per = f.per, root = per, stride = lines.stride();
    const int step = M * stride, len = f.len;
    const float inv = f.inv_m, inv_h = f.inv_h;
    const float2 *w = fft_sm + tw;
    auto place = [&](int b, int &q) {
        const int blk = M == 1 ? b : fast_div(b, inv);
        q = b - blk * M;
        return (blk * len + q) * stride;
    };
    {
        const int items = per * h * lines.count();
        for (int it = threadIdx.x; it < items; it += blockDim.x) {
            int off, r, q;
            lines.split(it, per * h, off, r);
            const int b = fast_div(r, inv_h), j = r - b * h + 1;
            float2 *base = fft_sm + z + off + place(b, q);
            float2 x = base[j * step], y = base[(p - j) * step];
            if (DIT && q) {
                x = cmul(x, w[spacing * q * j]);
                y = cmul(y, w[spacing * q * (p - j)]);
            }
            base[j * step] = fadd2(x, y);
            base[(p - j) * step] = fsub2(x, y);
        }
    }
    __syncthreads();
    const int per_line = lines.count() / CT, groups = per * per_line, kg = (h + KT - 1) / KT;
    const int block = max(1, min(groups, (int)blockDim.x / kg));                 // butterflies of a pass
    const int kq = threadIdx.x / block, cq = threadIdx.x - kq * block, next = lines.offset(1);
    for (int g0 = 0; g0 < groups; g0 += block) {
        const int g = g0 + cq;
        const bool on = kq < kg && g < groups;
        int q;
        float2 *base = fft_sm + z + (on ? lines.offset(CT * (g % per_line)) + place(g / per_line, q) : 0);
        if (!on) q = 0;
        float2 a[KT][CT], s[KT][CT], sum[CT];
        int idx[KT];
#pragma unroll
        for (int c = 0; c < CT; ++c) sum[c] = on ? base[c * next] : make_float2(0.f, 0.f);   // others are writing elsewhere
#pragma unroll
        for (int t = 0; t < KT; ++t) {
            idx[t] = 0;
#pragma unroll
            for (int c = 0; c < CT; ++c) {
                a[t][c] = sum[c];
                s[t][c] = make_float2(0.f, 0.f);
            }
        }
        if (on)
#pragma unroll 2
            for (int j = 1; j <= h; ++j) {
                float2 u[CT], v[CT];
#pragma unroll
                for (int c = 0; c < CT; ++c) {
                    u[c] = base[j * step + c * next];
                    v[c] = base[(p - j) * step + c * next];
                    sum[c] = fadd2(sum[c], u[c]);
                }
#pragma unroll
                for (int t = 0; t < KT; ++t) {
                    idx[t] += kq * KT + t + 1;
                    if (idx[t] >= p) idx[t] -= p;
                    const float2 r = w[root * idx[t]];           // (cos, -sin)
#pragma unroll
                    for (int c = 0; c < CT; ++c) {
                        a[t][c].x = fmaf(r.x, u[c].x, a[t][c].x);
                        a[t][c].y = fmaf(r.x, u[c].y, a[t][c].y);
                        s[t][c].x = fmaf(r.y, v[c].x, s[t][c].x);
                        s[t][c].y = fmaf(r.y, v[c].y, s[t][c].y);
                    }
                }
            }
        __syncthreads();
        if (on) {
#pragma unroll
            for (int t = 0; t < KT; ++t) {
                const int k = kq * KT + t + 1;
                if (k > h) continue;
#pragma unroll
                for (int c = 0; c < CT; ++c) {                   // a - i b with s = -b
                    float2 y1 = make_float2(a[t][c].x - s[t][c].y, a[t][c].y + s[t][c].x);
                    float2 y2 = make_float2(a[t][c].x + s[t][c].y, a[t][c].y - s[t][c].x);
                    if (!DIT && q) {
                        y1 = cmul(y1, w[spacing * q * k]);
                        y2 = cmul(y2, w[spacing * q * (p - k)]);
                    }
                    base[k * step + c * next] = y1;
                    base[(p - k) * step + c * next] = y2;
                }
            }
            if (kq == 0)
#pragma unroll
                for (int c = 0; c < CT; ++c) base[c * next] = sum[c];
        }
    }
}

// All stages of the lines at fft_sm[z], roots of unity at fft_sm[tw].  Ends
// with a barrier.  Tiles: many lines keep the block busy with large radices.
template <bool DIT, int LOG>
__device__ __noinline__ void fft_lines(int z, TileLines<LOG> lines, int plan, int tw) {
    const int stages = fft_plans[plan].stages;
#pragma unroll 1
    for (int st = 0; st < stages; ++st) {
        const FftStage &f = fft_plans[plan].at[DIT ? stages - 1 - st : st];
        switch (f.r) {
            case 2: stage_small<2, DIT>(z, lines, f, tw); break;
            case 3: stage_small<3, DIT>(z, lines, f, tw); break;
            case 4: stage_small<4, DIT>(z, lines, f, tw); break;
            case 5: stage_small<5, DIT>(z, lines, f, tw); break;
            case 6: stage_small<6, DIT>(z, lines, f, tw); break;
            case 7: stage_small<7, DIT>(z, lines, f, tw); break;
            case 8: stage_small<8, DIT>(z, lines, f, tw); break;
            case 9: stage_small<9, DIT>(z, lines, f, tw); break;
            case 10: stage_small<10, DIT>(z, lines, f, tw); break;
            case 11: stage_small<11, DIT>(z, lines, f, tw); break;
            case 12: stage_small<12, DIT>(z, lines, f, tw); break;
            case 13: stage_small<13, DIT>(z, lines, f, tw); break;
            case 16: stage_small<16, DIT>(z, lines, f, tw); break;
            case 17: stage_small<17, DIT>(z, lines, f, tw); break;
            case 19: stage_small<19, DIT>(z, lines, f, tw); break;
            case 23: stage_small<23, DIT>(z, lines, f, tw); break;
            case 24: stage_small<24, DIT>(z, lines, f, tw); break;
            default: {
                // outputs and lines per thread: more where that keeps the block busy
                const int h = (f.r - 1) / 2, wide = f.per * (lines.count() / 2) * ((h + 3) / 4);
                if (wide >= (int)blockDim.x / 2 || h > (int)blockDim.x) stage_prime<4, 2, DIT>(z, lines, f, tw);
                else stage_prime<1, 1, DIT>(z, lines, f, tw);
            }
        }
        __syncthreads();
    }
}
// One small grid: little to do in a stage, so small radices, many threads.
template <bool DIT>
__device__ __noinline__ void fft_lines(int z, GridLines lines, int plan, int tw) {
    const int stages = fft_plans[plan].stages;
#pragma unroll 1
    for (int st = 0; st < stages; ++st) {
        const FftStage &f = fft_plans[plan].at[DIT ? stages - 1 - st : st];
        switch (f.r) {
            case 2: stage_small<2, DIT>(z, lines, f, tw); break;
            case 3: stage_small<3, DIT>(z, lines, f, tw); break;
            case 4: stage_small<4, DIT>(z, lines, f, tw); break;
            case 5: stage_small<5, DIT>(z, lines, f, tw); break;
            case 6: stage_small<6, DIT>(z, lines, f, tw); break;
            case 7: stage_small<7, DIT>(z, lines, f, tw); break;
            case 8: stage_small<8, DIT>(z, lines, f, tw); break;
            default: {
                // outputs per thread: more where there is work enough for all threads
                const int work = f.per * lines.count() * ((f.r - 1) / 2), all = blockDim.x;
                if (work <= all) stage_prime<1, 1, DIT>(z, lines, f, tw);
                else if (work <= 2 * all) stage_prime<2, 1, DIT>(z, lines, f, tw);
                else stage_prime<4, 1, DIT>(z, lines, f, tw);
            }
        }
        __syncthreads();
    }
}

}  // namespace sim
}  // namespace wust
