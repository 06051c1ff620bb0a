// Complex FP32 transforms of lines held by one block of 256 threads, for
// arec_ccorr.cu (shift search, Fourier shift).
//
// Stockham passes with the data in registers: a block takes G = 4096 / N lines
// of N points, 16 points per thread.  The first pass reads its points straight
// from the caller (global memory), the last leaves the results in registers
// (or hands them to the caller), so P passes exchange through shared memory
// P - 1 times.  Twiddles come from a table laid out per pass (k contiguous,
// Ns entries per radix leg), so a warp's loads are consecutive: entry
// Ns - 1 + (r - 1) Ns + k is exp(-2 pi i r k / (Ns R)), N - 1 entries in all,
// computed in double on the host.
//
// Powers of two from 16 (template N): radix 16/8/4/2 passes, all indices
// compile-time.  Other lengths with prime factors 2, 3, 5 and 7 (and 2, 4, 8):
// a run-time list of radices out of {2..10, 16}, divisions by multiplication.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace arecgb {
namespace fft {

constexpr int kThreads = 256;
constexpr int kElems = 4096;  // points per block (16 per thread)
constexpr int kMaxPass = 8;

__device__ __forceinline__ float2 operator+(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 operator-(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 mul_mi(float2 a) { return make_float2(a.y, -a.x); }  // -i a
__device__ __forceinline__ float2 axpy(float c, float2 x, float2 y) {
    return make_float2(fmaf(c, x.x, y.x), fmaf(c, x.y, y.y));
}

// Forward DFT of R values in registers, natural order in and out.
template <int R>
__device__ __forceinline__ void dft(float2 *v) {
    if constexpr (R == 2) {
        const float2 a = v[0], b = v[1];
        v[0] = a + b;
        v[1] = a - b;
    } else if constexpr (R == 3) {
        const float2 t = v[1] + v[2], d = mul_mi(v[1] - v[2]);
        const float2 m = axpy(-0.5f, t, v[0]);
        const float s = 0.86602540378443865f;
        v[0] = v[0] + t;
        v[1] = axpy(s, d, m);
        v[2] = axpy(-s, d, m);
    } else if constexpr (R == 4) {
        const float2 t0 = v[0] + v[2], t1 = v[0] - v[2];
        const float2 t2 = v[1] + v[3], t3 = mul_mi(v[1] - v[3]);
        v[0] = t0 + t2;
        v[1] = t1 + t3;
        v[2] = t0 - t2;
        v[3] = t1 - t3;
    } else if constexpr (R == 5) {
        const float c1 = 0.30901699437494742f, c2 = -0.80901699437494742f;
        const float s1 = 0.95105651629515357f, s2 = 0.58778525229247313f;
        const float2 t1 = v[1] + v[4], t2 = v[2] + v[3];
        const float2 d1 = mul_mi(v[1] - v[4]), d2 = mul_mi(v[2] - v[3]);
        const float2 m1 = axpy(c2, t2, axpy(c1, t1, v[0])), m2 = axpy(c1, t2, axpy(c2, t1, v[0]));
        const float2 n1 = axpy(s2, d2, make_float2(s1 * d1.x, s1 * d1.y));
        const float2 n2 = axpy(-s1, d2, make_float2(s2 * d1.x, s2 * d1.y));
        v[0] = v[0] + t1 + t2;
        v[1] = m1 + n1;
        v[4] = m1 - n1;
        v[2] = m2 + n2;
        v[3] = m2 - n2;
    } else if constexpr (R == 7) {
        const float c1 = 0.62348980185873353f, c2 = -0.22252093395631440f, c3 = -0.90096886790241913f;
        const float s1 = 0.78183148246802981f, s2 = 0.97492791218182361f, s3 = 0.43388373911755812f;
        const float2 t1 = v[1] + v[6], t2 = v[2] + v[5], t3 = v[3] + v[4];
        const float2 d1 = mul_mi(v[1] - v[6]), d2 = mul_mi(v[2] - v[5]), d3 = mul_mi(v[3] - v[4]);
        const float2 z = make_float2(0.f, 0.f);
        const float2 m1 = axpy(c3, t3, axpy(c2, t2, axpy(c1, t1, v[0])));
        const float2 m2 = axpy(c1, t3, axpy(c3, t2, axpy(c2, t1, v[0])));
        const float2 m3 = axpy(c2, t3, axpy(c1, t2, axpy(c3, t1, v[0])));
        const float2 n1 = axpy(s3, d3, axpy(s2, d2, axpy(s1, d1, z)));
        const float2 n2 = axpy(-s1, d3, axpy(-s3, d2, axpy(s2, d1, z)));
        const float2 n3 = axpy(s2, d3, axpy(-s1, d2, axpy(s3, d1, z)));
        v[0] = v[0] + t1 + t2 + t3;
        v[1] = m1 + n1;
        v[6] = m1 - n1;
        v[2] = m2 + n2;
        v[5] = m2 - n2;
        v[3] = m3 + n3;
        v[4] = m3 - n3;
    } else if constexpr (R == 8) {
        const float h = 0.70710678118654752f;
        float2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
        dft<4>(e);
        dft<4>(o);
        o[1] = make_float2(h * (o[1].x + o[1].y), h * (o[1].y - o[1].x));
        o[2] = mul_mi(o[2]);
        o[3] = make_float2(h * (o[3].y - o[3].x), -h * (o[3].x + o[3].y));
#pragma unroll
        for (int k = 0; k < 4; k++) {
            v[k] = e[k] + o[k];
            v[k + 4] = e[k] - o[k];
        }
    } else if constexpr (R == 16) {
        const float h = 0.70710678118654752f, c = 0.92387953251128676f, s = 0.38268343236508977f;
        float2 a[4][4];
#pragma unroll
        for (int n = 0; n < 4; n++) {
#pragma unroll
            for (int m = 0; m < 4; m++) a[n][m] = v[n + 4 * m];
            dft<4>(a[n]);
        }
        // a[n][k] *= exp(-2 pi i n k / 16)
        a[1][1] = cmul(a[1][1], make_float2(c, -s));
        a[1][2] = make_float2(h * (a[1][2].x + a[1][2].y), h * (a[1][2].y - a[1][2].x));
        a[1][3] = cmul(a[1][3], make_float2(s, -c));
        a[2][1] = make_float2(h * (a[2][1].x + a[2][1].y), h * (a[2][1].y - a[2][1].x));
        a[2][2] = mul_mi(a[2][2]);
        a[2][3] = make_float2(h * (a[2][3].y - a[2][3].x), -h * (a[2][3].x + a[2][3].y));
        a[3][1] = cmul(a[3][1], make_float2(s, -c));
        a[3][2] = make_float2(h * (a[3][2].y - a[3][2].x), -h * (a[3][2].x + a[3][2].y));
        a[3][3] = cmul(a[3][3], make_float2(-c, s));
#pragma unroll
        for (int k = 0; k < 4; k++) {
            float2 b[4] = {a[0][k], a[1][k], a[2][k], a[3][k]};
            dft<4>(b);
#pragma unroll
            for (int m = 0; m < 4; m++) v[k + 4 * m] = b[m];
        }
    } else if constexpr (R == 6 || R == 10) {
        // prime-factor split R = 2 Q (Q = 3, 5): no twiddles.  With
        // n = Q n1 + 2 n2 and k = Q k1 + (Q + 1) k2 (mod R), n k / R is
        // n1 k1 / 2 + n2 k2 / Q modulo 1.
        constexpr int Q = R / 2;
        float2 a[2][Q];
#pragma unroll
        for (int n1 = 0; n1 < 2; n1++) {
#pragma unroll
            for (int n2 = 0; n2 < Q; n2++) a[n1][n2] = v[(Q * n1 + 2 * n2) % R];
            dft<Q>(a[n1]);
        }
#pragma unroll
        for (int k2 = 0; k2 < Q; k2++) {
            v[((Q + 1) * k2) % R] = a[0][k2] + a[1][k2];
            v[(Q + (Q + 1) * k2) % R] = a[0][k2] - a[1][k2];
        }
    } else {
        static_assert(R == 9, "radices 2..10 and 16");
        // exp(-2 pi i m / 9), m = 1, 2, 4
        const float2 w1 = make_float2(0.76604444311897804f, -0.64278760968653933f);
        const float2 w2 = make_float2(0.17364817766693036f, -0.98480775301220806f);
        const float2 w4 = make_float2(-0.93969262078590838f, -0.34202014332566873f);
        float2 a[3][3];
#pragma unroll
        for (int n = 0; n < 3; n++) {
#pragma unroll
            for (int m = 0; m < 3; m++) a[n][m] = v[n + 3 * m];
            dft<3>(a[n]);
        }
        a[1][1] = cmul(a[1][1], w1);
        a[1][2] = cmul(a[1][2], w2);
        a[2][1] = cmul(a[2][1], w2);
        a[2][2] = cmul(a[2][2], w4);
#pragma unroll
        for (int k = 0; k < 3; k++) {
            float2 b[3] = {a[0][k], a[1][k], a[2][k]};
            dft<3>(b);
#pragma unroll
            for (int m = 0; m < 3; m++) v[k + 3 * m] = b[m];
        }
    }
}

// Shared-memory lines carry one pad element per 16: a Stockham pass writes
// with a stride of its radix while Ns = 1, which would fall in few banks.
__device__ __host__ __forceinline__ constexpr int pz(int i) { return i + (i >> 4); }
__device__ __host__ __forceinline__ constexpr int plen(int n) { return n + (n >> 4); }

// ---------------------------------------------------------------------------
// Powers of two, 16 <= N <= 4096.

// Radices of the passes, in order; the reversed order starts a transform on
// the registers the other order ends with.
template <int N>
struct Pow2 {
    static constexpr int R0 = N >= 1024 || N == 256 || N <= 128 ? 16 : 8;
    static constexpr int R1 = N == 512 ? 8 : (N / R0 > 16 ? 16 : N / R0);
    static constexpr int R2 = N / (R0 * R1);
    static constexpr int TPL = N / 16;        // threads per line
    static constexpr int G = kElems / N;      // lines per block
    static constexpr int P = R2 > 1 ? 3 : (R1 > 1 ? 2 : 1);
    // radix of pass p in forward (REV = false) or reversed order
    template <bool REV>
    static constexpr int radix(int p) {
        const int q = REV ? P - 1 - p : p;
        return q == 0 ? R0 : (q == 1 ? R1 : R2);
    }
};

// A block's lines exchange only within a warp when a line has <= 32 threads
// (its threads are then in one warp: rows order).
template <bool WARP>
__device__ __forceinline__ void exchange_sync() {
    if constexpr (WARP)
        __syncwarp();
    else
        __syncthreads();
}

// One pass boundary: v holds pass p's outputs (radix R, stride Ns); leaves in
// v the inputs of the next pass (radix RN, stride Ns * R), twiddled.
// b: the thread's index in its line; L: the line in shared memory.
template <int N, int R, int RN, int Ns, bool WARP, int K, typename T>
__device__ __forceinline__ void exchange(float2 (&v)[K][16], T *L, int b, const float2 *tw) {
    constexpr int TPL = N / 16;
    exchange_sync<WARP>();  // earlier reads of the buffer
#pragma unroll
    for (int i = 0; i < 16 / R; i++) {
        const int j = b + i * TPL, k = j & (Ns - 1), d = (j / Ns) * Ns * R + k;
#pragma unroll
        for (int r = 0; r < R; r++) {
            if constexpr (K == 1)
                L[pz(d + r * Ns)] = v[0][i * R + r];
            else
                L[pz(d + r * Ns)] = make_float4(v[0][i * R + r].x, v[0][i * R + r].y,
                                                v[1][i * R + r].x, v[1][i * R + r].y);
        }
    }
    exchange_sync<WARP>();
    constexpr int NsN = Ns * R;
#pragma unroll
    for (int i = 0; i < 16 / RN; i++) {
        const int j = b + i * TPL, k = j & (NsN - 1);
#pragma unroll
        for (int r = 0; r < RN; r++) {
            const T x = L[pz(j + r * (N / RN))];
            v[0][i * RN + r] = make_float2(x.x, x.y);
            if constexpr (K == 2) v[1][i * RN + r] = make_float2(x.z, x.w);
            if (r > 0) {
                const float2 w = __ldg(tw + NsN - 1 + (r - 1) * NsN + k);
#pragma unroll
                for (int c = 0; c < K; c++) v[c][i * RN + r] = cmul(v[c][i * RN + r], w);
            }
        }
    }
}

template <int R, int K>
__device__ __forceinline__ void butterflies(float2 (&v)[K][16]) {
#pragma unroll
    for (int c = 0; c < K; c++)
#pragma unroll
        for (int i = 0; i < 16 / R; i++) dft<R>(&v[c][i * R]);
}

// Forward transforms of K lines' worth of points per thread, in step (K = 1:
// T = float2; K = 2: T = float4, the two lines interleaved).  In: v[c][i * R +
// r] = point (b + i TPL) + r N / R with R the first radix; out: the same with
// the last radix.
template <int N, bool REV, bool WARP, int K, typename T>
__device__ __forceinline__ void transform(float2 (&v)[K][16], T *L, int b, const float2 *tw) {
    using P = Pow2<N>;
    constexpr int Ra = P::template radix<REV>(0);
    butterflies<Ra, K>(v);
    if constexpr (P::P > 1) {
        constexpr int Rb = P::template radix<REV>(1);
        exchange<N, Ra, Rb, 1, WARP, K, T>(v, L, b, tw);
        butterflies<Rb, K>(v);
        if constexpr (P::P > 2) {
            constexpr int Rc = P::template radix<REV>(2);
            exchange<N, Rb, Rc, Ra, WARP, K, T>(v, L, b, tw);
            butterflies<Rc, K>(v);
        }
    }
}

// ---------------------------------------------------------------------------
// Any length 2..4096 with prime factors 2, 3, 5, 7.

// n / d for n * d < 2^32 (d > 1) by one multiplication.
struct FastDiv {
    uint32_t d, m;
};
__device__ __forceinline__ int fdiv(int n, FastDiv f) {
    return f.d == 1 ? n : (int)__umulhi((uint32_t)n, f.m);
}
static inline FastDiv make_fastdiv(int d) {
    return FastDiv{(uint32_t)d, d > 1 ? (uint32_t)((0x100000000ull + d - 1) / d) : 0u};
}

// A transform's passes: radix r[p], stride ns[p] (the product of the earlier
// radices), with the divisors its index arithmetic needs.
struct Passes {
    int n, np;
    FastDiv dn;  // by n
    int r[kMaxPass], ns[kMaxPass];
    FastDiv dnr[kMaxPass], dns[kMaxPass];  // by n / r and by ns
};

// One pass of radix R over G lines from shared memory src to dst (line l's
// point i at [l * ls + pz(i)]).  Two buffers, so a butterfly's registers live
// only through its own loads and stores.  COLS: consecutive threads take
// consecutive lines (the columns of a tile; G a power of two, lg = log2 G),
// else consecutive points.  K = 2: both complex halves of float4 points; K = 1
// over float4 points: the first half.
template <int R, int K, bool COLS, typename T>
__device__ __forceinline__ void mixed_pass(const Passes &P, int p, int G, int lg, const T *src,
                                           T *dst, int ls, const float2 *__restrict__ tw) {
    const int NR = P.n / R, B = G * NR, Ns = P.ns[p];
    const FastDiv dnr = P.dnr[p], dns = P.dns[p];
#pragma unroll 1
    for (int t = threadIdx.x; t < B; t += kThreads) {
        const int line = COLS ? t & (G - 1) : fdiv(t, dnr);
        const int j = COLS ? t >> lg : t - line * NR;
        const int q = fdiv(j, dns), k = j - q * Ns;
        const T *s = src + line * ls;
        T *d = dst + line * ls;
        const float2 *w = tw + Ns - 1 + k;
        float2 v[K][R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            if constexpr (K == 2) {
                const T x = s[pz(j + r * NR)];
                v[0][r] = make_float2(x.x, x.y);
                v[1][r] = make_float2(x.z, x.w);
            } else {
                v[0][r] = *reinterpret_cast<const float2 *>(s + pz(j + r * NR));
            }
            if (r > 0) {
                const float2 wr = __ldg(w + (r - 1) * Ns);
#pragma unroll
                for (int c = 0; c < K; c++) v[c][r] = cmul(v[c][r], wr);
            }
        }
#pragma unroll
        for (int c = 0; c < K; c++) dft<R>(v[c]);
        const int o = q * Ns * R + k;
#pragma unroll
        for (int r = 0; r < R; r++) {
            T &x = d[pz(o + r * Ns)];
            if constexpr (K == 2)
                x = make_float4(v[0][r].x, v[0][r].y, v[1][r].x, v[1][r].y);
            else
                *reinterpret_cast<float2 *>(&x) = v[0][r];
        }
    }
    __syncthreads();
}

// All passes over lines in the buffer a (written before a barrier), b the
// other one; returns the buffer that holds the result (after a barrier).
template <int K, bool COLS, typename T>
__device__ __forceinline__ T *mixed_transform(const Passes &P, int G, int lg, T *a, T *b, int ls,
                                              const float2 *__restrict__ tw) {
    for (int p = 0; p < P.np; p++) {
#define ARECGB_FFT_PASS(R) \
    case R: mixed_pass<R, K, COLS, T>(P, p, G, lg, a, b, ls, tw); break;
        switch (P.r[p]) {
            ARECGB_FFT_PASS(2) ARECGB_FFT_PASS(3) ARECGB_FFT_PASS(4) ARECGB_FFT_PASS(5)
            ARECGB_FFT_PASS(6) ARECGB_FFT_PASS(7) ARECGB_FFT_PASS(8) ARECGB_FFT_PASS(9)
            ARECGB_FFT_PASS(10) ARECGB_FFT_PASS(16)
        }
#undef ARECGB_FFT_PASS
        T *t = a;
        a = b;
        b = t;
    }
    return a;
}

// Points in and out of shared memory for the run-time lengths, kLoad at a time
// in flight per thread: f(line, point) over G lines of n points.
constexpr int kLoad = 8;
template <bool COLS, typename T, typename LD>
__device__ __forceinline__ void mixed_fill(int n, FastDiv dn, int G, int lg, T *L, int ls, LD &&ld) {
    for (int t0 = threadIdx.x; t0 < G * n; t0 += kLoad * kThreads) {
        T x[kLoad];
#pragma unroll
        for (int e = 0; e < kLoad; e++) {
            const int t = t0 + e * kThreads, line = COLS ? t & (G - 1) : fdiv(t, dn);
            if (t < G * n) x[e] = ld(line, COLS ? t >> lg : t - line * n);
        }
#pragma unroll
        for (int e = 0; e < kLoad; e++) {
            const int t = t0 + e * kThreads, line = COLS ? t & (G - 1) : fdiv(t, dn);
            if (t < G * n) L[line * ls + pz(COLS ? t >> lg : t - line * n)] = x[e];
        }
    }
    __syncthreads();
}
template <bool COLS, typename T, typename ST>
__device__ __forceinline__ void mixed_drain(int n, FastDiv dn, int G, int lg, const T *L, int ls,
                                            ST &&st) {
    for (int t = threadIdx.x; t < G * n; t += kThreads) {
        const int line = COLS ? t & (G - 1) : fdiv(t, dn), i = COLS ? t >> lg : t - line * n;
        st(line, i, L[line * ls + pz(i)]);
    }
}

}  // namespace fft
}  // namespace arecgb
