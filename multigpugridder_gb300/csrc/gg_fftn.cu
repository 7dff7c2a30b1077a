// FFT passes between images and CAS images for sizes M = 2^a 3^b 5^c 7^d up to 400,
// and between a volume and its CAS volume up to 512 (sm_103a).
//
// Each pass transforms tiles of C lines of length M in shared memory (Stockham
// autosort, radices 8, 7, 5, 4, 3, 2, the two buffers swapped between stages) and does
// the stage's index work as it loads and stores: pads, crops, shifts and the
// CAS conversions.  Zero rows are never written, read or transformed, cropped
// ones never stored.
//
//   images -> CAS images: the N image rows in pairs (z = a + i b) along x,
//     split into half spectra; then M/2+1 columns along y, stored as Re+Im and,
//     mirrored, Re-Im.
//   CAS images -> images: the columns back along y, N rows kept; then rows in
//     pairs along x, N pixels kept.
//
//   volume -> CAS volume: rows in pairs along x of the N planes, columns along
//     y, then along z with the CAS values of a voxel and its mirror image: the
//     zero rows and planes of the padded volume are left out of the
//     first two (10.5 M^3 bytes for N = M/2, against about 36).
//   CAS volume -> volume: the same backwards; only what is kept is stored.
//
// Bound: the latency of a tile's load, stages and store at 16 to 32 warps an SM;
// 9 M^2 bytes an image with N = M/2 (1 in, 2 x 2 for the half spectra between
// the passes, 4 out), where the library's batched transforms with a stage
// kernel on either side moved about 29 M^2.  Measured: 300 images at M = 200
// back to real space 115 -> 67 us; 700 images at M = 384 to CAS images 724 -> 562
// us (and the FP16 storage scale without a pass of its own, 177 us).  Tried and
// slower: one buffer with the values held in registers between stages (spills),
// 512 threads, the index divisions as multiplications (67 -> 76 us).
//
// The inverse transform is the forward one with real and imaginary parts
// swapped on the way in and out.  Twiddles: cos and sin of 2 pi k / M in FP64,
// rounded to FP32.
#include <algorithm>
#include <cmath>
#include <vector>

#include "gg_common.cuh"
#include "gg_internal.h"
#include "gg_pair.cuh"

namespace gg {

constexpr int kFnThreads = 256; // 512 measured 10 to 70% slower (barriers between short stages)
constexpr int kFnC = 16;        // lines a tile: rows of half spectra move in 128 bytes
constexpr int kFnStages = 12;

struct FnPlan {
    int M, stages, radix[kFnStages];
};

__device__ __forceinline__ float2 c_add(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 c_sub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 c_mul(float2 a, float2 b) { return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
__device__ __forceinline__ float2 c_mi(float2 a) { return make_float2(a.y, -a.x); } // times -i

// Forward DFTs of 2, 4 and 8 values in place, natural order.
__device__ __forceinline__ void dft2(float2 &a, float2 &b)
{
    const float2 t = a;
    a = c_add(t, b);
    b = c_sub(t, b);
}
__device__ __forceinline__ void dft4(float2 &a, float2 &b, float2 &c, float2 &d)
{
    const float2 s = c_add(a, c), t = c_sub(a, c), u = c_add(b, d), v = c_mi(c_sub(b, d));
    a = c_add(s, u);
    b = c_add(t, v);
    c = c_sub(s, u);
    d = c_sub(t, v);
}
template <int R> __device__ __forceinline__ void dft(float2 (&x)[R])
{
    if constexpr (R == 2) {
        dft2(x[0], x[1]);
    } else if constexpr (R == 4) {
        dft4(x[0], x[1], x[2], x[3]);
    } else if constexpr (R == 8) {
        // even and odd halves, the odd one turned by W_8^k
        const float h = 0.70710678118654752f;
        dft4(x[0], x[2], x[4], x[6]);
        dft4(x[1], x[3], x[5], x[7]);
        const float2 o1 = make_float2(h * (x[3].x + x[3].y), h * (x[3].y - x[3].x)), o2 = c_mi(x[5]),
                     o3 = make_float2(h * (x[7].y - x[7].x), -h * (x[7].x + x[7].y));
        const float2 e0 = x[0], e1 = x[2], e2 = x[4], e3 = x[6], o0 = x[1];
        x[0] = c_add(e0, o0);
        x[1] = c_add(e1, o1);
        x[2] = c_add(e2, o2);
        x[3] = c_add(e3, o3);
        x[4] = c_sub(e0, o0);
        x[5] = c_sub(e1, o1);
        x[6] = c_sub(e2, o2);
        x[7] = c_sub(e3, o3);
    } else {
        // odd R: pairs t and R - t, whose sums and differences meet cos and sin
        constexpr int Q = (R - 1) / 2;
        constexpr float c3[2] = {1.0f, -0.5f}, s3[2] = {0.0f, 0.86602540378443865f};
        constexpr float c5[3] = {1.0f, 0.30901699437494742f, -0.80901699437494742f},
                        s5[3] = {0.0f, 0.95105651629515357f, 0.58778525229247313f};
        constexpr float c7[4] = {1.0f, 0.62348980185873353f, -0.22252093395631440f, -0.90096886790241913f},
                        s7[4] = {0.0f, 0.78183148246802981f, 0.97492791218182361f, 0.43388373911755812f};
        float2 p[Q + 1], m[Q + 1];
#pragma unroll
        for (int t = 1; t <= Q; t++) {
            p[t] = c_add(x[t], x[R - t]);
            m[t] = c_sub(x[t], x[R - t]);
        }
        const float2 x0 = x[0];
        float2 sum = x0;
#pragma unroll
        for (int t = 1; t <= Q; t++) sum = c_add(sum, p[t]);
        x[0] = sum;
#pragma unroll
        for (int k = 1; k <= Q; k++) {
            float2 a = x0, b = make_float2(0.0f, 0.0f);
#pragma unroll
            for (int t = 1; t <= Q; t++) {
                const int q = k * t % R, i = q <= Q ? q : R - q;
                const float c = R == 3 ? c3[i < 2 ? i : 0] : R == 5 ? c5[i < 3 ? i : 0] : c7[i < 4 ? i : 0];
                const float s = (q <= Q ? 1.0f : -1.0f) * (R == 3 ? s3[i < 2 ? i : 0] : R == 5 ? s5[i < 3 ? i : 0] : s7[i < 4 ? i : 0]);
                a.x = fmaf(c, p[t].x, a.x);
                a.y = fmaf(c, p[t].y, a.y);
                b.x = fmaf(s, m[t].x, b.x);
                b.y = fmaf(s, m[t].y, b.y);
            }
            // a - i b and its mirror
            x[k] = make_float2(a.x + b.y, a.y - b.x);
            x[R - k] = make_float2(a.x - b.y, a.y + b.x);
        }
    }
}

// One Stockham stage over C lines (line index fastest, rows C + 1 apart): Ns
// points are transformed already.
template <int R, int C>
__device__ __forceinline__ void fn_stage(const float2 *__restrict__ in, float2 *__restrict__ out,
                                         const float2 *__restrict__ tw, int M, int Ns)
{
    constexpr int CP = C + 1;
    const int per = M / R, step = per / Ns;
    for (int e = threadIdx.x; e < per * C; e += kFnThreads) {
        const int c = e % C, j = e / C, k = j % Ns;
        float2 x[R];
#pragma unroll
        for (int t = 0; t < R; t++) x[t] = in[(j + t * per) * CP + c];
        if (Ns > 1) {
#pragma unroll
            for (int t = 1; t < R; t++) x[t] = c_mul(x[t], tw[k * t * step]);
        }
        dft<R>(x);
        const int o = (j - k) * R + k;
#pragma unroll
        for (int t = 0; t < R; t++) out[(o + t * Ns) * CP + c] = x[t];
    }
}

// A pass: load a tile of C lines, transform, store.  blockIdx.x: tile;
// blockIdx.y walks the images (slices).
template <int C, class Load, class Store>
__global__ void __launch_bounds__(kFnThreads)
fn_pass_kernel(const FnPlan p, const float2 *__restrict__ d_tw, int n, const Load load, const Store store)
{
    extern __shared__ __align__(16) float2 fn_tile[];
    const int M = p.M;
    float2 *const tw = fn_tile, *a = tw + M, *b = a + M * (C + 1);
    for (int t = threadIdx.x; t < M; t += kFnThreads) tw[t] = __ldg(d_tw + t);
    for (int s = blockIdx.y; s < n; s += gridDim.y) {
        load(a, s, blockIdx.x);
        __syncthreads();
        int Ns = 1;
        for (int q = 0; q < p.stages; q++) {
            const int R = p.radix[q];
            if (R == 8) fn_stage<8, C>(a, b, tw, M, Ns);
            else if (R == 4) fn_stage<4, C>(a, b, tw, M, Ns);
            else if (R == 2) fn_stage<2, C>(a, b, tw, M, Ns);
            else if (R == 3) fn_stage<3, C>(a, b, tw, M, Ns);
            else if (R == 5) fn_stage<5, C>(a, b, tw, M, Ns);
            else fn_stage<7, C>(a, b, tw, M, Ns);
            __syncthreads();
            float2 *const x = a;
            a = b;
            b = x;
            Ns *= R;
        }
        store(a, s, blockIdx.x);
        __syncthreads();
    }
}

__device__ __forceinline__ int fn_shift(int q, int M) { return q + M / 2 >= M ? q + M / 2 - M : q + M / 2; }
// Where element o of the centred N-line lies on the shifted M-line.
__device__ __forceinline__ int fn_wrap(int o, int N, int M) { return o >= N / 2 ? o - N / 2 : o + M - N / 2; }

// Zeroes the rows of the M-line that the wrapped N-line leaves free.
template <int C> __device__ __forceinline__ void fn_zero_gap(float2 *a, int N, int M)
{
    constexpr int CP = C + 1;
    for (int e = threadIdx.x; e < (M - N) * CP; e += kFnThreads) a[(N / 2) * CP + e] = make_float2(0.0f, 0.0f);
}

// ---- rows of real data, two to a line (2c -> real, 2c + 1 -> imaginary) --------

// N real rows of N (slice s at src + s N^2) -> lines along x, wrapped and padded.
template <int C> struct LoadRealRows {
    const float *src;
    int N, M;
    __device__ void operator()(float2 *a, int s, int tile) const
    {
        constexpr int CP = C + 1;
        const float *im = src + (size_t)s * N * N;
        fn_zero_gap<C>(a, N, M);
        float *f = reinterpret_cast<float *>(a);
        for (int r = threadIdx.x >> 5; r < 2 * C; r += kFnThreads / 32) {
            const int row = tile * 2 * C + r;
#pragma unroll 4
            for (int o = threadIdx.x & 31; o < N; o += 32)
                f[2 * (fn_wrap(o, N, M) * CP + (r >> 1)) + (r & 1)] = row < N ? __ldg(im + (size_t)row * N + o) : 0.0f;
        }
    }
};

// The same of a volume (slice s: plane s) times the precomp factors' product.
template <int C> struct LoadVolumeRows {
    const float *src;
    const float2 *pc;
    int N, M;
    __device__ void operator()(float2 *a, int s, int tile) const
    {
        constexpr int CP = C + 1;
        const int b = M / 2 - N / 2;
        const float *im = src + (size_t)s * N * N;
        fn_zero_gap<C>(a, N, M);
        float *f = reinterpret_cast<float *>(a);
        for (int r = threadIdx.x >> 5; r < 2 * C; r += kFnThreads / 32) {
            const int row = tile * 2 * C + r;
            const FF jk = ff_mul(ff_at(pc, min(row, N - 1) + b), ff_at(pc, s + b));
#pragma unroll 4
            for (int o = threadIdx.x & 31; o < N; o += 32)
                f[2 * (fn_wrap(o, N, M) * CP + (r >> 1)) + (r & 1)] =
                    row < N ? __ldg(im + (size_t)row * N + o) * ff_mul(ff_at(pc, o + b), jk).h : 0.0f;
        }
    }
};

// Lines of row pairs -> half spectra, N rows of H a slice.
template <int C> struct StoreHalfRows {
    float2 *dst;
    int N, M;
    __device__ void operator()(const float2 *a, int s, int tile) const
    {
        constexpr int CP = C + 1;
        const int H = M / 2 + 1;
        float2 *g = dst + (size_t)s * N * H;
        for (int c = threadIdx.x >> 5; c < C; c += kFnThreads / 32) {
            const int row = 2 * (tile * C + c);
            if (row >= N) continue;
            for (int u = threadIdx.x & 31; u < H; u += 32) {
                const float2 z = a[u * CP + c], y = a[(u ? M - u : 0) * CP + c];
                // A = (Z(u) + conj Z(-u)) / 2, B = (Z(u) - conj Z(-u)) / 2i
                g[(size_t)row * H + u] = make_float2(0.5f * (z.x + y.x), 0.5f * (z.y - y.y));
                if (row + 1 < N) g[(size_t)(row + 1) * H + u] = make_float2(0.5f * (z.y + y.y), 0.5f * (y.x - z.x));
            }
        }
    }
};

// Half spectra of real rows (N a slice) -> lines of row pairs, inverse (swapped).
template <int C> struct LoadHalfRows {
    const float2 *src;
    int N, M;
    __device__ void operator()(float2 *a, int s, int tile) const
    {
        constexpr int CP = C + 1;
        const int H = M / 2 + 1;
        const float2 *g = src + (size_t)s * N * H;
        for (int c = threadIdx.x >> 5; c < C; c += kFnThreads / 32) {
            const int row = 2 * (tile * C + c);
#pragma unroll 2
            for (int u = threadIdx.x & 31; u < H; u += 32) {
                const float2 zero = make_float2(0.0f, 0.0f);
                const float2 p = row < N ? __ldg(g + (size_t)row * H + u) : zero;
                const float2 q = row + 1 < N ? __ldg(g + (size_t)(row + 1) * H + u) : zero;
                // Z(u) = P + i Q, Z(-u) = conj P + i conj Q; real at u = 0 and M/2
                if (u == 0 || u == M / 2) {
                    a[u * CP + c] = make_float2(q.x, p.x);
                } else {
                    a[u * CP + c] = make_float2(p.y + q.x, p.x - q.y);
                    a[(M - u) * CP + c] = make_float2(q.x - p.y, p.x + q.y);
                }
            }
        }
    }
};

// Lines of row pairs -> N cropped pixels of N rows a slice, times `scale`.
template <int C> struct StoreRealRows {
    float *dst;
    int N, M;
    float scale;
    __device__ void operator()(const float2 *a, int s, int tile) const
    {
        constexpr int CP = C + 1;
        const float *f = reinterpret_cast<const float *>(a);
        float *im = dst + (size_t)s * N * N;
        for (int r = threadIdx.x >> 5; r < 2 * C; r += kFnThreads / 32) {
            const int row = tile * 2 * C + r;
            if (row >= N) break;
            for (int o = threadIdx.x & 31; o < N; o += 32) // swapped back: the even row is the imaginary part
                im[(size_t)row * N + o] = f[2 * (fn_wrap(o, N, M) * CP + (r >> 1)) + 1 - (r & 1)] * scale;
        }
    }
};

// ---- columns of half spectra ------------------------------------------------------

// N rows of half spectra a slice -> columns u0 .. u0 + C - 1, wrapped and padded.
template <int C> struct LoadPaddedCols {
    const float2 *src;
    int N, M;
    __device__ void operator()(float2 *a, int s, int tile) const
    {
        constexpr int CP = C + 1;
        const int H = M / 2 + 1, c = threadIdx.x % C, u = tile * C + c;
        const float2 *g = src + (size_t)s * N * H + u;
        fn_zero_gap<C>(a, N, M);
#pragma unroll 4
        for (int r = threadIdx.x / C; r < N; r += kFnThreads / C)
            a[fn_wrap(r, N, M) * CP + c] = u < H ? __ldg(g + (size_t)r * H) : make_float2(0.0f, 0.0f);
    }
};

// Columns of an image's spectrum -> its CAS image (Re+Im, and Re-Im mirrored).
// ADJ: the adjoint form (first row and column zero, times post).
// top (optional): the largest magnitude's bits (atomicMax).
template <int C, bool ADJ> struct StoreCasCols {
    float *dst;
    int M;
    float post;
    unsigned *top;
    __device__ void operator()(const float2 *a, int s, int tile) const
    {
        constexpr int CP = C + 1;
        const int c = threadIdx.x % C, u = tile * C + c;
        float *cas = dst + (size_t)s * M * M;
        float most = 0.0f;
        if (u <= M / 2) {
            const int i = fn_shift(u, M), im = M / 2 - u; // of u and of M - u
            const bool mirror = u != 0 && u != M / 2;
            for (int v = threadIdx.x / C; v < M; v += kFnThreads / C) {
                const int j = fn_shift(v, M), jm = fn_shift(v ? M - v : 0, M);
                const float2 z = a[v * CP + c];
                float d = z.x + z.y, e = z.x - z.y;
                if (ADJ) {
                    d = (i == 0 || j == 0) ? 0.0f : d * post;
                    e = (im == 0 || jm == 0) ? 0.0f : e * post;
                }
                cas[(size_t)j * M + i] = d;
                if (mirror) cas[(size_t)jm * M + im] = e;
                most = fmaxf(most, fmaxf(fabsf(d), fabsf(e)));
            }
        }
        if (top) {
            const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(most));
            if ((threadIdx.x & 31) == 0) atomicMax(top, m);
        }
    }
};

// Columns of a plane -> M rows of H a plane.
template <int C> struct StoreSpecCols {
    float2 *dst;
    int M;
    __device__ void operator()(const float2 *a, int s, int tile) const
    {
        constexpr int CP = C + 1;
        const int H = M / 2 + 1, c = threadIdx.x % C, u = tile * C + c;
        if (u >= H) return;
        float2 *g = dst + (size_t)s * M * H + u;
        for (int v = threadIdx.x / C; v < M; v += kFnThreads / C) g[(size_t)v * H] = a[v * CP + c];
    }
};

// N planes of M rows of H -> columns along z of row s, wrapped and padded.
template <int C> struct LoadDepthCols {
    const float2 *src;
    int N, M;
    __device__ void operator()(float2 *a, int s, int tile) const
    {
        constexpr int CP = C + 1;
        const int H = M / 2 + 1, c = threadIdx.x % C, u = tile * C + c;
        const float2 *g = src + (size_t)s * H + u;
        fn_zero_gap<C>(a, N, M);
#pragma unroll 4
        for (int r = threadIdx.x / C; r < N; r += kFnThreads / C)
            a[fn_wrap(r, N, M) * CP + c] = u < H ? __ldg(g + (size_t)r * M * H) : make_float2(0.0f, 0.0f);
    }
};

// Columns along z of row v = s of the half spectrum -> the CAS volume: Re+Im,
// and Re-Im at the mirror image through the centre; the rows' borders zero.
template <int C> struct StoreCasVolume {
    float *dst;
    int M, V;
    __device__ void operator()(const float2 *a, int s, int tile) const
    {
        constexpr int CP = C + 1;
        const int c = threadIdx.x % C, u = tile * C + c, pad = V / 2 - M / 2;
        const int j = fn_shift(s, M), jm = fn_shift(s ? M - s : 0, M);
        const size_t VV = (size_t)V * V;
        float *row = dst + pad * VV + (size_t)(j + pad) * V + pad;  // of plane pad
        float *rowm = dst + pad * VV + (size_t)(jm + pad) * V + pad;
        if (u <= M / 2) {
            const int i = fn_shift(u, M), im = M / 2 - u; // of u and of M - u
            const bool mirror = u != 0 && u != M / 2;
            for (int w = threadIdx.x / C; w < M; w += kFnThreads / C) {
                const float2 z = a[w * CP + c];
                row[fn_shift(w, M) * VV + i] = z.x + z.y;
                if (mirror) rowm[fn_shift(w ? M - w : 0, M) * VV + im] = z.x - z.y;
            }
        }
        if (tile == 0) {
            const int edge = V - M; // columns outside a row's M
            for (int e = threadIdx.x; e < M * edge; e += kFnThreads) {
                const int k = e / edge, x = e - k * edge;
                row[k * VV + (x < pad ? x - pad : x - pad + M)] = 0.0f;
            }
        }
    }
};

// M planes of M rows of H -> columns along z of row s, inverse (swapped).
template <int C> struct LoadSpecDepth {
    const float2 *src;
    int M;
    __device__ void operator()(float2 *a, int s, int tile) const
    {
        constexpr int CP = C + 1;
        const int H = M / 2 + 1, c = threadIdx.x % C, u = tile * C + c;
        const float2 *g = src + (size_t)s * H + u;
#pragma unroll 4
        for (int w = threadIdx.x / C; w < M; w += kFnThreads / C) {
            const float2 z = u < H ? __ldg(g + (size_t)w * M * H) : make_float2(0.0f, 0.0f);
            a[w * CP + c] = make_float2(z.y, z.x);
        }
    }
};

// The same from the CAS volume itself (FromCAS over the inner M^3).
template <int C> struct LoadCasDepth {
    const float *src;
    int M, V;
    __device__ void operator()(float2 *a, int s, int tile) const
    {
        constexpr int CP = C + 1;
        const int c = threadIdx.x % C, u = tile * C + c, pad = V / 2 - M / 2, j = fn_shift(s, M);
        const size_t VV = (size_t)V * V;
        const bool live = j != 0 && u < M / 2; // u = M/2 is column 0: zero
        const float *g = src + pad * VV + (size_t)(j + pad) * V + pad + M / 2 + u;
        const float *gm = src + pad * VV + (size_t)(M - j + pad) * V + pad + M / 2 - u;
#pragma unroll 4
        for (int w = threadIdx.x / C; w < M; w += kFnThreads / C) {
            const int k = fn_shift(w, M);
            const bool on = live && k != 0;
            const float x = on ? __ldg(g + k * VV) : 0.0f, y = on ? __ldg(gm + (M - k) * VV) : 0.0f;
            a[w * CP + c] = make_float2(0.5f * (x - y), 0.5f * (x + y));
        }
    }
};

// Inverse columns along z of row s -> N cropped planes of M rows of H.
template <int C> struct StoreCroppedDepth {
    float2 *dst;
    int N, M;
    __device__ void operator()(const float2 *a, int s, int tile) const
    {
        constexpr int CP = C + 1;
        const int H = M / 2 + 1, c = threadIdx.x % C, u = tile * C + c;
        if (u >= H) return;
        float2 *g = dst + (size_t)s * H + u;
        for (int r = threadIdx.x / C; r < N; r += kFnThreads / C) {
            const float2 z = a[fn_wrap(r, N, M) * CP + c];
            g[(size_t)r * M * H] = make_float2(z.y, z.x);
        }
    }
};

// M rows of H a plane -> columns along y, inverse (swapped).
template <int C> struct LoadSpecCols {
    const float2 *src;
    int M;
    __device__ void operator()(float2 *a, int s, int tile) const
    {
        constexpr int CP = C + 1;
        const int H = M / 2 + 1, c = threadIdx.x % C, u = tile * C + c;
        const float2 *g = src + (size_t)s * M * H + u;
#pragma unroll 4
        for (int v = threadIdx.x / C; v < M; v += kFnThreads / C) {
            const float2 z = u < H ? __ldg(g + (size_t)v * H) : make_float2(0.0f, 0.0f);
            a[v * CP + c] = make_float2(z.y, z.x);
        }
    }
};

// Lines of row pairs -> N cropped voxels of N rows of plane s, times the precomp
// factors' product and `inv`, rounded once.
template <int C> struct StoreVolumeRows {
    float *dst;
    const float2 *pc;
    int N, M;
    FF inv;
    __device__ void operator()(const float2 *a, int s, int tile) const
    {
        constexpr int CP = C + 1;
        const int b = M / 2 - N / 2;
        const float *f = reinterpret_cast<const float *>(a);
        float *im = dst + (size_t)s * N * N;
        for (int r = threadIdx.x >> 5; r < 2 * C; r += kFnThreads / 32) {
            const int row = tile * 2 * C + r;
            if (row >= N) break;
            const FF jk = ff_mul(inv, ff_mul(ff_at(pc, row + b), ff_at(pc, s + b)));
            for (int o = threadIdx.x & 31; o < N; o += 32)
                im[(size_t)row * N + o] =
                    ff_scale(f[2 * (fn_wrap(o, N, M) * CP + (r >> 1)) + 1 - (r & 1)], ff_mul(ff_at(pc, o + b), jk));
        }
    }
};

// Zeroes the rows of the CAS volume that lie outside the spectrum.
__global__ void __launch_bounds__(256) zero_border_rows_kernel(float *__restrict__ cas, int M, int V)
{
    const int pad = V / 2 - M / 2, warp = threadIdx.x >> 5;
    const int slab = (V - M) * V, rows = slab + M * (V - M); // whole planes, then rows of the others
    for (int r = blockIdx.x * 8 + warp; r < rows; r += gridDim.x * 8) {
        int k, j;
        if (r < slab) {
            k = r / V;
            j = r - k * V;
            if (k >= pad) k += M;
        } else {
            const int t = r - slab;
            k = t / (V - M);
            j = t - k * (V - M);
            k += pad;
            if (j >= pad) j += M;
        }
        float *row = cas + ((size_t)k * V + j) * V;
        for (int c = threadIdx.x & 31; c < V; c += 32) row[c] = 0.0f;
    }
}

// A CAS image -> columns of its Hermitian spectrum (FromCAS), inverse (swapped).
template <int C> struct LoadCasCols {
    const float *src;
    int M;
    __device__ void operator()(float2 *a, int s, int tile) const
    {
        constexpr int CP = C + 1;
        const int c = threadIdx.x % C, u = tile * C + c;
        const float *cas = src + (size_t)s * M * M;
        const bool live = u < M / 2; // u = M/2 is column 0: zero
#pragma unroll 4
        for (int v = threadIdx.x / C; v < M; v += kFnThreads / C) {
            const int j = fn_shift(v, M);
            const bool on = live && j != 0;
            const float x = on ? __ldg(cas + (size_t)j * M + M / 2 + u) : 0.0f;
            const float y = on ? __ldg(cas + (size_t)(M - j) * M + M / 2 - u) : 0.0f;
            a[v * CP + c] = make_float2(0.5f * (x - y), 0.5f * (x + y));
        }
    }
};

// Inverse columns -> N cropped rows of half spectra a slice.
template <int C> struct StoreCroppedCols {
    float2 *dst;
    int N, M;
    __device__ void operator()(const float2 *a, int s, int tile) const
    {
        constexpr int CP = C + 1;
        const int H = M / 2 + 1, c = threadIdx.x % C, u = tile * C + c;
        if (u >= H) return;
        float2 *g = dst + (size_t)s * N * H + u;
        for (int r = threadIdx.x / C; r < N; r += kFnThreads / C) {
            const float2 z = a[fn_wrap(r, N, M) * CP + c];
            g[(size_t)r * H] = make_float2(z.y, z.x);
        }
    }
};

// ---- host side -----------------------------------------------------------------

// False if M has a prime factor above 7 or is too long.
static bool fn_plan(int M, FnPlan &p)
{
    p.M = M;
    p.stages = 0;
    if (M < 4 || (M & 1)) return false;
    int m = M;
    for (int r : {7, 5, 3, 8, 4, 2})
        while (m % r == 0 && p.stages < kFnStages) {
            p.radix[p.stages++] = r;
            m /= r;
        }
    return m == 1;
}

static size_t fn_smem(int M, int C) { return ((size_t)M + 2 * (size_t)M * (C + 1)) * sizeof(float2); }

// Longer lines leave room for one tile of 16 an SM or tiles of 8, and either way
// the passes lose to the library (M = 512: 705 us against 694 for 512 images).
constexpr int kFnMaxM = 400;

bool fftn_ok(int N, int M)
{
    FnPlan p;
    return N > 0 && N <= M && (N & 1) == 0 && M <= kFnMaxM && fn_plan(M, p);
}

// A volume's three passes against the library's 3-D transform and its two stage
// kernels (setVolume and 16 projections, us): M = 64: 41 (39), 96: 61 (63), 192:
// 127 (142), 200: 139 (177), 256: 215 (235), 320: 354 (502), 384: 597 (789), 400: 695
// (1166), 448: 960 (1450), 500: 1396 (1722).  Above 400 in tiles of 8 lines,
// which leave room for two an SM.
constexpr int kFnMinVolM = 96, kFnMaxVolM = 512;

bool fftn_volume_ok(int N, int M)
{
    FnPlan p;
    return N > 0 && N <= M && (N & 1) == 0 && M >= kFnMinVolM && M <= kFnMaxVolM && fn_plan(M, p);
}

// Back: the z pass reads the CAS volume (or the divided one's spectrum) in full
// and there is less to prune.  16 images back and the volume, us: M = 96: 94
// (99), 200: 177 (215), 384: 945 (987), 400: 1065 (1385), 420: 1133 (1327); but
// 256: 294 (292), 512: 1976 (1850), where the library has powers of two.
bool fftn_volume_back_ok(int N, int M) { return fftn_volume_ok(N, M) && (M & (M - 1)) != 0; }

void fftn_twiddles(int M, float2 *out)
{
    const double pi = 3.14159265358979323846;
    for (int k = 0; k < M; k++) {
        // from the first octant's angles, so that quarter and half turns are exact
        const int q = (int)((long long)k * 8 / M);
        int r = k;
        double sc = 1.0, ss = 1.0;
        if (q >= 4) { // theta - pi
            r -= M / 2;
            sc = ss = -1.0;
        }
        double c, s;
        if (8 * r <= M) {
            c = std::cos(2 * pi * r / M);
            s = std::sin(2 * pi * r / M);
        } else if (8 * r <= 3 * M) {
            const double t = pi / 2 - 2 * pi * r / M;
            c = std::sin(t);
            s = std::cos(t);
        } else {
            const double t = pi - 2 * pi * r / M;
            c = -std::cos(t);
            s = std::sin(t);
        }
        out[k] = make_float2((float)(sc * c), (float)(-ss * s)); // e^(-i theta)
    }
}

template <int C, class Load, class Store>
static cudaError_t fn_launch(const FnPlan &p, const float2 *d_tw, int tiles, int n, const Load &load, const Store &store,
                             cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    const size_t smem = fn_smem(p.M, C);
    auto kern = fn_pass_kernel<C, Load, Store>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    kern<<<dim3((unsigned)tiles, (unsigned)std::min(n, 65535)), kFnThreads, smem, s>>>(p, d_tw, n, load, store);
    count_launches(1);
    return cudaGetLastError();
}

template <int C, bool ADJ>
static cudaError_t images_to_cas_t(const FnPlan &p, const float2 *d_tw, const float *d_img, int N, int n, float *d_cas,
                                   float post, float2 *d_half, unsigned *top, cudaStream_t s)
{
    const int M = p.M, H = M / 2 + 1;
    cudaError_t e = fn_launch<C>(p, d_tw, (N + 2 * C - 1) / (2 * C), n, LoadRealRows<C>{d_img, N, M},
                                 StoreHalfRows<C>{d_half, N, M}, s);
    if (e != cudaSuccess) return e;
    return fn_launch<C>(p, d_tw, (H + C - 1) / C, n, LoadPaddedCols<C>{d_half, N, M},
                        StoreCasCols<C, ADJ>{d_cas, M, post, top}, s);
}

cudaError_t launch_images_to_cas_passes(const float *d_img, int N, int M, int n, float *d_cas, bool adjoint,
                                        const float2 *d_tw, float2 *d_half, unsigned *top, cudaStream_t s)
{
    FnPlan p;
    if (!fftn_ok(N, M) || !fn_plan(M, p)) return cudaErrorInvalidValue;
    const float post = 1.0f / ((float)M * (float)M);
    if (adjoint) return images_to_cas_t<kFnC, true>(p, d_tw, d_img, N, n, d_cas, post, d_half, top, s);
    return images_to_cas_t<kFnC, false>(p, d_tw, d_img, N, n, d_cas, 1.0f, d_half, top, s);
}

cudaError_t launch_cas_to_images_passes(const float *d_cas, int M, int N, int n, float *d_img, const float2 *d_tw,
                                        float2 *d_half, cudaStream_t s)
{
    FnPlan p;
    if (!fftn_ok(N, M) || !fn_plan(M, p)) return cudaErrorInvalidValue;
    constexpr int C = kFnC;
    cudaError_t e = fn_launch<C>(p, d_tw, (M / 2 + C) / C, n, LoadCasCols<C>{d_cas, M}, StoreCroppedCols<C>{d_half, N, M}, s);
    if (e != cudaSuccess) return e;
    return fn_launch<C>(p, d_tw, (N + 2 * C - 1) / (2 * C), n, LoadHalfRows<C>{d_half, N, M},
                        StoreRealRows<C>{d_img, N, M, 1.0f / ((float)M * (float)M)}, s);
}

template <int C>
static cudaError_t volume_to_cas_t(const FnPlan &p, const float2 *d_tw, const float *d_vol, int N, int V, const float2 *d_pc,
                                   float *d_cas, float2 *d_half, float2 *d_planes, cudaStream_t s)
{
    const int M = p.M, H = M / 2 + 1, cols = (H + C - 1) / C;
    cudaError_t e = fn_launch<C>(p, d_tw, (N + 2 * C - 1) / (2 * C), N, LoadVolumeRows<C>{d_vol, d_pc, N, M},
                                 StoreHalfRows<C>{d_half, N, M}, s);
    if (e != cudaSuccess) return e;
    e = fn_launch<C>(p, d_tw, cols, N, LoadPaddedCols<C>{d_half, N, M}, StoreSpecCols<C>{d_planes, M}, s);
    if (e != cudaSuccess) return e;
    e = fn_launch<C>(p, d_tw, cols, M, LoadDepthCols<C>{d_planes, N, M}, StoreCasVolume<C>{d_cas, M, V}, s);
    if (e != cudaSuccess || V == M) return e;
    zero_border_rows_kernel<<<(unsigned)(((V - M) * (V + M) + 7) / 8), 256, 0, s>>>(d_cas, M, V);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_volume_to_cas_passes(const float *d_vol, int N, int M, int V, const float2 *d_pc, float *d_cas,
                                        const float2 *d_tw, float2 *d_half, float2 *d_planes, cudaStream_t s)
{
    FnPlan p;
    if (!fftn_volume_ok(N, M) || !fn_plan(M, p) || V < M) return cudaErrorInvalidValue;
    if (M <= kFnMaxM) return volume_to_cas_t<kFnC>(p, d_tw, d_vol, N, V, d_pc, d_cas, d_half, d_planes, s);
    return volume_to_cas_t<kFnC / 2>(p, d_tw, d_vol, N, V, d_pc, d_cas, d_half, d_planes, s);
}

template <int C>
static cudaError_t cas_to_volume_t(const FnPlan &p, const float2 *d_tw, const float *d_cas, const float2 *d_spec, int N, int V,
                                   const float2 *d_pc, float *d_vol, float2 *d_half, float2 *d_planes, cudaStream_t s)
{
    const int M = p.M, H = M / 2 + 1, cols = (H + C - 1) / C;
    const double m3 = 1.0 / ((double)M * M * M);
    const FF inv{(float)m3, (float)(m3 - (double)(float)m3)};
    const StoreCroppedDepth<C> planes{d_planes, N, M};
    cudaError_t e = d_spec ? fn_launch<C>(p, d_tw, cols, M, LoadSpecDepth<C>{d_spec, M}, planes, s)
                           : fn_launch<C>(p, d_tw, cols, M, LoadCasDepth<C>{d_cas, M, V}, planes, s);
    if (e != cudaSuccess) return e;
    e = fn_launch<C>(p, d_tw, cols, N, LoadSpecCols<C>{d_planes, M}, StoreCroppedCols<C>{d_half, N, M}, s);
    if (e != cudaSuccess) return e;
    return fn_launch<C>(p, d_tw, (N + 2 * C - 1) / (2 * C), N, LoadHalfRows<C>{d_half, N, M},
                        StoreVolumeRows<C>{d_vol, d_pc, N, M, inv}, s);
}

cudaError_t launch_cas_to_volume_passes(const float *d_cas, const float2 *d_spec, int N, int M, int V, const float2 *d_pc,
                                        float *d_vol, const float2 *d_tw, float2 *d_half, float2 *d_planes, cudaStream_t s)
{
    FnPlan p;
    if (!fftn_volume_back_ok(N, M) || !fn_plan(M, p) || V < M) return cudaErrorInvalidValue;
    if (M <= kFnMaxM) return cas_to_volume_t<kFnC>(p, d_tw, d_cas, d_spec, N, V, d_pc, d_vol, d_half, d_planes, s);
    return cas_to_volume_t<kFnC / 2>(p, d_tw, d_cas, d_spec, N, V, d_pc, d_vol, d_half, d_planes, s);
}

} // namespace gg
