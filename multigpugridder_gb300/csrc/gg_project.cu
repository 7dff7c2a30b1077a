// Kaiser-Bessel Fourier-slice projection kernels for GB300 (sm_103a).
//
//   forward projection   CAS volume -> CAS images (pixel-driven gather)
//   back projection      CAS images -> CAS volume, reference window rule
//
// Conventions follow the reference kernels (src/Projection/gpuForwardProject.cu,
// src/Projection/gpuBackProject.cu): x fastest, CAS-volume centre V/2, image
// centre M/2, nearest-index lookup into the KB table, int mask radius.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "gg_internal.h"
#include "gg_project.cuh"

namespace gg {

// ---------------------------------------------------------------------------
// Shared pieces
// ---------------------------------------------------------------------------

// A voxel's image-frame coordinate (gpuBackProject.cu:62-64),
// fma(a2, n2, fma(a0, n0, a1*n1)); every grouping of the three products gave
// the same results against the reference kernel, this one is fixed here.
__device__ __forceinline__ float voxel_proj(float a0, float a1, float a2, float n0, float n1, float n2)
{
    return __fmaf_rn(a2, n2, __fmaf_rn(a0, n0, __fmul_rn(a1, n1)));
}

// An attribute of the current device, cached per device ordinal (a process
// may drive GPUs of different kinds).  cache[] starts at zero; a racing
// first read stores the same value twice.
constexpr int kAttrCacheDevices = 64;

static int device_attr(cudaDeviceAttr attr, std::atomic<int> *cache, int fallback)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return fallback;
    }
    const bool cached = dev >= 0 && dev < kAttrCacheDevices;
    if (cached) {
        const int v = cache[dev].load(std::memory_order_relaxed);
        if (v > 0) return v;
    }
    int v = 0;
    if (cudaDeviceGetAttribute(&v, attr, dev) != cudaSuccess || v <= 0) {
        cudaGetLastError();
        return fallback;
    }
    if (cached) cache[dev].store(v, std::memory_order_relaxed);
    return v;
}

static int num_sms()
{
    static std::atomic<int> cache[kAttrCacheDevices];
    return device_attr(cudaDevAttrMultiProcessorCount, cache, 1);
}

// ---------------------------------------------------------------------------
// Forward projection
// ---------------------------------------------------------------------------
// The gridder's own volumes take fp_tile_kernel (gg_fp_tile.cu).  fp_kernel
// reads the taps from global memory: for a caller's dense volume, which TMA
// cannot address (its rows are not multiples of 16 bytes), and for KB tables
// whose edges are not zero.
//
// One CTA = a 16x16 pixel tile of one direction; persistent grid-stride loop
// over (direction, tile) items, direction-major so that the CTAs resident at
// any time read the same few slabs of the volume.  Warps cover 8x4 pixel
// blocks, which keeps a warp's tap addresses compact in the volume.
//
// With a KB table whose first and last entries are zero (getKernelFiltTable
// forces both, getKernelFiltTable.m:12-13), only the 4 taps floor(f)-1 ..
// floor(f)+2 per axis can carry weight: of the reference's 5 taps around
// round(f) (gpuForwardProject.cu:63-98) the fifth always has |r| >= 2, is
// clamped to the table edge and weighs exactly zero.  TAPS = 5 keeps the
// reference's full window for tables without zero edges.
//
// The volume may be stored with a row pitch P >= V (plane pitch P*V; the
// reference's dense layout is P = V).
constexpr int kFpTile = 16;
constexpr int kFpThreads = 256;

template <typename TV, int TAPS>
__global__ void __launch_bounds__(kFpThreads)
fp_kernel(const TV *__restrict__ vol, int V, int P, float *__restrict__ img, int M,
          const float *__restrict__ axes, int maskR, const float *__restrict__ ker, int kerSize,
          float kerHW, int tilesX, long long nItems, const float *__restrict__ d_scale)
{
    const float outScale = d_scale ? *d_scale : 1.0f;
    __shared__ float sker[kMaxKerSize];
    load_table(sker, ker, kerSize);
    __syncthreads();

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // 8x4 warp tiles (2 x 4 per CTA)
    const int lx = (lane & 7) | ((warp & 1) << 3), ly = (lane >> 3) | ((warp >> 1) << 2);
    const int ic = M / 2, vc = V / 2;
    const float kerCenter = ((float)kerSize - 1) / 2;
    const float kerScale = kerCenter / kerHW;
    const float kerCenterHalf = kerCenter + 0.5f;
    const float convW = (float)(int)roundf(kerHW);
    const long long R2 = (long long)maskR * maskR;
    const int tilesPerImg = tilesX * tilesX;
    const size_t VV = (size_t)V * V, PV = (size_t)P * V;
    const long long V3 = (long long)VV * V;

    const bool items32 = nItems <= 0x7fffffffLL; // 32-bit division per item whenever it fits
    for (long long item = blockIdx.x; item < nItems; item += gridDim.x) {
        const int a = items32 ? (int)((unsigned)item / (unsigned)tilesPerImg) : (int)(item / tilesPerImg);
        const int t = (int)(item - (long long)a * tilesPerImg);
        const float *ax = axes + 9 * (size_t)a;
        const int i = (t % tilesX) * kFpTile + lx;
        const int j = (t / tilesX) * kFpTile + ly;
        if (i >= M || j >= M) continue;
        float *out = img + (size_t)a * M * M + (size_t)j * M + i;
        const int di = i - ic, dj = j - ic;
        if ((long long)di * di + (long long)dj * dj > R2) {
            *out = 0.0f;
            continue;
        }
        const float nx0 = __ldg(ax + 0), nx1 = __ldg(ax + 1), nx2 = __ldg(ax + 2);
        const float ny0 = __ldg(ax + 3), ny1 = __ldg(ax + 4), ny2 = __ldg(ax + 5);
        const float fi = sample_coord(nx0, ny0, di, dj, vc);
        const float fj = sample_coord(nx1, ny1, di, dj, vc);
        const float fk = sample_coord(nx2, ny2, di, dj, vc);

        int b0, b1, b2;
        float wi[TAPS], wj[TAPS], wk[TAPS];
        if (TAPS == 4) {
            b0 = (int)floorf(fi) - 1;
            b1 = (int)floorf(fj) - 1;
            b2 = (int)floorf(fk) - 1;
#pragma unroll
            for (int d = 0; d < TAPS; d++) {
                // r lies in (-2, 2] for these taps: no clamp needed
                wi[d] = kb_weight(sker, (float)(b0 + d) - fi, kerScale, kerCenterHalf, kerSize);
                wj[d] = kb_weight(sker, (float)(b1 + d) - fj, kerScale, kerCenterHalf, kerSize);
                wk[d] = kb_weight(sker, (float)(b2 + d) - fk, kerScale, kerCenterHalf, kerSize);
            }
        } else {
            b0 = (int)roundf(fi) - 2;
            b1 = (int)roundf(fj) - 2;
            b2 = (int)roundf(fk) - 2;
#pragma unroll
            for (int d = 0; d < TAPS; d++) {
                wi[d] = kb_weight(sker, fminf(fmaxf((float)(b0 + d) - fi, -convW), convW), kerScale, kerCenterHalf, kerSize);
                wj[d] = kb_weight(sker, fminf(fmaxf((float)(b1 + d) - fj, -convW), convW), kerScale, kerCenterHalf, kerSize);
                wk[d] = kb_weight(sker, fminf(fmaxf((float)(b2 + d) - fk, -convW), convW), kerScale, kerCenterHalf, kerSize);
            }
        }

        float acc = 0.0f;
        const bool inside = b0 >= 0 && b1 >= 0 && b2 >= 0 && b0 <= V - TAPS && b1 <= V - TAPS && b2 <= V - TAPS;
        if (inside) {
            const TV *base = vol + (size_t)b2 * PV + (size_t)b1 * P + b0;
#pragma unroll
            for (int dk = 0; dk < TAPS; dk++) {
#pragma unroll
                for (int dj2 = 0; dj2 < TAPS; dj2++) {
                    const TV *p = base + (size_t)dk * PV + (size_t)dj2 * P;
                    float s = 0.0f;
#pragma unroll
                    for (int d = 0; d < TAPS; d++) s = fmaf(wi[d], ld_f32(p + d), s);
                    acc = fmaf(wj[dj2] * wk[dk], s, acc);
                }
            }
        } else {
            // Near the volume edge: the reference's linear-index test on the
            // dense layout (gpuForwardProject.cu:90), plus a lower bound.
            for (int dk = 0; dk < TAPS; dk++)
                for (int dj2 = 0; dj2 < TAPS; dj2++)
                    for (int d = 0; d < TAPS; d++) {
                        const long long lin = (long long)(b2 + dk) * (long long)VV + (long long)(b1 + dj2) * V + (b0 + d);
                        if (lin >= 0 && lin < V3) {
                            const long long row = lin / V;
                            acc = fmaf(wi[d] * wj[dj2] * wk[dk], ld_f32(vol + row * P + (lin - row * V)), acc);
                        }
                    }
        }
        *out = acc * outScale;
    }
}

template <typename TV, int TAPS>
static cudaError_t launch_fp_t(const void *d_vol, int P, float *img, const float *ker, const float *axes, int n,
                               const Geom &g, const float *scale, cudaStream_t s)
{
    const int tilesX = (g.M + kFpTile - 1) / kFpTile;
    const long long nItems = (long long)n * tilesX * tilesX;
    if (nItems == 0) return cudaSuccess;
    int perSm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, fp_kernel<TV, TAPS>, kFpThreads, 0);
    if (perSm <= 0) perSm = 1;
    long long grid = (long long)num_sms() * perSm;
    if (grid > nItems) grid = nItems;
    fp_kernel<TV, TAPS><<<(unsigned)grid, kFpThreads, 0, s>>>((const TV *)d_vol, g.V, P, img, g.M, axes, g.mask_radius,
                                                              ker, g.ker_size, g.ker_hw, tilesX, nItems, scale);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_forward_project(const void *d_vol, int vprec, int pitch, float *d_img, const float *d_ker,
                                   const float *d_axes, int n, const Geom &g, bool five_taps, const float *scale,
                                   cudaStream_t s)
{
    if (vprec == kF32 && !five_taps) return launch_fp_t<float, 4>(d_vol, pitch, d_img, d_ker, d_axes, n, g, scale, s);
    if (!five_taps) return cudaErrorInvalidValue; // 2-byte volumes with zero table edges are projected by tiles
    if (vprec == kF32) return launch_fp_t<float, 5>(d_vol, pitch, d_img, d_ker, d_axes, n, g, scale, s);
    if (vprec == kF16) return launch_fp_t<__half, 5>(d_vol, pitch, d_img, d_ker, d_axes, n, g, scale, s);
    return launch_fp_t<__nv_bfloat16, 5>(d_vol, pitch, d_img, d_ker, d_axes, n, g, scale, s);
}

// ---------------------------------------------------------------------------
// Back projection: the reference window and shared constants
// ---------------------------------------------------------------------------
// Each warp takes the directions in batches of kBpBatch, one per lane for the
// cull.
constexpr int kBpBatch = 32;

// Conservative reach of the slab test: fp32 rounding of f_imgk is far below this.
constexpr float kCullEps = 1e-2f;

struct RefWindow {
    float nx0, nx1, nx2, ny0, ny1, ny2; // direction columns x, y
    float vi, vj, vk;                   // voxel coordinates
    float vc;                           // volume centre
    float kerScale, kerCenterHalf;      // index = floor(r*kerScale + kerCenter + 1/2)
};

// Pixel (i1, j1)'s position along one volume axis, as the reference's build
// evaluates `(i1 - imgCenter) * nx + (j1 - imgCenter) * ny + volCenter`
// (gpuBackProject.cu:77,84,91): fma(pi, nx, pj*ny) + vc, identified by
// replaying the reference kernel's outputs.  Written with round-to-nearest
// intrinsics so no unrolling or hoisting can change which product is fused.
__device__ __forceinline__ float ref_pixel_pos(float pi, float pj, float n_x, float n_y, float vc)
{
    return __fadd_rn(__fmaf_rn(pi, n_x, __fmul_rn(pj, n_y)), vc);
}

// One voxel's 5x5 pixel window under the reference rule (gpuBackProject.cu:74-104),
// unrolled.  The table index floor(fma(r, kerScale, kerCenter + 1/2)) equals
// the reference's roundf(fma(r, kerScale, kerCenter)) for every float r in
// [-2, 2] (checked exhaustively): both round the same exact value once.
// INSIDE: the whole window lies in the image, so the reference's
// linear-index test always passes.  Table entry k is read at sker[k * rep].
// DW: cumW sums img2 * w (a second image back-projected in the same pass,
// fused as cumSum is) instead of w.
template <bool DENS, bool INSIDE, bool DW = false>
__device__ __forceinline__ void ref_window(const RefWindow &q, const float *sker, int rep, const float *__restrict__ img_ptr,
                                           int M, int imgi, int imgj, int imgCenter, float &cumSum, float &cumW,
                                           const float *__restrict__ img2_ptr = nullptr)
{
#pragma unroll
    for (int jo = -2; jo <= 2; jo++) {
        const int j1 = imgj + jo;
        const float pj = (float)(j1 - imgCenter);
#pragma unroll
        for (int io = -2; io <= 2; io++) {
            const int i1 = imgi + io;
            const float pi = (float)(i1 - imgCenter);
            float r = fminf(fmaxf(ref_pixel_pos(pi, pj, q.nx0, q.ny0, q.vc) - q.vi, -2.0f), 2.0f);
            float w = sker[__float2int_rd(__fmaf_rn(r, q.kerScale, q.kerCenterHalf)) * rep];
            r = fminf(fmaxf(ref_pixel_pos(pi, pj, q.nx1, q.ny1, q.vc) - q.vj, -2.0f), 2.0f);
            w = __fmul_rn(w, sker[__float2int_rd(__fmaf_rn(r, q.kerScale, q.kerCenterHalf)) * rep]);
            r = fminf(fmaxf(ref_pixel_pos(pi, pj, q.nx2, q.ny2, q.vc) - q.vk, -2.0f), 2.0f);
            w = __fmul_rn(w, sker[__float2int_rd(__fmaf_rn(r, q.kerScale, q.kerCenterHalf)) * rep]);
            const int lin = j1 * M + i1;
            if (INSIDE || (lin < M * M && lin >= 0)) {
                // cumSum += img * w, fused as the reference's build fuses it
                cumSum = __fmaf_rn(ld_f32(img_ptr + lin), w, cumSum);
                if (DENS) cumW = __fadd_rn(cumW, w);
                if (DW) cumW = __fmaf_rn(__ldg(img2_ptr + lin), w, cumW);
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Back projection, reference window rule
// ---------------------------------------------------------------------------
// Only the voxels inside a direction's slab (|f_imgk| <= 2, a few percent of
// the volume) run the 25-pixel window.  A warp owns an 8x4xBD block of the
// volume, BD voxels per lane: block voxel l = lane + 32 s (x = l & 7, y =
// (l >> 3) & 3, z = l >> 5); eight blocks make a 16x8x(2 BD) brick, the unit in
// which the volume is numbered.  The warp culls the directions 32 at a time,
// one per lane, and for each that reaches its block tests its 32 BD voxels
// against the slab, lists the active ones in shared memory and runs them 32 at
// a time, one per lane.  Every voxel still receives its directions one by one
// in order and its window in the reference's order, so the per-voxel sums are
// those of the reference kernel's loops, bit for bit.  A CTA holds the warps of
// kBpGroups bricks, which share one copy of the KB table (below) and run
// independently.
constexpr int kCBX = 16, kCBY = 8; // brick: 2x2x2 warp blocks of 8x4xBD (BD = 6, or 8 on large images)
constexpr int kCThreads = 256;  // threads of a brick's eight warps
constexpr int kBpGroups = 3;    // bricks' worth of warps per CTA, one CTA per SM
// The two-stack form's 6-deep kernel runs 16 warps per CTA: with the second
// stack's footprints, 24 warps' two buffers do not fit.
template <bool DW, bool DEEP> constexpr int kGroupsOf = (DW && !DEEP) ? 2 : kBpGroups;
// Depth of a warp block: 6 voxels, or 8 (DEEP, reference rule) on CAS images
// of 512^2 and more.  Deeper blocks have more active voxels per direction
// (fewer idle lanes in the last round of 32) and stage a footprint for more
// voxels, which pays most where the images are large (each staging reads from
// L2 or DRAM); on 256^2 images 8-deep blocks measured 20% slower than 4-deep
// ones and 6-deep ones 0.7% faster.  With 6 the footprint still fits 16
// pixels for any orthonormal axes (2 |(3.5, 1.5, 2.5)| + 1.2 < 11).  The
// two-stack form had 4 while its 256-thread CTAs held a padded table each; with
// the shared table copies 6-deep blocks measured faster (CTF-corrected
// reconstructVol 88.6 -> 84.1 ms).
template <bool DW, bool DEEP>
struct BpShape {
    static constexpr int BD = DEEP ? 8 : 6;
    static constexpr int WV = 32 * BD;                         // voxels per warp block
    static constexpr int BZ = 2 * BD;                          // brick depth
    static constexpr int FW = BD == 8 ? 20 : 16;  // footprint width and height
};

// The fast window.  For a voxel coordinate v and a window pixel whose
// volume-frame position along the same axis is Q, the reference's table
// index is floor(fma(clamp(fl(Q - v), -2, 2), s, h)), s = kerScale,
// h = kerCenter + 1/2 (see kb_weight).  For v >= 4 and |Q - v| <= 2,
// Sterbenz's lemma makes fl(Q - v) = Q - v exact, so that fma and
// fma(Q, s, h - v*s) round the same real number (h - v*s is exact: s and h
// are multiples of 1/4).  Scaled by 1/P, P a power of two >= kerSize - 1,
// y = fma(Q, s/P, (h - v*s)/P) is that rounded value over P exactly, and the
// saturating fma clamps it to [0, 1]: for |Q - v| > 2 it lands at or beyond
// the same end of the table as the reference's clamp, and a table of P + 1
// entries that repeats the last one past kerSize - 1 gives the clamped
// entry.  floor(P y) is the low bits of y + 1.5*2^23/P added with round-down.
// The unscaled index was checked on the CPU against the reference formula for
// every float Q within 4.2 of v (v = 4..40; tables of 501 and 1000 entries);
// the scaled, clamped entry on 1.4e8 values of Q within 4.2 of v (v up to
// 600), both neighbours of every index boundary among them, for tables of
// 501, 1000, 101 and 513 entries: identical entries.
//
// The table is held in `copies` interleaved copies (entry k of copy c at word
// k * copies + c) and lane l reads copy l % copies.  With 32 copies (66 KB
// for P = 512) each lane reads its own bank, so the three data-dependent
// lookups per pixel never conflict; shared by the groups of a CTA, the table
// fits beside their working sets.
//
// The pixels come from a per-warp footprint in shared memory: the pixels any
// window of the warp's block can touch, staged per direction with the
// reference's linear-index rule (a pixel whose index falls outside the image
// reads as zero), so the windows read them at constant offsets.
struct BpTable {
    int copies;          // interleaved copies (32: conflict-free)
    int entries;         // P + 1
    float scale;         // 1 / P
    float magic;         // 1.5 * 2^23 / P
    unsigned magic_bits; // its bits: entry floor(P y) sits at bits(y + magic) - magic_bits
};

// Four consecutive values from a 4-element-aligned address.
__device__ __forceinline__ void ld_quad(const float *p, float (&v)[4])
{
    const float4 q = __ldg(reinterpret_cast<const float4 *>(p));
    v[0] = q.x;
    v[1] = q.y;
    v[2] = q.z;
    v[3] = q.w;
}
__device__ __forceinline__ float lds_f32(unsigned addr)
{
    float v;
    asm("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}

__device__ __forceinline__ void cp_async16(float *dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

struct FootWin {
    float nx0, nx1, nx2, ny0, ny1, ny2;
    float vc;         // volume centre
    float s;          // kerScale / P
    float c0, c1, c2; // (h - v*s) / P per axis
    float mg;         // 1.5 * 2^23 / P
    unsigned stride;  // bytes between table entries
};

// fma rounded to nearest, clamped to [0, 1] (a NaN gives 0).
__device__ __forceinline__ float fma_sat(float a, float b, float c)
{
    float d;
    asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// One voxel's WI x WJ window from the footprint (fbase = its top-left pixel,
// rows FS apart); table entry floor(P y) is read at
// tab + bits(y + q.mg) * stride.  Sums row by row, as the reference.  TS: the
// stride in bytes when known at compile time (128 for 32 interleaved table
// copies), so the address is a shift-add on the integer pipe rather than a
// multiply on the FMA pipe; 0: q.stride.  Adjacent pixels of a row go in pairs
// through the packed FP32x2 instructions (sm_100+): the pixel positions, the table
// addresses and the weight products of two pixels per instruction (the
// saturating index fma has no packed form).  Each lane of a packed instruction
// rounds as the scalar instruction does and the sums take one pixel at a time,
// in order, so every weight and sum has the scalar form's bits.
__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }

template <bool DENS, int WI, int WJ, int FS, bool DW = false, int TS = 0>
__device__ __forceinline__ void foot_window_x2(const FootWin &q, const float *fbase, unsigned tab, float pi0,
                                               float pj0, float &cumSum, float &cumW, const float *fbase2 = nullptr)
{
    const unsigned st = TS ? (unsigned)TS : q.stride;
    const float2 nx0 = f2(q.nx0, q.nx0), nx1 = f2(q.nx1, q.nx1), nx2 = f2(q.nx2, q.nx2);
    const float2 vc = f2(q.vc, q.vc), mg = f2(q.mg, q.mg);
#pragma unroll
    for (int jo = 0; jo < WJ; jo++) {
        const float pj = pj0 + (float)jo;
        const float py0 = __fmul_rn(pj, q.ny0), py1 = __fmul_rn(pj, q.ny1), py2 = __fmul_rn(pj, q.ny2);
        const float2 qy0 = f2(py0, py0), qy1 = f2(py1, py1), qy2 = f2(py2, py2);
#pragma unroll
        for (int io = 0; io + 1 < WI; io += 2) {
            const float2 pi = f2(pi0 + (float)io, pi0 + (float)(io + 1));
            const float2 q0 = __fadd2_rn(__ffma2_rn(pi, nx0, qy0), vc);
            const float2 q1 = __fadd2_rn(__ffma2_rn(pi, nx1, qy1), vc);
            const float2 q2 = __fadd2_rn(__ffma2_rn(pi, nx2, qy2), vc);
            const float2 b0 = __fadd2_rd(f2(fma_sat(q0.x, q.s, q.c0), fma_sat(q0.y, q.s, q.c0)), mg);
            const float2 b1 = __fadd2_rd(f2(fma_sat(q1.x, q.s, q.c1), fma_sat(q1.y, q.s, q.c1)), mg);
            const float2 b2 = __fadd2_rd(f2(fma_sat(q2.x, q.s, q.c2), fma_sat(q2.y, q.s, q.c2)), mg);
            const float2 t0 = f2(lds_f32(tab + __float_as_uint(b0.x) * st),
                                 lds_f32(tab + __float_as_uint(b0.y) * st));
            const float2 t1 = f2(lds_f32(tab + __float_as_uint(b1.x) * st),
                                 lds_f32(tab + __float_as_uint(b1.y) * st));
            const float2 t2 = f2(lds_f32(tab + __float_as_uint(b2.x) * st),
                                 lds_f32(tab + __float_as_uint(b2.y) * st));
            const float2 w = __fmul2_rn(__fmul2_rn(t0, t1), t2);
            cumSum = __fmaf_rn(fbase[jo * FS + io], w.x, cumSum);
            if (DENS) cumW = __fadd_rn(cumW, w.x);
            if (DW) cumW = __fmaf_rn(fbase2[jo * FS + io], w.x, cumW);
            cumSum = __fmaf_rn(fbase[jo * FS + io + 1], w.y, cumSum);
            if (DENS) cumW = __fadd_rn(cumW, w.y);
            if (DW) cumW = __fmaf_rn(fbase2[jo * FS + io + 1], w.y, cumW);
        }
        if (WI & 1) {
            constexpr int io = WI - 1;
            const float pi = pi0 + (float)io;
            const float q0 = __fadd_rn(__fmaf_rn(pi, q.nx0, py0), q.vc);
            const float q1 = __fadd_rn(__fmaf_rn(pi, q.nx1, py1), q.vc);
            const float q2 = __fadd_rn(__fmaf_rn(pi, q.nx2, py2), q.vc);
            const unsigned b0 = __float_as_uint(__fadd_rd(fma_sat(q0, q.s, q.c0), q.mg));
            const unsigned b1 = __float_as_uint(__fadd_rd(fma_sat(q1, q.s, q.c1), q.mg));
            const unsigned b2 = __float_as_uint(__fadd_rd(fma_sat(q2, q.s, q.c2), q.mg));
            float w = lds_f32(tab + b0 * st);
            w = __fmul_rn(w, lds_f32(tab + b1 * st));
            w = __fmul_rn(w, lds_f32(tab + b2 * st));
            cumSum = __fmaf_rn(fbase[jo * FS + io], w, cumSum);
            if (DENS) cumW = __fadd_rn(cumW, w);
            if (DW) cumW = __fmaf_rn(fbase2[jo * FS + io], w, cumW);
        }
    }
}

static int max_dyn_smem()
{
    static std::atomic<int> cache[kAttrCacheDevices];
    return device_attr(cudaDevAttrMaxSharedMemoryPerBlockOptin, cache, 48 * 1024);
}

// The table layout for kerSize entries beside other_bytes of shared memory:
// P = 512 (kerSize <= 513) or the next power of two, and as many copies, 32
// down to 1, as fit.  copies = 0: not even one copy fits.
static BpTable bp_table(int kerSize, size_t other_bytes, int max_copies = 32, size_t limit_bytes = 0)
{
    int P = 512;
    while (P < kerSize - 1) P *= 2;
    BpTable t;
    t.entries = P + 1;
    t.scale = 1.0f / (float)P;
    t.magic = 12582912.0f / (float)P;
    std::memcpy(&t.magic_bits, &t.magic, sizeof(float));
    t.copies = max_copies;
    const size_t limit = limit_bytes ? limit_bytes : (size_t)max_dyn_smem();
    while (t.copies > 0 && (((size_t)t.entries * t.copies + 3) & ~(size_t)3) * sizeof(float) + other_bytes > limit)
        t.copies /= 2;
    return t;
}

// DW (reference rule, FP32 images): pd accumulates the back projection of a
// second image stack img2 (the same directions) in the same pass, with the
// same weights and summation order as a separate back projection of img2.
// What a queued voxel's window needs of its direction, copied when the
// direction's footprint is staged.
struct alignas(16) BpDirMeta {
    float nx0, nx1, nx2, ny0, ny1, ny2;
    int fi0, fj0, fh, foot, dir, pad;
};

// A warp's queue of voxel windows: entries (block voxel | footprint buffer
// << 8) in direction order, run 32 at a time, so that rounds are full across
// directions.  NB footprint buffers per warp: 2 where shared memory allows
// (the 6-deep forms; a direction's footprint is staged while the previous
// direction's last voxels still wait in the queue); else 1, and each direction's active voxels
// run at once from the same array (a plain list, no queue): queue rounds with
// one buffer measured slower (per-lane direction records, spills).
template <bool DW, bool DEEP>
struct BpQueue {
    static constexpr int NB = !DEEP ? 2 : 1;
    static constexpr int NEED = (NB - 1) * 31 + BpShape<DW, DEEP>::WV; // most entries held at once
    static constexpr int CAP = NEED <= 128 ? 128 : (NEED <= 256 ? 256 : 512);
};

// One warp's working set in shared memory (after the table).  LEAN (the
// launches that own the GPU): 8-bit queue entries with the footprint buffer
// tracked per warp, and in the two-buffer form footprint rows of FW + 4 pixels
// from fi0 & ~3 (16-byte aligned, copied in 16-byte quads).  Otherwise (the
// serving lanes' one-brick CTAs): 16-bit entries carrying the buffer bit, rows
// of FW + 1 pixels from fi0.
template <bool DENS, bool DW, bool DEEP, bool LEAN = true>
struct alignas(16) BpWarpMem {
    using Shape = BpShape<DW, DEEP>;
    using Q = BpQueue<DW, DEEP>;
    using QEnt = typename std::conditional<LEAN, unsigned char, unsigned short>::type;
    static constexpr int WV = Shape::WV, FP = Shape::FW * (Shape::FW + (LEAN && Q::NB == 2 ? 4 : 1));
    float sfoot[Q::NB * FP];
    float sfoot2[DW ? Q::NB * FP : 4];
    BpDirMeta smeta[Q::NB];
    float sdir[2][kBpBatch * 9]; // two batches of directions
    // per-voxel sums; a voxel is updated by at most one lane per direction,
    // directions in order, so no atomics are needed
    float sacc[WV];
    float saccw[DENS || DW ? WV : 4];
    QEnt squeue[Q::CAP];
};

// Bricks of x-width kCBX in row (y brick j, z brick k) that meet the sphere of
// radius reach about the volume centre c (within the +1 margin of the test
// d^2 <= reach^2 + 1, d the distance from the centre to the brick's box):
// x bricks lo .. lo + n - 1.  In doubled coordinates the box's distance per
// axis is max(|2 B i + B - 1 - 2c| - (B - 1), 0) for bricks of size B, all
// integers, so the test is exact; along x the bricks that pass form the
// interval |2 B i + B - 1 - 2c| <= B - 1 + t, t = isqrt(rem).
__host__ __device__ __forceinline__ int box_dist2(int i, int B, int c)
{
    const int d = 2 * B * i + B - 1 - 2 * c, e = (d < 0 ? -d : d) - (B - 1);
    return e > 0 ? e : 0;
}

__host__ __device__ __forceinline__ int floor_div(int a, int b) { return a >= 0 ? a / b : -((-a + b - 1) / b); }

__host__ __device__ inline void brick_row(int j, int k, int bricksX, int c, int BZ, int reach, int &lo, int &n)
{
    const long long dy = box_dist2(j, kCBY, c), dz = box_dist2(k, BZ, c);
    const long long rem = 4 * ((long long)reach * reach + 1) - dy * dy - dz * dz;
    lo = 0;
    n = 0;
    if (rem < 0) return;
    long long t = (long long)sqrtf((float)rem); // a guess, corrected below
    while (t * t > rem) t--;
    while ((t + 1) * (t + 1) <= rem) t++;
    const int B = kCBX;
    int ilo = -floor_div(-(2 * c - 2 * (B - 1) - (int)t), 2 * B); // ceil
    if (ilo < 0) ilo = 0;
    int ihi = floor_div(2 * c + (int)t, 2 * B);
    if (ihi > bricksX - 1) ihi = bricksX - 1;
    if (ihi >= ilo) {
        lo = ilo;
        n = ihi - ilo + 1;
    }
}

// Rank r of 0 .. n - 1 from the middle outwards: the bricks near the centre,
// which the most directions reach, start first, and the light ones at the rim
// fill the last wave (two-stack form, 1,000 images at M = 256: 7.94 -> 7.53 ms
// a call; reconstructVol of 1,000 at M = 128: 4.81 -> 4.58 ms before the
// segments).
__host__ __device__ __forceinline__ int middle_out(int r, int n)
{
    const int c = (n - 1) / 2;
    return r & 1 ? c + (r + 1) / 2 : c - r / 2;
}

// The bricks of a launch, layer by layer from the middle outwards: layer rank r
// holds bricks pre[r] .. pre[r + 1] - 1, row by row.  Counted on the host, so that
// no CTA starts (and takes a whole SM) without bricks: at M = 256 the box of
// bricks holds 6,182 runs, of which 1,900 meet the sphere (reconstructVol of
// 1,000 images 6.99 -> 6.66 ms, of 16 images 688 -> 618 us).
constexpr int kMaxLayers = 511; // 6,132 voxels of 12-deep bricks: 860 GB of CAS volume
struct BpLayers {
    int layers, pre[kMaxLayers + 1];
};

// Place (x, y, z) of a brick in its layer's rows, by a scan over the rows; the
// whole warp calls it for one brick.  Out of line: inlined, its invariants
// took registers through the window loops.
__device__ __noinline__ int3 brick_at(int brick, const BpLayers &lay, int bricksX, int bricksY, int c, int BZ, int maskR)
{
    const int lane = threadIdx.x & 31;
    int rank = 0; // the last layer rank whose first brick is <= brick
    for (int hi = lay.layers - 1; rank < hi;) {
        const int mid = (rank + hi + 1) >> 1;
        if (lay.pre[mid] <= brick) rank = mid;
        else hi = mid - 1;
    }
    int3 at = make_int3(0, 0, middle_out(rank, lay.layers));
    for (int j0 = 0, before = lay.pre[rank]; j0 < bricksY; j0 += 32) {
        int lo = 0, cnt = 0;
        if (j0 + lane < bricksY) brick_row(j0 + lane, at.z, bricksX, c, BZ, maskR, lo, cnt);
        int incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += up;
        }
        const int first = before + incl - cnt;
        const unsigned hit = __ballot_sync(0xffffffffu, brick >= first && brick < first + cnt);
        if (hit) {
            const int src = __ffs(hit) - 1;
            at.x = __shfl_sync(0xffffffffu, lo + brick - first, src);
            at.y = j0 + src;
            break;
        }
        before += __shfl_sync(0xffffffffu, incl, 31);
    }
    return at;
}

__device__ __forceinline__ void cp_async4(float *dst, const float *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.wait_all;" ::: "memory");
}

template <bool DENS, bool DW = false, bool DEEP = false, int G = kBpGroups,
          int TS = 0, bool LEAN = true, bool SPLIT = false>
__global__ void __launch_bounds__(kCThreads *G, G == 1 ? 3 : 1)
bp_ref_compact_kernel(float *__restrict__ vol, float *__restrict__ pd, int V, const float *__restrict__ img, int M,
                      const float *__restrict__ axes, int n, int maskR, const float *__restrict__ ker, int kerSize,
                      float kerHW, int bricksX, int bricksY, BpTable tb,
                      const float *__restrict__ d_scale, const float *__restrict__ img2, int vecImg, BpSplit split,
                      const __grid_constant__ BpLayers lay)
{
    static_assert(!DW || !DENS, "the second image stack is a reference-rule option");
    constexpr int W = 5, HALF = W / 2;
    using Shape = BpShape<DW, DEEP>;
    constexpr int BD = Shape::BD, kWarpVox = Shape::WV, kCBZ = Shape::BZ;
    // LEAN two-buffer form: footprint rows hold the pixels from fi0 & ~3 (16-byte aligned rows)
    constexpr bool QALIGN = LEAN && BpQueue<DW, DEEP>::NB == 2;
    constexpr int FW = Shape::FW, FH = FW, FS = FW + (QALIGN ? 4 : 1);
    using Mem = BpWarpMem<DENS, DW, DEEP, LEAN>;
    using QEnt = typename Mem::QEnt;
    constexpr int NW = kCThreads / 32 * G; // warps of the CTA
    // [table: tb.entries x tb.copies][NW x Mem]
    extern __shared__ __align__(16) float bp_smem[];
    const int cp = tb.copies, tabWords = tb.entries * cp;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    Mem &sm = reinterpret_cast<Mem *>(bp_smem + ((tabWords + 3) & ~3))[warp]; // 16-byte aligned
    const int volCenter = (int)((float)V) / 2;
    const int imgCenter = (int)((float)M) / 2;

    if (TS == 128) { // 32 copies: a warp's lanes store 16 copies of 8 entries
        for (int t = threadIdx.x; t < tb.entries * 8; t += blockDim.x) {
            const float w = __ldg(ker + min(t >> 3, kerSize - 1));
            reinterpret_cast<float4 *>(bp_smem)[t] = make_float4(w, w, w, w);
        }
    } else {
        for (int t = threadIdx.x; t < tabWords; t += blockDim.x) bp_smem[t] = __ldg(ker + min(t / cp, kerSize - 1));
    }
    __syncthreads();

    // Items: the warp blocks of the bricks that meet the mask sphere (SPLIT:
    // times the segments of the directions, a block's side by side), heaviest
    // layers first.  With a counter (split.next) each warp takes the next item
    // on its own: the warps share the table and nothing else.  Barriers between
    // the eight warps of a brick (for each 512 staged directions) held them 23%
    // of their time, and a CTA that ended with the slowest of three bricks idled
    // 15% of its warps.  reconstructVol, before the counter / with a counter per
    // brick group / per warp: 700 images (FP16) at M = 384 11.93 / 11.22 / 10.19
    // ms; CTF-corrected 1,000 at M = 256 6.96 / 6.55 / 5.89 ms; 512 at M = 512
    // 15.24 / 14.56 / 13.86 ms; 16 at M = 256 530 / 477 / 409 us.
    const int ns = SPLIT ? split.nseg : 1, items = lay.pre[lay.layers] * 8 * ns;
    // With a counter the first items are dealt out across the SMs, so that an
    // SM's warps share the heavy ones with others (reconstructVol of 16 images
    // at M = 128: 131 us against 142 for neighbouring items; no difference for
    // large launches); without one, a CTA's warps take neighbouring items.
    for (int item = split.next ? warp * gridDim.x + blockIdx.x : blockIdx.x * NW + warp; item < items;) {
        const int block = SPLIT ? item / ns : item;
        const int3 at = brick_at(block >> 3, lay, bricksX, bricksY, volCenter, kCBZ, maskR);
        const int d0 = SPLIT ? (int)((long long)n * (item % ns) / ns) : 0;
        const int d1 = SPLIT ? (int)((long long)n * (item % ns + 1) / ns) : n;
        const int bx = at.x * kCBX + (block & 1) * 8, by = at.y * kCBY + ((block >> 1) & 1) * 4,
                  bz = at.z * kCBZ + ((block >> 2) & 1) * BD;
        const float *sker = bp_smem + lane % cp; // entry k at sker[k * cp]
        const unsigned stride = 4u * (unsigned)cp;
        const unsigned tab = (unsigned)__cvta_generic_to_shared(bp_smem) + 4u * (unsigned)(lane % cp) - tb.magic_bits * stride;
        constexpr int NB = BpQueue<DW, DEEP>::NB, QM = BpQueue<DW, DEEP>::CAP - 1;
        float *const wfoot0 = sm.sfoot, *const wfoot20 = sm.sfoot2;
        BpDirMeta *const wmeta = sm.smeta;
        QEnt *const wq = sm.squeue;
        float *const wacc = sm.sacc, *const waccw = sm.saccw;

        // this lane's voxels: x = lx, y = ly, z = bz + s
        const int lx = bx + (lane & 7), ly = by + (lane >> 3);
        const long long R2 = (long long)maskR * maskR;
        unsigned inmask = 0;
#pragma unroll
        for (int s = 0; s < BD; s++) {
            const int lz = bz + s;
            const long long d2 = (long long)(lx - volCenter) * (lx - volCenter) + (long long)(ly - volCenter) * (ly - volCenter) +
                                 (long long)(lz - volCenter) * (lz - volCenter);
            if (lx < V && ly < V && lz < V && d2 <= R2) inmask |= 1u << s;
            wacc[lane + 32 * s] = 0.0f;
            if (DENS || DW) waccw[lane + 32 * s] = 0.0f;
        }
        const float kerCenter = ((float)kerSize - 1) / 2;
        const float kerScale = kerCenter / kerHW;
        const float kerCenterHalf = kerCenter + 0.5f;
        const float ax0 = (float)lx - volCenter, ay0 = (float)ly - volCenter;
        const float wcx = bx + 3.5f - volCenter, wcy = by + 1.5f - volCenter, wcz = bz + 0.5f * (BD - 1) - volCenter;
        const float slab = kerHW + kCullEps; // half-thickness
        const int MM = M * M;
        const unsigned lt_mask = (1u << lane) - 1u;
        // the warp's queue (uniform): qsize entries from qhead.  LEAN: the first
        // nfront belong to footprint buffer bfront, the rest to the other
        // buffer; otherwise each entry carries its buffer in bit 8
        int qhead = 0, qsize = 0, nbuf = 0, nfront = 0, bfront = 0;

        // One voxel's window sum for one direction: the fast window from the
        // footprint, or the reference's window from the image.
        auto voxel_window = [&](const int l, const float nx0, const float nx1, const float nx2, const float ny0,
                                const float ny1, const float ny2, const int fi0, const int fj0, const int fh,
                                const bool foot, const float *img_ptr, const float *img2_ptr, const float *wfoot,
                                const float *wfoot2, float &cs, float &cw) {
            const int vi = bx + (l & 7), vj = by + ((l >> 3) & 3), vk = bz + (l >> 5);
            const float a0 = (float)vi - volCenter, a1 = (float)vj - volCenter, a2 = (float)vk - volCenter;
            const float f_imgi = __fadd_rn(voxel_proj(a0, a1, a2, nx0, nx1, nx2), (float)imgCenter);
            const float f_imgj = __fadd_rn(voxel_proj(a0, a1, a2, ny0, ny1, ny2), (float)imgCenter);
            const int imgi = (int)roundf(f_imgi);
            const int imgj = (int)roundf(f_imgj);
            const bool inside = imgi >= 2 && imgj >= 2 && imgi < M - 2 && imgj < M - 2; // no sum: axes may be anything
            const int ri = imgi - HALF - fi0, rj = imgj - HALF - fj0;
            if (foot && (unsigned)ri <= (unsigned)(FW - W) && (unsigned)rj <= (unsigned)(fh - W) && vi >= 4 &&
                vj >= 4 && vk >= 4 && (inside || !DENS)) {
                // index of r = Q - v, scaled by 1/P (exact): the saturating index form
                const float sg = kerScale;
                const FootWin fwin{nx0, nx1, nx2, ny0, ny1, ny2, (float)volCenter, sg * tb.scale,
                                   (kerCenterHalf - (float)vi * sg) * tb.scale,
                                   (kerCenterHalf - (float)vj * sg) * tb.scale,
                                   (kerCenterHalf - (float)vk * sg) * tb.scale, tb.magic, stride};
                const float *fb = wfoot + rj * FS + ri + (QALIGN ? (fi0 & 3) : 0);
                const float pi0 = (float)(imgi - HALF - imgCenter), pj0 = (float)(imgj - HALF - imgCenter);
                foot_window_x2<DENS, W, W, FS, DW, TS>(fwin, fb, tab, pi0, pj0, cs, cw,
                                                DW ? wfoot2 + rj * FS + ri + (QALIGN ? (fi0 & 3) : 0) : nullptr);
            } else {
                const RefWindow rw{nx0, nx1, nx2, ny0, ny1, ny2, (float)vi, (float)vj, (float)vk,
                                   (float)volCenter, kerScale, kerCenterHalf};
                if (inside)
                    ref_window<DENS, true, DW>(rw, sker, cp, img_ptr, M, imgi, imgj, imgCenter, cs, cw,
                                                         img2_ptr);
                else
                    ref_window<DENS, false, DW>(rw, sker, cp, img_ptr, M, imgi, imgj, imgCenter, cs, cw,
                                                          img2_ptr);
            }
        };

        // One round of the queue (NB = 2): its first cnt (<= 32) voxels, one per
        // lane.  Each voxel's window sum is added to its total in direction
        // order: the round holds at most one direction per buffer, the older
        // one's first.
        auto run_round = [&](const int cnt) {
            float cs = 0.0f, cw = 0.0f;
            int l = 0, b = 0;
            if (lane < cnt) {
                const unsigned ent = wq[(qhead + lane) & QM];
                l = ent & 0xff;
                b = LEAN ? (lane < nfront ? bfront : (bfront ^ 1)) : (int)(ent >> 8);
                const BpDirMeta m = wmeta[b];
                voxel_window(l, m.nx0, m.nx1, m.nx2, m.ny0, m.ny1, m.ny2, m.fi0, m.fj0, m.fh, m.foot != 0,
                             img + (size_t)m.dir * MM, DW ? img2 + (size_t)m.dir * MM : nullptr, wfoot0 + b * (FH * FS),
                             wfoot20 + (DW ? b * (FH * FS) : 0), cs, cw);
            }
            // cumSumAllAxes += cumSum (gpuBackProject.cu:106), in direction order
            const int bf = LEAN ? bfront : (int)(wq[qhead & QM] >> 8);
            if (lane < cnt && b == bf) {
                wacc[l] = __fadd_rn(wacc[l], cs);
                if (DENS || DW) waccw[l] = __fadd_rn(waccw[l], cw);
            }
            __syncwarp();
            if (lane < cnt && b != bf) {
                wacc[l] = __fadd_rn(wacc[l], cs);
                if (DENS || DW) waccw[l] = __fadd_rn(waccw[l], cw);
            }
            __syncwarp(); // the entries, buffers and sums are free again
            qhead = (qhead + cnt) & QM;
            qsize -= cnt;
            nfront -= cnt;
            if (nfront <= 0) { // the front direction is done: the rest are the other buffer's
                bfront ^= 1;
                nfront = qsize;
            }
        };

        // a batch of directions, a lane's nine floats each, copied a batch ahead
        auto fetch = [&](const int c) {
            if (c + lane < d1) {
#pragma unroll
                for (int u = 0; u < 9; u++)
                    cp_async4(sm.sdir[(c - d0) / kBpBatch & 1] + lane * 9 + u, axes + (size_t)(c + lane) * 9 + u);
            }
        };
        fetch(d0);
        for (int c0 = d0; c0 < d1; c0 += kBpBatch) {
            const float *const sdir = sm.sdir[(c0 - d0) / kBpBatch & 1];
            cp_async_wait();
            __syncwarp(); // the batch is here, for every lane; the other buffer is free
            fetch(c0 + kBpBatch);
            // cull: lane l tests direction c0 + l against the warp's 8x4xBD block
            bool keep = false, ortho = false;
            if (c0 + lane < d1) {
                const float *ax = sdir + lane * 9;
                const float zx = ax[6], zy = ax[7], zz = ax[8];
                const float dd = wcx * zx + wcy * zy + wcz * zz;
                const float ext = 0.5f * (7.0f * fabsf(zx) + 3.0f * fabsf(zy) + (float)(BD - 1) * fabsf(zz));
                keep = fabsf(dd) <= slab + ext;
                // the fast window needs orthonormal axes (they bound |Q - v|);
                // NaN or infinite entries fail these tests
                const float xx = ax[0] * ax[0] + ax[1] * ax[1] + ax[2] * ax[2];
                const float yy = ax[3] * ax[3] + ax[4] * ax[4] + ax[5] * ax[5];
                const float zz2 = zx * zx + zy * zy + zz * zz;
                const float xy = ax[0] * ax[3] + ax[1] * ax[4] + ax[2] * ax[5];
                const float xz = ax[0] * zx + ax[1] * zy + ax[2] * zz;
                const float yz = ax[3] * zx + ax[4] * zy + ax[5] * zz;
                ortho = fabsf(xx - 1.0f) <= 1e-3f && fabsf(yy - 1.0f) <= 1e-3f && fabsf(zz2 - 1.0f) <= 1e-3f &&
                        fabsf(xy) <= 1e-3f && fabsf(xz) <= 1e-3f && fabsf(yz) <= 1e-3f;
            }
            unsigned hits = __ballot_sync(0xffffffffu, keep);
            const unsigned orthos = __ballot_sync(0xffffffffu, ortho);
            // NB = 2: a pass beyond the last batch's hits runs what is left in
            // the queue, so that the window code is expanded once
            const bool last = NB > 1 && c0 + kBpBatch >= d1;
            while (hits || last) {
                const bool flush = NB > 1 && hits == 0;
                const int al = flush ? 0 : __ffs(hits) - 1;
                hits &= hits - 1;
                const float *ax = sdir + al * 9;
                const float nz0 = ax[6], nz1 = ax[7], nz2 = ax[8];
                // Whole rounds, and whatever buffer b's earlier direction still
                // has in the queue (at its front), run before b is refilled.
                const int b = NB > 1 ? nbuf : 0;
                if (NB > 1) {
                    if (QALIGN) {
                        cp_async_wait();
                        __syncwarp(); // the footprints' copies are complete, for every lane
                    }
                    while (qsize >= 32 || (qsize > 0 && (flush || (LEAN ? bfront : (int)(wq[qhead & QM] >> 8)) == b)))
                        run_round(min(qsize, 32));
                    if (flush) break;
                }
                // the reference's per-voxel slab test (gpuBackProject.cu:64-66);
                // the active voxels join the queue (NB = 1: the list) slot by
                // slot in lane order
                const int tail = NB > 1 ? qhead + qsize : 0;
                int total = 0;
#pragma unroll
                for (int s = 0; s < BD; s++) {
                    const float az = (float)(bz + s) - volCenter;
                    const float fk = voxel_proj(ax0, ay0, az, nz0, nz1, nz2);
                    const bool act = ((inmask >> s) & 1u) && fabsf(fk) <= kerHW;
                    const unsigned bal = __ballot_sync(0xffffffffu, act);
                    if (act) wq[(tail + total + __popc(bal & lt_mask)) & QM] = (QEnt)((lane + 32 * s) | (LEAN ? 0 : b << 8));
                    total += __popc(bal);
                }
                if (total == 0) continue;
                if (NB > 1) nbuf ^= 1;
                float *const wfoot = wfoot0 + b * (FH * FS);
                float *const wfoot2 = wfoot20 + (DW ? b * (FH * FS) : 0);
                const float nx0 = ax[0], nx1 = ax[1], nx2 = ax[2];
                const float ny0 = ax[3], ny1 = ax[4], ny2 = ax[5];
                const float *img_ptr = img + (size_t)(c0 + al) * MM;
                const float *img2_ptr = DW ? img2 + (size_t)(c0 + al) * MM : nullptr;
                // this warp's footprint (uniform across the warp)
                int fi0 = 0, fj0 = 0, fh = 0;
                bool foot = false;
                if ((orthos >> al) & 1u) {
                    const float ic = wcx * nx0 + wcy * nx1 + wcz * nx2 + (float)imgCenter;
                    const float jc = wcx * ny0 + wcy * ny1 + wcz * ny2 + (float)imgCenter;
                    const float hz = 0.5f * (float)(BD - 1);
                    const float hi = 3.5f * fabsf(nx0) + 1.5f * fabsf(nx1) + hz * fabsf(nx2);
                    const float hj = 3.5f * fabsf(ny0) + 1.5f * fabsf(ny1) + hz * fabsf(ny2);
                    // at most 2 |(3.5, 1.5, hz)| + 1.2 apart: width and height fit FW
                    fi0 = __float2int_rd(ic - hi - 0.6f) - HALF;
                    fj0 = __float2int_rd(jc - hj - 0.6f) - HALF;
                    fh = __float2int_rd(jc + hj + 0.6f) + HALF - fj0 + 1;
                    foot = fh <= FH;
                    if (foot && vecImg) {
                        // vector loads of aligned pixel quads (rows start at
                        // multiples of 4 elements: 4 divides M, the image stacks
                        // are aligned), the linear-index rule still applied
                        // pixel by pixel
                        constexpr int NQ = FW / 4 + 1; // quads per footprint row
                        const int base = fi0 & ~3, sh = fi0 & 3;
                        const int first = fj0 * M + base, nq = fh * NQ;
                        if constexpr (QALIGN) {
                            if (first >= 0 && first + (fh - 1) * M + 4 * NQ <= MM) {
                                // no pixel outside the image's index range: quad t of
                                // the footprint lies at its word 4 t (FS = 4 NQ).
                                // Copied behind the warp's back: nothing is held in
                                // registers, and the copies are waited for when the
                                // next direction's rounds begin
                                for (int t = lane; t < nq; t += 32) {
                                    const int o = first + (t / NQ) * (M - 4 * NQ) + 4 * t;
                                    cp_async16(wfoot + 4 * t, img_ptr + o);
                                    if (DW) cp_async16(wfoot2 + 4 * t, img2_ptr + o);
                                }
                            } else {
#pragma unroll 1
                                for (int t = lane; t < nq; t += 32) {
                                    const int lin0 = first + (t / NQ) * (M - 4 * NQ) + 4 * t;
#pragma unroll
                                    for (int e = 0; e < 4; e++) {
                                        const bool in = lin0 + e >= 0 && lin0 + e < MM;
                                        wfoot[4 * t + e] = in ? ld_f32(img_ptr + lin0 + e) : 0.0f;
                                        if (DW) wfoot2[4 * t + e] = in ? __ldg(img2_ptr + lin0 + e) : 0.0f;
                                    }
                                }
                            }
                        } else {
                            // a lane's quads (at most KQ) are all loaded before any is
                            // stored, so their L2 latencies overlap
                            static_assert(!DW, "the two-stack form stages by copies");
                            constexpr int KQ = (FH * NQ + 31) / 32;
                            float v[KQ][4];
#pragma unroll
                            for (int u = 0; u < KQ; u++) {
                                const int t = lane + 32 * u;
#pragma unroll
                                for (int e = 0; e < 4; e++) v[u][e] = 0.0f;
                                if (t < nq) {
                                    const int r = t / NQ, qq = t - r * NQ;
                                    const int lin0 = (fj0 + r) * M + base + 4 * qq;
                                    if (lin0 >= 0 && lin0 + 3 < MM) {
                                        ld_quad(img_ptr + lin0, v[u]);
                                    } else {
#pragma unroll
                                        for (int e = 0; e < 4; e++)
                                            if (lin0 + e >= 0 && lin0 + e < MM) v[u][e] = ld_f32(img_ptr + lin0 + e);
                                    }
                                }
                            }
#pragma unroll
                            for (int u = 0; u < KQ; u++) {
                                const int t = lane + 32 * u;
                                if (t < nq) {
                                    const int r = t / NQ, qq = t - r * NQ;
                                    const int c0 = 4 * qq - sh; // footprint column of the quad's first pixel
#pragma unroll
                                    for (int e = 0; e < 4; e++)
                                        if (c0 + e >= 0 && c0 + e < FW) wfoot[r * FS + c0 + e] = v[u][e];
                                }
                            }
                        }
                    } else if (foot) {
                        // the reference's linear-index rule (gpuBackProject.cu:99)
                        for (int t = lane; t < fh * FW; t += 32) {
                            const int r = t / FW, c = t - r * FW;
                            const int lin = (fj0 + r) * M + (fi0 + c);
                            float v = 0.0f, v2 = 0.0f;
                            if (lin >= 0 && lin < MM) {
                                v = ld_f32(img_ptr + lin);
                                if (DW) v2 = __ldg(img2_ptr + lin);
                            }
                            wfoot[r * FS + c + (QALIGN ? (fi0 & 3) : 0)] = v;
                            if (DW) wfoot2[r * FS + c + (QALIGN ? (fi0 & 3) : 0)] = v2;
                        }
                    }
                }
                if (NB > 1) {
                    if (lane == 0)
                        wmeta[b] = BpDirMeta{nx0, nx1, nx2, ny0, ny1, ny2, fi0, fj0, fh, foot ? 1 : 0, c0 + al, 0};
                    if (qsize == 0) {
                        bfront = b;
                        nfront = total;
                    }
                    qsize += total;
                    __syncwarp(); // the queue entries, the footprint and its record are complete
                } else {
                    __syncwarp(); // the voxel list and the footprint are complete
                    for (int base = 0; base < total; base += 32) {
                        const int t = base + lane;
                        if (t < total) {
                            float cs = 0.0f, cw = 0.0f;
                            const int l = wq[t];
                            voxel_window(l, nx0, nx1, nx2, ny0, ny1, ny2, fi0, fj0, fh, foot, img_ptr, img2_ptr, wfoot,
                                         wfoot2, cs, cw);
                            // cumSumAllAxes += cumSum (gpuBackProject.cu:106), in direction order
                            wacc[l] = __fadd_rn(wacc[l], cs);
                            if (DENS || DW) waccw[l] = __fadd_rn(waccw[l], cw);
                        }
                    }
                    __syncwarp(); // the next direction rewrites the list, the footprint and these sums
                }
            }
        }
        __syncwarp();
        const float sc = d_scale ? *d_scale : 1.0f;
#pragma unroll
        for (int s = 0; s < BD; s++) {
            if (!((inmask >> s) & 1u)) continue;
            if (!SPLIT || item % ns == 0) {
                const size_t o = (size_t)(bz + s) * V * V + (size_t)ly * V + lx;
                vol[o] = vol[o] + wacc[lane + 32 * s] * sc;
                if (DENS || DW) pd[o] = pd[o] + waccw[lane + 32 * s];
            } else {
                const size_t E = split.edge, E3 = E * E * E;
                float *const pv = split.part + (size_t)(item % ns - 1) * (DENS || DW ? 2 : 1) * E3 +
                                  ((size_t)(bz + s - split.lo) * E + (ly - split.lo)) * E + (lx - split.lo);
                pv[0] = wacc[lane + 32 * s] * sc;
                if (DENS || DW) pv[E3] = waccw[lane + 32 * s];
            }
        }
        if (!split.next) return;
        // every item is fetched or started on once: the fetch that returns
        // items - 1 is the last, and leaves the counter at 0 for the next launch
        unsigned f = 0;
        if (lane == 0) {
            f = atomicAdd(split.next, 1u);
            if (f == (unsigned)items - 1) atomicExch(split.next, 0u);
        }
        item = (int)gridDim.x * NW + (int)__shfl_sync(0xffffffffu, f, 0);
    }
}

// Adds the segments' sums of a split launch to the volume (and the density),
// in segment order: (((v + s1) + s2) + ...).  Voxels of the mask sphere, which
// every segment has written; the grid covers the sphere's box.  Bound: HBM /
// L2, 4 (segments + 1) bytes a voxel.
__global__ void __launch_bounds__(256)
bp_merge_kernel(float *__restrict__ vol, float *__restrict__ pd, int V, int maskR, BpSplit split)
{
    const int x = blockIdx.x * 256 + threadIdx.x, y = blockIdx.y, z = blockIdx.z;
    if (x >= split.edge) return;
    const long long c = V / 2 - split.lo, dx = x - c, dy = y - c, dz = z - c;
    if (dx * dx + dy * dy + dz * dz > (long long)maskR * maskR) return;
    const size_t E = split.edge, E3 = E * E * E, q = ((size_t)z * E + y) * E + x;
    const size_t o = ((size_t)(z + split.lo) * V + (y + split.lo)) * V + (x + split.lo);
    const int per = pd ? 2 : 1;
    float v = vol[o], d = pd ? pd[o] : 0.0f;
    for (int s = 0; s + 1 < split.nseg; s++) {
        v = __fadd_rn(v, split.part[s * per * E3 + q]);
        if (pd) d = __fadd_rn(d, split.part[(s * per + 1) * E3 + q]);
    }
    vol[o] = v;
    if (pd) pd[o] = d;
}

template <bool DENS, bool DW, bool DEEP, int G>
static cudaError_t launch_bp_compact_g(float *vol, const float *img, const float *ker, const float *axes, int n,
                                       const Geom &g, const float *scale, cudaStream_t s, float *pd, const float *img2,
                                        int max_copies, BpSplit split)
{
    constexpr int kCBZ = BpShape<DW, DEEP>::BZ;
    const int bx = (g.V + kCBX - 1) / kCBX, by = (g.V + kCBY - 1) / kCBY, bz = (g.V + kCBZ - 1) / kCBZ;
    // one group per CTA (the serving lanes): the non-LEAN layout
    constexpr bool LEAN = G > 1;
    using Mem = BpWarpMem<DENS, DW, DEEP, LEAN>;
    constexpr int NW = kCThreads / 32 * G;
    const size_t other = NW * sizeof(Mem);
    // one group per CTA: three CTAs an SM (228 KB, 1 KB reserved per CTA)
    const size_t limit = G == 1 ? (size_t)(228 * 1024 / 3 - 1024) : 0;
    const BpTable tb = bp_table(g.ker_size, other, max_copies, limit);
    if (tb.copies == 0) return cudaErrorInvalidValue; // a KB table too long for shared memory
    const size_t dyn = (((size_t)tb.entries * tb.copies + 3) & ~(size_t)3) * sizeof(float) + other;
    // quad loads of image rows: 4 | M and the stacks aligned to 4 elements
    const size_t qa = 4 * sizeof(float);
    const int vec = (g.M % 4 == 0) && ((size_t)img % qa == 0) && (!img2 || (size_t)img2 % 16 == 0) ? 1 : 0;
    if (bz > kMaxLayers) return cudaErrorInvalidValue;
    BpLayers lay;
    lay.layers = bz;
    lay.pre[0] = 0;
    for (int r = 0; r < bz; r++) {
        int bricks = 0;
        for (int j = 0; j < by; j++) {
            int lo, cnt;
            brick_row(j, middle_out(r, bz), bx, (int)((float)g.V) / 2, kCBZ, g.mask_radius, lo, cnt);
            bricks += cnt;
        }
        lay.pre[r + 1] = lay.pre[r] + bricks;
    }
    const long long items = (long long)lay.pre[bz] * 8 * split.nseg;
    if (items == 0) return cudaSuccess;
    if (items > 0x40000000LL) return cudaErrorInvalidValue;
    long long grid = (items + NW - 1) / NW;
    if (split.next) grid = std::min<long long>(grid, num_sms()); // one CTA an SM
    // the table stride as a compile-time constant where the copy count gives one
    auto go = [&](auto kern) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
        if (e != cudaSuccess) return e;
        kern<<<(unsigned)grid, kCThreads * G, dyn, s>>>(vol, pd, g.V, img, g.M, axes, n, g.mask_radius, ker, g.ker_size,
                                              g.ker_hw, bx, by, tb, scale, img2, vec, split, lay);
        count_launches(1);
        if (split.nseg > 1) {
            const dim3 mg((unsigned)((split.edge + 255) / 256), (unsigned)split.edge, (unsigned)split.edge);
            bp_merge_kernel<<<mg, 256, 0, s>>>(vol, DENS || DW ? pd : nullptr, g.V, g.mask_radius, split);
            count_launches(1);
        }
        return cudaGetLastError();
    };
    if constexpr (LEAN) {
        if (split.nseg > 1) // bp_segments splits only tables that get 32 copies
            return tb.copies == 32 ? go(bp_ref_compact_kernel<DENS, DW, DEEP, G, 128, true, true>) : cudaErrorInvalidValue;
        if (tb.copies == 32) return go(bp_ref_compact_kernel<DENS, DW, DEEP, G, 128, true>);
    }
    return go(bp_ref_compact_kernel<DENS, DW, DEEP, G, 0, LEAN>);
}

template <bool DENS, bool DW = false, bool DEEP = false>
static cudaError_t launch_bp_compact_t(float *vol, const float *img, const float *ker, const float *axes, int n,
                                       const Geom &g, const float *scale, cudaStream_t s, float *pd = nullptr,
                                       const float *img2 = nullptr, bool shared = false,
                                       BpSplit split = BpSplit())
{
    if (n <= 0) return cudaSuccess;
    // A GPU shared with concurrent launches (the serving lanes): one group
    // and one table copy per CTA, three CTAs an SM, which the launches of
    // other lanes can fill as they free (serving capacity 172 -> 195 req/s when
    // the rule was made); alone, 24 warps sharing 32 table copies (batched back
    // projection 78.5 -> 71.7 ms per 10k images then, 51 now).
    if constexpr (!DENS && !DW) {
        if (shared)
            return launch_bp_compact_g<DENS, DW, DEEP, 1>(vol, img, ker, axes, n, g, scale, s, pd,
                                                                         img2, 1, BpSplit());
    }
    return launch_bp_compact_g<DENS, DW, DEEP, kGroupsOf<DW, DEEP>>(vol, img, ker, axes, n, g, scale, s, pd,
                                                                         img2, 32, split);
}

// Reference-rule launch with the block depth chosen by the image size.
template <bool DENS>
static cudaError_t launch_bp_ref_sized(float *vol, const float *img, const float *ker, const float *axes, int n,
                                       const Geom &g, const float *scale, cudaStream_t s, float *pd, bool shared,
                                       BpSplit split)
{
    if (g.M >= 512)
        return launch_bp_compact_t<DENS, false, true>(vol, img, ker, axes, n, g, scale, s, pd, nullptr,
                                                                 shared, split);
    return launch_bp_compact_t<DENS>(vol, img, ker, axes, n, g, scale, s, pd, nullptr, shared, split);
}

cudaError_t launch_back_project_ref(float *d_vol, const float *d_img, const float *d_ker, const float *d_axes, int n,
                                    const Geom &g, const float *scale, cudaStream_t s, bool shared, BpSplit split)
{
    return launch_bp_ref_sized<false>(d_vol, d_img, d_ker, d_axes, n, g, scale, s, nullptr, shared, split);
}

cudaError_t launch_back_project_ref_density(float *d_vol, float *d_pd, const float *d_img, const float *d_ker,
                                            const float *d_axes, int n, const Geom &g, const float *scale,
                                            cudaStream_t s, BpSplit split)
{
    return launch_bp_ref_sized<true>(d_vol, d_img, d_ker, d_axes, n, g, scale, s, d_pd, false, split);
}

cudaError_t launch_back_project_ref_pair(float *d_vol, float *d_pd, const float *d_img, const float *d_img2,
                                         const float *d_ker, const float *d_axes, int n, const Geom &g, cudaStream_t s,
                                         BpSplit split)
{
    return launch_bp_compact_t<false, true>(d_vol, d_img, d_ker, d_axes, n, g, nullptr, s, d_pd, d_img2,
                                                           false, split);
}

// How many segments.  Every direction reaches the blocks at the centre, so a
// centre block is a serial chain over all n of them while the others' work
// falls as 1 / radius; where a launch has few blocks (6,000 at M = 128 for
// 3,648 warps) that chain is the launch's time.  Segments cut it, but each pays
// a block's start and merge and fills rounds less well, so `want` bricks times
// segments suffice, the fewer the fewer the directions.  Measured,
// reconstructVol in us by segment count: M = 64, n = 1000: 3137 (1), 648 (8),
// 567 (12); M = 128, n = 1000: 3698 (1), 1669 (4), 1504 (6), 1539 (8), n = 256:
// 1011 (1), 533 (4), 537 (6), n = 64: 306 (1), 229 (3), 231 (4), n = 16: 130
// (1), 137 (2); M = 160, n = 1000: 4155 (1), 2386 (4), 2444 (6); M = 200,
// n = 1000: 5116 (1), 3703 (3), 3742 (4), n = 256: 1433 (1), 1162 (2), 1208
// (3); M = 256, n = 1000: 6164 (1), 5483 (2), 5541 (3), n = 256: 1734 (1), 1743
// (2); M = 320, n = 1000: 9276 (1), 9466 (2).
// The rule looks at n and the geometry only, so the plain, density and
// two-stack forms of one call add the same partial sums (the two-stack form
// alone would stay at 1 for M = 256: 5,885 against 6,056 us).
int bp_segments(int n, const Geom &g)
{
    if (g.ker_size > 513) return 1; // no room for the 32 table copies of the split form
    const double r = g.mask_radius + 2.0;
    const int bricks = (int)(4.19 * r * r * r / (kCBX * kCBY * 12)) + 1; // in the mask's sphere
    const int want = n < 32 ? 500 : n < 192 ? 2000 : n < 512 ? 3000 : 6000;
    const int most = n < 32 ? n / 4 : std::min(n / 10, 12);
    return std::max(1, std::min((want + bricks - 1) / bricks, most));
}

} // namespace gg
