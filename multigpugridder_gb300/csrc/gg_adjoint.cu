// Exact adjoint of the forward projection (sm_103a): every in-mask pixel adds
// its value, times the forward weights, to the 4^3 voxels of its window.
//
// A warp takes an 8x8 pixel tile of one direction.  The windows lie in a small
// box of the volume (2,044 elements on average) which the warp keeps in shared
// memory as its own: it adds the pixels' windows one after another, two
// 32-tap halves of a window at a time, and then adds the box's nonzero quads
// to the volume with vector reductions in L2.
//
// Why this split.  The adjoint used to gather: each voxel near a direction's
// plane summed a 7x7 pixel window, of which 22% carry weight, with three table
// lookups per pixel (about 150 warp instructions a pixel).  Scattered, the
// weights of a pixel are separable (12 lookups) and every product counts: 15
// warp instructions a pixel and 12.5 shared-memory wavefronts in all (ncu),
// which bound it: 4 its taps' reads and writes, 4 the broadcasts of its terms.
// The lanes of a half window are 4 x 4 x 2 taps: with a row pitch of 12 or 20
// words and a slice pitch of 16 mod 32 their addresses fall in 32 different
// banks from any start.  The box is private to the warp, so plain loads and
// stores suffice; the additions to the volume are the only atomics, and the
// order of a voxel's sum is that of their arrival.
// Measured: gradient step of 512 images at 128^3, 10,195 -> 3,420 us with this
// kernel in the gathering one's place (8,079 -> 1,854 us of it); with each
// lane's quads of the box placed once a tile and 13 warps for 12, 1,445 us.
#include <algorithm>

#include "gg_internal.h"
#include "gg_project.cuh"

namespace gg {

constexpr int kAdjTile = 8;
constexpr int kAdjWarps = 13;    // warps a CTA, one CTA an SM
constexpr int kAdjBox = 3600;    // floats of a warp's box (99.8% of random tiles need less, none more than 4,100)
constexpr int kAdjStage = 32 * 21; // staged pixels: 16 xy products, 4 z weights, the window's place
constexpr int kAdjRep = 4;       // interleaved table copies (1 where a long table leaves no room)

__device__ __forceinline__ float box_ld(unsigned a)
{
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void box_st(unsigned a, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v)); }

// VW: floats per addition to the volume (4: rows of 16 bytes; 2: even rows; 1).
template <int VW>
__device__ __forceinline__ void add_quad(float *p, float4 v, int left)
{
    if constexpr (VW == 4) {
        if (left >= 4 && (v.x != 0.0f || v.y != 0.0f || v.z != 0.0f || v.w != 0.0f))
            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                         : "memory");
    } else if constexpr (VW == 2) {
        if (left >= 2 && (v.x != 0.0f || v.y != 0.0f))
            asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(v.x), "f"(v.y) : "memory");
        if (left >= 4 && (v.z != 0.0f || v.w != 0.0f))
            asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p + 2), "f"(v.z), "f"(v.w) : "memory");
    } else {
        if (left >= 1 && v.x != 0.0f) atomicAdd(p, v.x);
        if (left >= 2 && v.y != 0.0f) atomicAdd(p + 1, v.y);
        if (left >= 3 && v.z != 0.0f) atomicAdd(p + 2, v.z);
        if (left >= 4 && v.w != 0.0f) atomicAdd(p + 3, v.w);
    }
}

// One pixel straight into the volume: windows that leave it (their taps inside
// it), and tiles whose box does not fit (axes far from orthonormal).
__device__ __noinline__ void pixel_to_global(float *__restrict__ vol, int V, int P, float fi, float fj, float fk, float y,
                                             const float *sker, int rep, float kerScale, float kerCenterHalf, int kerSize)
{
    const float li = floorf(fi), lj = floorf(fj), lk = floorf(fk);
    // no window of a coordinate this far (or not finite) meets the volume
    if (!(fabsf(fi) < 1e6f && fabsf(fj) < 1e6f && fabsf(fk) < 1e6f)) return;
    const int b0 = (int)li - 1, b1 = (int)lj - 1, b2 = (int)lk - 1;
#pragma unroll 1
    for (int u = 0; u < 64; u++) {
        const int x = b0 + (u & 3), yy = b1 + ((u >> 2) & 3), z = b2 + (u >> 4);
        if ((unsigned)x >= (unsigned)V || (unsigned)yy >= (unsigned)V || (unsigned)z >= (unsigned)V) continue;
        const float w = kb_weight(sker, (float)x - fi, kerScale, kerCenterHalf, kerSize, rep) *
                        kb_weight(sker, (float)yy - fj, kerScale, kerCenterHalf, kerSize, rep) *
                        kb_weight(sker, (float)z - fk, kerScale, kerCenterHalf, kerSize, rep);
        atomicAdd(vol + ((size_t)z * V + yy) * P + x, w * y);
    }
}

template <int VW>
__global__ void __launch_bounds__(kAdjWarps * 32, 1)
adjoint_tile_kernel(float *__restrict__ vol, int V, int P, const float *__restrict__ img, int M,
                    const float *__restrict__ axes, int maskR, const float *__restrict__ ker, int kerSize, float kerHW,
                    int tilesX, long long nItems, const float *__restrict__ d_scale, int rep)
{
    // [boxes][stages][table: kerSize entries x rep copies]
    extern __shared__ __align__(16) float adj_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float *const box = adj_smem + warp * kAdjBox;
    float *const stage = adj_smem + kAdjWarps * kAdjBox + warp * kAdjStage;
    float *const tab = adj_smem + kAdjWarps * (kAdjBox + kAdjStage);
    for (int t = threadIdx.x; t < kerSize * rep; t += blockDim.x) tab[t] = __ldg(ker + t / rep);
    for (int t = lane; t < kAdjBox / 4; t += 32) reinterpret_cast<float4 *>(box)[t] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    __syncthreads();
    const float *sker = tab + lane % rep;
    const unsigned tab_step = 4u * (unsigned)rep; // bytes between entries
    const unsigned box_addr = (unsigned)__cvta_generic_to_shared(box);
    const float scale = d_scale ? *d_scale : 1.0f;
    const int ic = M / 2, vc = V / 2;
    const long long R2 = (long long)maskR * maskR; // a caller's radius may be any int
    const float kerCenter = ((float)kerSize - 1) / 2, kerScale = kerCenter / kerHW, kerCenterHalf = kerCenter + 0.5f;
    const unsigned tab_base = (unsigned)__cvta_generic_to_shared(sker) - __float_as_uint(12582912.0f) * tab_step;
    const int per = tilesX * tilesX;
    const bool items32 = nItems <= 0x7fffffffLL;

    for (long long item = (long long)blockIdx.x * kAdjWarps + warp; item < nItems; item += (long long)gridDim.x * kAdjWarps) {
        const int a = items32 ? (int)((unsigned)item / (unsigned)per) : (int)(item / per);
        const int t = (int)(item - (long long)a * per), tj = t / tilesX;
        const int i0 = (t - tj * tilesX) * kAdjTile, j0 = tj * kAdjTile;
        {   // the tile's nearest pixel to the centre is outside the mask: none is inside
            const int dia = i0 - ic, dib = dia + kAdjTile - 1, dja = j0 - ic, djb = dja + kAdjTile - 1;
            const int ni = dia > 0 ? dia : dib < 0 ? dib : 0, nj = dja > 0 ? dja : djb < 0 ? djb : 0;
            if ((long long)ni * ni + (long long)nj * nj > R2) continue;
        }
        const float *ax = axes + 9 * (size_t)a;
        const float *im = img + (size_t)a * M * M;
        const float nx0 = __ldg(ax), nx1 = __ldg(ax + 1), nx2 = __ldg(ax + 2);
        const float ny0 = __ldg(ax + 3), ny1 = __ldg(ax + 4), ny2 = __ldg(ax + 5);

        // Each lane's two pixels, four rows apart.
        float f[2][3], val[2];
        bool on[2], in[2]; // in the mask; and its window inside the volume
        int lo[3] = {0x7fffffff, 0x7fffffff, 0x7fffffff}, hi[3] = {-0x7fffffff, -0x7fffffff, -0x7fffffff};
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int i = i0 + (lane & 7), j = j0 + (lane >> 3) + 4 * h, di = i - ic, dj = j - ic;
            on[h] = i < M && j < M && (long long)di * di + (long long)dj * dj <= R2;
            val[h] = on[h] ? ld_f32(im + (size_t)j * M + i) * scale : 0.0f;
            f[h][0] = sample_coord(nx0, ny0, di, dj, vc);
            f[h][1] = sample_coord(nx1, ny1, di, dj, vc);
            f[h][2] = sample_coord(nx2, ny2, di, dj, vc);
            in[h] = on[h];
#pragma unroll
            for (int d = 0; d < 3; d++) in[h] = in[h] && f[h][d] >= 1.0f && f[h][d] < (float)(V - 2); // false for NaN
            if (in[h]) {
#pragma unroll
                for (int d = 0; d < 3; d++) {
                    const int b = (int)floorf(f[h][d]) - 1;
                    lo[d] = min(lo[d], b);
                    hi[d] = max(hi[d], b);
                }
            }
        }
        bool boxed = __any_sync(0xffffffffu, in[0] || in[1]);
        int RP = 12, SP = 16, nz = 0, x0 = 0;
        if (boxed) {
#pragma unroll
            for (int d = 0; d < 3; d++) {
                lo[d] = __reduce_min_sync(0xffffffffu, lo[d]);
                hi[d] = __reduce_max_sync(0xffffffffu, hi[d]);
            }
            x0 = lo[0] & ~3;
            const int ex = hi[0] + 4 - x0, ey = hi[1] + 4 - lo[1];
            nz = hi[2] + 4 - lo[2];
            RP = ex <= 12 ? 12 : 20;
            SP = RP * ey;
            SP += (16 - SP) & 31; // 16 mod 32
            boxed = ex <= 20 && SP <= 384 && nz <= 32 && SP * nz <= kAdjBox; // 384: three quads a lane
        }

#pragma unroll
        for (int h = 0; h < 2; h++) {
            // stage the half tile's pixels, those in the box first to last
            const bool use = boxed && in[h];
            if (on[h] && !use) {
                pixel_to_global(vol, V, P, f[h][0], f[h][1], f[h][2], val[h], sker, rep, kerScale, kerCenterHalf, kerSize);
            }
            const unsigned who = __ballot_sync(0xffffffffu, use);
            __syncwarp(); // the previous half's staged pixels have been read
            if (use) {
                float *st = stage + 21 * __popc(who & ((1u << lane) - 1u));
                float w[3][4];
                int b[3];
#pragma unroll
                for (int d = 0; d < 3; d++) {
                    const float fl = floorf(f[h][d]);
                    b[d] = (int)fl - 1;
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        // kb_weight of r in (-2, 2]: floor as the low bits of a sum rounded down
                        const float r = __fsub_rn(__fadd_rn(fl, (float)(u - 1)), f[h][d]);
                        const unsigned e = __float_as_uint(__fadd_rd(__fmaf_rn(r, kerScale, kerCenterHalf), 12582912.0f));
                        asm("ld.shared.f32 %0, [%1];" : "=f"(w[d][u]) : "r"(tab_base + e * tab_step));
                    }
                }
#pragma unroll
                for (int u = 0; u < 16; u++) st[u] = w[0][u & 3] * w[1][u >> 2] * val[h];
#pragma unroll
                for (int u = 0; u < 4; u++) st[16 + u] = w[2][u];
                st[20] = __int_as_float(4 * ((b[2] - lo[2]) * SP + (b[1] - lo[1]) * RP + (b[0] - x0)));
            }
            __syncwarp();
            // Lane (x, y, z) = (l & 3, (l >> 2) & 3, l >> 4) adds taps z and z + 2.
            const int cnt = __popc(who);
            const unsigned mine = box_addr + 4u * ((lane & 3) + RP * ((lane >> 2) & 3) + SP * (lane >> 4));
            const unsigned step = 8u * SP;
            const float *const sxy = stage + (lane & 15), *const sz = stage + 16 + (lane >> 4);
            float xy = sxy[0], z0 = sz[0], z1 = sz[2];
            unsigned at = mine + __float_as_uint(stage[20]);
#pragma unroll 2
            for (int p = 0; p < cnt; p++) {
                // the next pixel's terms are read while this one's voxels are
                const int nx = 21 * min(p + 1, 31);
                const float nxy = sxy[nx], nz0 = sz[nx], nz1 = sz[nx + 2], nat = stage[nx + 20];
                const float v0 = box_ld(at), v1 = box_ld(at + step);
                box_st(at, fmaf(xy, z0, v0));
                box_st(at + step, fmaf(xy, z1, v1));
                xy = nxy;
                z0 = nz0;
                z1 = nz1;
                at = mine + __float_as_uint(nat);
                __syncwarp(); // the next window may share voxels, in other lanes
            }
        }

        // The box's nonzero quads to the volume; the box is zero again.  A lane
        // takes the same (at most three) quads of every slice, so their places
        // are worked out once.
        if (boxed) {
            const int rq = RP >> 2, sq = SP >> 2, ey = hi[1] + 4 - lo[1];
            float *slice = vol + ((size_t)lo[2] * V + lo[1]) * P + x0;
            int off[3], left[3];
#pragma unroll
            for (int u = 0; u < 3; u++) {
                const int q = lane + 32 * u, r = rq == 3 ? q / 3 : q / 5, c = 4 * (q - r * rq);
                off[u] = r * P + c;
                left[u] = r < ey ? (VW == 4 ? P : V) - (x0 + c) : 0;
            }
            float4 *bz = reinterpret_cast<float4 *>(box) + lane;
            for (int z = 0; z < nz; z++, slice += (size_t)V * P, bz += sq) {
#pragma unroll
                for (int u = 0; u < 3; u++) {
                    if (lane + 32 * u < sq) {
                        const float4 v = bz[32 * u];
                        bz[32 * u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                        add_quad<VW>(slice + off[u], v, left[u]);
                    }
                }
            }
        }
        __syncwarp();
    }
}

cudaError_t launch_back_project_adjoint(float *d_vol, int P, const float *d_img, const float *d_ker, const float *d_axes,
                                        int n, const Geom &g, const float *scale, cudaStream_t s)
{
    const int tilesX = (g.M + kAdjTile - 1) / kAdjTile;
    const long long nItems = (long long)n * tilesX * tilesX;
    if (nItems <= 0) return cudaSuccess;
    int dev = 0, sms = 0, optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    const size_t boxes = (size_t)kAdjWarps * (kAdjBox + kAdjStage) * sizeof(float);
    const int rep = boxes + (size_t)g.ker_size * kAdjRep * sizeof(float) <= (size_t)optin ? kAdjRep : 1;
    const size_t smem = boxes + (size_t)g.ker_size * rep * sizeof(float);
    const long long grid = std::min<long long>((nItems + kAdjWarps - 1) / kAdjWarps, std::max(sms, 1));
    // vector additions where every row of the volume starts aligned for them
    const size_t at = (size_t)d_vol;
    auto go = [&](auto kern) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        kern<<<(unsigned)grid, kAdjWarps * 32, smem, s>>>(d_vol, g.V, P, d_img, g.M, d_axes, g.mask_radius, d_ker,
                                                         g.ker_size, g.ker_hw, tilesX, nItems, scale, rep);
        count_launches(1);
        return cudaGetLastError();
    };
    if (P % 4 == 0 && at % 16 == 0) return go(adjoint_tile_kernel<4>);
    if (P % 2 == 0 && g.V % 2 == 0 && at % 8 == 0) return go(adjoint_tile_kernel<2>);
    return go(adjoint_tile_kernel<1>);
}

} // namespace gg
