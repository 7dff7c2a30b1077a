// Forward projection from volume boxes staged in shared memory (sm_103a).
//
// A CTA takes a 16x16 pixel tile of one direction.  The windows of its pixels
// lie in an axis-aligned box of the CAS volume, at most 32 x 29 x 26 elements
// for orthonormal axes; one thread copies that box to shared memory by TMA
// (3-D tiles of the pitched volume, 2 to 8 slices each) while all threads look
// up their 12 weights, and the 64 taps are then read from shared memory.
//
// Bound: shared-memory wavefronts.  A warp's 64 (FP32) or 48 (2-byte storage,
// element pairs) gathers cost as many wavefronts as lanes collide in a bank.
// Read straight from global memory through L1 they cost 6.9 cycles each (one
// per distinct 128-byte line; three transposed copies of the volume were kept
// to get there), from a box with a fixed slice pitch 3.0 and with the pitch
// and the warp's shape chosen per direction 2.2 (a CPU model over random
// directions).  fp_plan_kernel makes that choice.  Measured at M = 256: kernel
// for 1,024 directions 2,270 -> 1,452 us (ncu), shared-memory pipe 75% busy;
// whole call for 1,000 2,389 -> 1,638 us, images the same bit for bit (FP32).  The two transposed
// copies (175 us a volume at 128^3, 1,700 us of BF16 ones at 256^3) went away.
#include <cuda.h>

#include <algorithm>
#include <vector>

#include "gg_internal.h"
#include "gg_project.cuh"

namespace gg {

constexpr int kTile = 16;         // pixels along a tile's edge
constexpr int kTileThreads = 256; // one thread per pixel
constexpr int kTabRep = 4;        // interleaved table copies (fewer bank conflicts in the 12 lookups)
constexpr int kByMin = 4, kNBY = 29; // box heights with a tensor map: 4 .. 32
constexpr int kDepths = 4;           // and depths of one copy: 2, 4, 6, 8 slices
constexpr unsigned kWaitLimit = 1u << 22; // polls of a copy's barrier (far beyond a second)

template <typename TV> struct TileCfg {
    static constexpr int QA = 16 / (int)sizeof(TV);           // elements in 16 bytes: box x starts and widths
    static constexpr int BX0 = sizeof(TV) == 4 ? 8 : 16;      // smallest box width
    static constexpr int NBX = sizeof(TV) == 4 ? 7 : 4;       // widths BX0, BX0 + QA, ...: up to 32 / 40
    static constexpr int CAP = sizeof(TV) == 4 ? 14336 : 18432; // box elements (13,728 / 18,304 needed at most)
};

// The box of a direction: bx x by elements a slice, bz the most slices; tall:
// warps take 2 columns x 16 rows of the tile instead of 16 columns x 2 rows.
// bx = 0: no box fits (axes far from orthonormal); the tile reads global memory.
struct FpPlan {
    int bx, by, bz, tall;
};

// The box dimensions a direction needs at least; false: none fits.  Along an
// axis the tile's coordinates span 15 (|X| + |Y|), and a window takes 4.
template <typename TV>
__device__ __forceinline__ bool box_needs(const float *__restrict__ ax, int &bx, int &by, int &bz)
{
    using C = TileCfg<TV>;
    int need[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const float s = (kTile - 1) * (fabsf(__ldg(ax + d)) + fabsf(__ldg(ax + 3 + d)));
        if (!(s < 64.0f)) return false; // NaN too
        need[d] = (int)ceilf(s + 1e-3f) + 4;
    }
    bx = max((need[0] + 2 * C::QA - 2) / C::QA * C::QA, C::BX0);
    by = max(need[1], kByMin);
    bz = (need[2] + 1) & ~1;
    return bx < C::BX0 + C::NBX * C::QA && by < kByMin + kNBY && bx * by * bz <= C::CAP;
}

// The plan without the search: the least height, and the warp shape that runs
// along x.  For launches of few tiles, where the search's own launch costs
// more than its pitch saves (16 directions at M = 128: 26.4 us a call against
// 33.5 with the search).
template <typename TV>
__device__ __forceinline__ FpPlan quick_plan(const float *__restrict__ ax)
{
    FpPlan p{0, 0, 0, 0};
    int bx, by, bz;
    if (box_needs<TV>(ax, bx, by, bz)) p = FpPlan{bx, by, bz, 0};
    p.tall = fabsf(__ldg(ax + 3)) > fabsf(__ldg(ax)) ? 1 : 0;
    return p;
}

// One warp per direction: of the box heights need .. need + 3 and the two
// warp shapes, the pair with the fewest bank conflicts over three sample
// positions.  (The slice pitch bx * by mod 32 is what matters; wider choices
// gain nothing in the CPU model: 2.28 with 8 heights against 2.22.)
template <typename TV>
__global__ void fp_plan_kernel(const float *__restrict__ axes, int n, FpPlan *__restrict__ plans)
{
    using C = TileCfg<TV>;
    const int lane = threadIdx.x & 31, a = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (a >= n) return;
    const float *ax = axes + 9 * (size_t)a;
    const float X[3] = {__ldg(ax), __ldg(ax + 1), __ldg(ax + 2)}, Y[3] = {__ldg(ax + 3), __ldg(ax + 4), __ldg(ax + 5)};
    int bx, by0, bz;
    const bool fits = box_needs<TV>(ax, bx, by0, bz);
    int best = 0x7fffffff;
    constexpr int SH = sizeof(TV) == 4 ? 0 : 1; // words of shared memory: element pairs for 2-byte storage
    const float off[3][3] = {{0.3f, 0.6f, 0.1f}, {0.7f, 0.2f, 0.5f}, {0.05f, 0.9f, 0.8f}};
#pragma unroll 1
    for (int c = 0; c < 8; c++) {
        const int tall = c & 1, by = by0 + (c >> 1);
        if (!fits || by >= kByMin + kNBY || bx * by * bz > C::CAP) continue; // uniform
        const float li = (float)(tall ? lane >> 4 : lane & 15), lj = (float)(tall ? lane & 15 : lane >> 4);
        int cost = 0;
#pragma unroll
        for (int s = 0; s < 3; s++) {
            int p[3];
#pragma unroll
            for (int d = 0; d < 3; d++) p[d] = (int)floorf(off[s][d] + li * X[d] + lj * Y[d]);
            const int word = (p[0] >> SH) + (bx >> SH) * p[1] + ((bx * by) >> SH) * p[2];
            const unsigned same = __match_any_sync(0xffffffffu, word);
            const bool first = (same & ((1u << lane) - 1u)) == 0; // lanes on one word share its wavefront
            const unsigned bank = __match_any_sync(0xffffffffu, first ? word & 31 : 32 + lane);
            cost += __reduce_max_sync(0xffffffffu, first ? __popc(bank) : 0);
        }
        best = min(best, cost * 8 + c);
    }
    if (lane == 0) {
        FpPlan p{0, 0, 0, 0};
        if (best != 0x7fffffff) p = FpPlan{bx, by0 + ((best & 7) >> 1), bz, best & 1};
        plans[a] = p;
    }
}

__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity)
{
    for (unsigned k = 0; k < kWaitLimit; k++) {
        unsigned done;
        asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
                     : "=r"(done)
                     : "r"(bar), "r"(parity)
                     : "memory");
        if (done) return true;
    }
    return false;
}

// Four taps of a row from the box, row start e (an element index).  FP32: the
// taps one by one.  2-byte storage: the two (even starts) or three element
// pairs that hold them, the x weights w6 placed at their offsets (the extra
// terms are exact zeros for a finite volume).
__device__ __forceinline__ float row_sum(const float *box, int e, const float (&w)[4])
{
    float s = 0.0f;
#pragma unroll
    for (int d = 0; d < 4; d++) s = fmaf(w[d], box[e + d], s);
    return s;
}
__device__ __forceinline__ float2 widen2(unsigned u, const __half *)
{
    return __half22float2(*reinterpret_cast<const __half2 *>(&u));
}
__device__ __forceinline__ float2 widen2(unsigned u, const __nv_bfloat16 *)
{
    return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xFFFF0000u));
}
template <typename T>
__device__ __forceinline__ float row_sum(const T *box, int pair, bool odd, const float (&w)[6])
{
    const unsigned *p = reinterpret_cast<const unsigned *>(box) + pair;
    float s = 0.0f;
#pragma unroll
    for (int q = 0; q < 3; q++) {
        const float2 v = widen2(q < 2 || odd ? p[q] : 0u, (const T *)nullptr);
        s = fmaf(w[2 * q], v.x, s);
        s = fmaf(w[2 * q + 1], v.y, s);
    }
    return s;
}

// The KB table in shared memory: kTabRep interleaved copies, a lane reads its own.
struct TileTable {
    const float *entry; // entry k at entry[k * kTabRep]
    unsigned base;      // its shared address, less the bits of 1.5 * 2^23 times the stride
    float scale, half;  // the entry of distance r is floor(fma(r, scale, half))
    int size;
};

// The weights of the four taps around f (fl = floor(f), f finite): kb_weight of
// r = fl - 1 + d - f in (-2, 2], the floor taken as the low bits of the sum
// with 1.5 * 2^23 rounded down, so no conversion and no clamp.
__device__ __forceinline__ void tap_weights(const TileTable &t, float f, float fl, float (&w)[4])
{
#pragma unroll
    for (int d = 0; d < 4; d++) {
        const float r = __fsub_rn(__fadd_rn(fl, (float)(d - 1)), f);
        const unsigned e = __float_as_uint(__fadd_rd(__fmaf_rn(r, t.scale, t.half), 12582912.0f));
        asm("ld.shared.f32 %0, [%1];" : "=f"(w[d]) : "r"(t.base + e * (4u * kTabRep)));
    }
}

// A window inside the volume, read from global memory, for tiles without a box
// (axes longer than one by 2% or more begin to miss it); p: its
// first tap, rows P and planes PV elements apart.  Out of line, as the next one:
// neither takes registers from the box's path.  Both have the 12 weights at hand
// and their taps unrolled: 1,000 CAS images at M = 256 from axes 1.2 times as
// long, 2,903 us (6,275 with the weights looked up again at every tap; 3,646
// when every pixel was read from transposed copies of the volume), 1.05 times
// 1,591 (1,831; 2,324), 1.8 times 6,729 (14,486; 10,027).
template <typename TV>
__device__ __noinline__ float window_from_global(const TV *__restrict__ p, int P, size_t PV, float4 wi, float4 wj, float4 wk)
{
    const float w[3][4] = {{wi.x, wi.y, wi.z, wi.w}, {wj.x, wj.y, wj.z, wj.w}, {wk.x, wk.y, wk.z, wk.w}};
    float acc = 0.0f;
#pragma unroll
    for (int dk = 0; dk < 4; dk++)
#pragma unroll
        for (int dj = 0; dj < 4; dj++) {
            float s = 0.0f;
#pragma unroll
            for (int d = 0; d < 4; d++) s = fmaf(w[0][d], ld_f32(p + dk * PV + (size_t)dj * P + d), s);
            acc = fmaf(w[1][dj] * w[2][dk], s, acc);
        }
    return acc;
}

// A window that leaves the volume, any axes: the reference's linear-index test
// on the dense layout (gpuForwardProject.cu:90), plus a lower bound.  A tap's
// index is row * V + column, its column within a row of the dense layout.
template <typename TV>
__device__ __noinline__ float window_at_edge(const TV *__restrict__ vol, int V, int P, float fi, float fj, float fk,
                                             TileTable t)
{
    const int b0 = (int)floorf(fi) - 1, b1 = (int)floorf(fj) - 1, b2 = (int)floorf(fk) - 1;
    const long long VV = (long long)V * V;
    long long row = (long long)b2 * V + b1, q = 0;
    if (b0 < 0 || b0 >= V) {
        q = b0 / V;
        if (q * V > b0) q--; // towards minus infinity
        row += q;
    }
    const int col = (int)(b0 - q * V);
    // the rows of the window's first tap and, at least, of its last
    if (row + 3 * (long long)V + 3 + (col + 3) / V < 0 || row >= VV) return 0.0f;
    float w[3][4];
#pragma unroll
    for (int d = 0; d < 4; d++) {
        w[0][d] = kb_weight(t.entry, (float)(b0 + d) - fi, t.scale, t.half, t.size, kTabRep);
        w[1][d] = kb_weight(t.entry, (float)(b1 + d) - fj, t.scale, t.half, t.size, kTabRep);
        w[2][d] = kb_weight(t.entry, (float)(b2 + d) - fk, t.scale, t.half, t.size, kTabRep);
    }
    float acc = 0.0f;
#pragma unroll
    for (int dk = 0; dk < 4; dk++)
#pragma unroll
        for (int dj = 0; dj < 4; dj++)
#pragma unroll
            for (int d = 0; d < 4; d++) {
                long long r = row + (long long)dk * V + dj;
                int c = col + d;
                while (c >= V) {
                    c -= V;
                    r++;
                }
                if (r >= 0 && r < VV) acc = fmaf(w[0][d] * w[1][dj] * w[2][dk], ld_f32(vol + r * P + c), acc);
            }
    return acc;
}

// A work item: a direction and a tile of its image (first pixel i0, j0), with
// the tile's range of pixel offsets from the image centre.
struct TileAt {
    int a, i0, j0, dia, dib, dja, djb;
};
__device__ __forceinline__ TileAt tile_at(long long item, int tilesX, bool items32, int M)
{
    const int per = tilesX * tilesX;
    const int a = items32 ? (int)((unsigned)item / (unsigned)per) : (int)(item / per);
    const int t = (int)(item - (long long)a * per), tj = t / tilesX;
    const int i0 = (t - tj * tilesX) * kTile, j0 = tj * kTile, ic = M / 2;
    return TileAt{a, i0, j0, i0 - ic, min(i0 + kTile, M) - 1 - ic, j0 - ic, min(j0 + kTile, M) - 1 - ic};
}
// Whether any pixel of the tile is in the mask (the nearest one to the centre
// is).  32-bit: a handle's radius is at most M, and M^2 stays below 2^31 for any
// volume that fits the GPU.
__device__ __forceinline__ bool tile_live(const TileAt &t, int R2)
{
    const int ni = t.dia > 0 ? t.dia : t.dib < 0 ? t.dib : 0, nj = t.dja > 0 ? t.dja : t.djb < 0 ? t.djb : 0;
    return ni * ni + nj * nj <= R2;
}

// What a tile's threads need of its box; bx = 0: no box.
struct TileBox {
    int x0, y0, z0, nz, bx, by, pad[2];
};

// The box of a tile's windows.  sample_coord is monotone in di and in dj (its
// products and sums round monotonically), so the corners bound every pixel's
// coordinates exactly.
template <typename TV>
__device__ __forceinline__ TileBox tile_box(const TileAt &t, const float *__restrict__ axes,
                                            const FpPlan *__restrict__ plans, int vc)
{
    const float *ax = axes + 9 * (size_t)t.a;
    const FpPlan pl = plans ? plans[t.a] : quick_plan<TV>(ax);
    int lo[3], hi[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const float nx = __ldg(ax + d), ny = __ldg(ax + 3 + d);
        const float c0 = sample_coord(nx, ny, nx < 0 ? t.dib : t.dia, ny < 0 ? t.djb : t.dja, vc);
        const float c1 = sample_coord(nx, ny, nx < 0 ? t.dia : t.dib, ny < 0 ? t.dja : t.djb, vc);
        lo[d] = (int)floorf(c0) - 1;
        hi[d] = (int)floorf(c1) + 2;
    }
    TileBox b;
    b.x0 = lo[0] & ~(TileCfg<TV>::QA - 1);
    b.y0 = lo[1];
    b.z0 = lo[2];
    b.nz = (hi[2] - lo[2] + 2) & ~1;
    const bool fits = pl.bx > 0 && hi[0] - b.x0 < pl.bx && hi[1] - b.y0 < pl.by && b.nz <= pl.bz;
    b.bx = fits ? pl.bx : 0;
    b.by = pl.by;
    return b;
}

template <typename TV>
__global__ void __launch_bounds__(kTileThreads, 3)
fp_tile_kernel(const TV *__restrict__ vol, int V, int P, const CUtensorMap *__restrict__ maps,
               const FpPlan *__restrict__ plans, float *__restrict__ img, int M, const float *__restrict__ axes,
               int maskR, const float *__restrict__ ker, int kerSize, float kerHW, int tilesX, long long nItems,
               const float *__restrict__ d_scale, int *__restrict__ fault)
{
    using C = TileCfg<TV>;
    // [box][barrier, pad][the box's place][table: kerSize entries x kTabRep copies]
    extern __shared__ __align__(128) unsigned char fp_smem[];
    TV *const box = reinterpret_cast<TV *>(fp_smem);
    unsigned char *const rest = fp_smem + C::CAP * sizeof(TV);
    TileBox *const place = reinterpret_cast<TileBox *>(rest + 16);
    float *const tab = reinterpret_cast<float *>(rest + 16 + sizeof(TileBox));
    const unsigned bar = smem_addr(rest), box_addr = smem_addr(box);
    for (int t = threadIdx.x; t < kerSize * kTabRep; t += kTileThreads) tab[t] = __ldg(ker + t / kTabRep);
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();

    const float outScale = d_scale ? *d_scale : 1.0f;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ic = M / 2, vc = V / 2, R2 = maskR * maskR;
    const float kerCenter = ((float)kerSize - 1) / 2;
    TileTable table;
    table.entry = tab + lane % kTabRep;
    table.base = smem_addr(table.entry) - __float_as_uint(12582912.0f) * (4u * kTabRep);
    table.scale = kerCenter / kerHW;
    table.half = kerCenter + 0.5f;
    table.size = kerSize;
    const bool items32 = nItems <= 0x7fffffffLL; // 32-bit division per item whenever it fits

    // Thread 0 announces a tile's box: its place to the other threads and the
    // bytes to the barrier, then starts the copies (8 slices each, the last 2
    // to 8).  A tile without a box completes the barrier by the arrival alone.
    auto start_box = [&](const TileBox &b) {
        *place = b;
        if (b.bx == 0) {
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
            return;
        }
        const int SP = b.bx * b.by;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                     "r"((unsigned)(SP * b.nz * (int)sizeof(TV)))
                     : "memory");
        const CUtensorMap *m = maps + (((b.bx - C::BX0) / C::QA) * kNBY + (b.by - kByMin)) * kDepths;
        for (int z = 0; z < b.nz; z += 8) {
            const int dep = min(b.nz - z, 8);
            asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, "
                         "%5}], [%2];" ::"r"(box_addr + (unsigned)(z * SP * (int)sizeof(TV))),
                         "l"(m + dep / 2 - 1), "r"(bar), "r"(b.x0), "r"(b.y0), "r"(b.z0 + z)
                         : "memory");
        }
    };
    // The CTA's next item whose tile meets the mask; the pixels of those
    // passed over are zeroed.
    auto next_live = [&](long long item, TileAt &t) {
        for (; item < nItems; item += gridDim.x) {
            t = tile_at(item, tilesX, items32, M);
            if (tile_live(t, R2)) break;
            const int i = t.i0 + (threadIdx.x & 15), j = t.j0 + (threadIdx.x >> 4);
            if (i < M && j < M) img[((size_t)t.a * M + j) * M + i] = 0.0f;
        }
        return item;
    };

    TileAt at{};
    long long item = next_live(blockIdx.x, at);
    if (item < nItems && threadIdx.x == 0) start_box(tile_box<TV>(at, axes, plans, vc));
    for (unsigned phase = 0; item < nItems; phase ^= 1) {
        const float *ax = axes + 9 * (size_t)at.a;
        const bool tall = plans ? __ldg(&plans[at.a].tall) != 0 : fabsf(__ldg(ax + 3)) > fabsf(__ldg(ax));
        const int lx = tall ? 2 * warp + (lane >> 4) : lane & 15, ly = tall ? lane & 15 : 2 * warp + (lane >> 4);
        const int i = at.i0 + lx, j = at.j0 + ly, di = i - ic, dj = j - ic;
        const float fi = sample_coord(__ldg(ax), __ldg(ax + 3), di, dj, vc);
        const float fj = sample_coord(__ldg(ax + 1), __ldg(ax + 4), di, dj, vc);
        const float fk = sample_coord(__ldg(ax + 2), __ldg(ax + 5), di, dj, vc);
        const float li = floorf(fi), lj = floorf(fj), lk = floorf(fk);
        const bool on = i < M && j < M && di * di + dj * dj <= R2;
        const int b0 = (int)li - 1, b1 = (int)lj - 1, b2 = (int)lk - 1;
        const bool inside = b0 >= 0 && b1 >= 0 && b2 >= 0 && b0 <= V - 4 && b1 <= V - 4 && b2 <= V - 4;
        float wi[4], wj[4], wk[4];
        if (on && inside) { // finite coordinates
            tap_weights(table, fi, li, wi);
            tap_weights(table, fj, lj, wj);
            tap_weights(table, fk, lk, wk);
        }
        float *const out = img + ((size_t)at.a * M + j) * M + i;

        // the next tile, and its box by thread 0 while this one's arrives
        const long long next = next_live(item + gridDim.x, at);
        TileBox nb{};
        if (threadIdx.x == 0 && next < nItems) nb = tile_box<TV>(at, axes, plans, vc);

        if (!mbar_wait(bar, phase)) {
            // the copies did not arrive: report it and leave, after one more
            // wait for those in flight
            *fault = 1;
            mbar_wait(bar, phase);
            return;
        }
        const int4 pl0 = *reinterpret_cast<const int4 *>(place); // x0, y0, z0, nz
        const int RP = place->bx, SP = RP * place->by;
        float acc = 0.0f;
        if (RP > 0 && on && inside) {
            const int e0 = (b2 - pl0.z) * SP + (b1 - pl0.y) * RP + (b0 - pl0.x);
            if constexpr (sizeof(TV) == 4) {
#pragma unroll
                for (int dk = 0; dk < 4; dk++)
#pragma unroll
                    for (int dj2 = 0; dj2 < 4; dj2++)
                        acc = fmaf(wj[dj2] * wk[dk], row_sum(box, e0 + dk * SP + dj2 * RP, wi), acc);
            } else {
                const bool odd = e0 & 1;
                const float w6[6] = {odd ? 0.0f : wi[0], odd ? wi[0] : wi[1], odd ? wi[1] : wi[2],
                                     odd ? wi[2] : wi[3], odd ? wi[3] : 0.0f, 0.0f};
#pragma unroll
                for (int dk = 0; dk < 4; dk++)
#pragma unroll
                    for (int dj2 = 0; dj2 < 4; dj2++)
                        acc = fmaf(wj[dj2] * wk[dk], row_sum(box, (e0 >> 1) + dk * (SP >> 1) + dj2 * (RP >> 1), odd, w6),
                                   acc);
            }
        } else if (on && inside) {
            acc = window_from_global(vol + ((size_t)b2 * V + b1) * P + b0, P, (size_t)P * V,
                                     make_float4(wi[0], wi[1], wi[2], wi[3]), make_float4(wj[0], wj[1], wj[2], wj[3]),
                                     make_float4(wk[0], wk[1], wk[2], wk[3]));
        } else if (on) {
            acc = window_at_edge(vol, V, P, fi, fj, fk, table);
        }
        __syncthreads(); // the box is free for the next tile
        if (threadIdx.x == 0 && next < nItems) start_box(nb);
        if (i < M && j < M) *out = acc * outScale;
        item = next;
    }
}

// ---- host side -----------------------------------------------------------------

size_t fp_tile_map_bytes(int prec)
{
    return (size_t)(prec == kF32 ? TileCfg<float>::NBX : TileCfg<__half>::NBX) * kNBY * kDepths * sizeof(CUtensorMap);
}

size_t fp_plan_bytes(int n) { return (size_t)(n > 0 ? n : 1) * sizeof(FpPlan); }

template <typename TV>
static cudaError_t encode_maps(const void *d_vol, int V, int P, CUtensorMapDataType type, CUtensorMap *out)
{
    using C = TileCfg<TV>;
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    cudaError_t e = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q);
    if (e != cudaSuccess) return e;
    if (q != cudaDriverEntryPointSuccess || !fn) return cudaErrorNotSupported;
    auto encode = reinterpret_cast<decltype(&cuTensorMapEncodeTiled)>(fn);
    const cuuint64_t dims[3] = {(cuuint64_t)P, (cuuint64_t)V, (cuuint64_t)V};
    const cuuint64_t strides[2] = {(cuuint64_t)P * sizeof(TV), (cuuint64_t)P * V * sizeof(TV)};
    const cuuint32_t one[3] = {1, 1, 1};
    for (int bx = 0; bx < C::NBX; bx++)
        for (int by = 0; by < kNBY; by++)
            for (int d = 0; d < kDepths; d++) {
                const cuuint32_t box[3] = {(cuuint32_t)(C::BX0 + bx * C::QA), (cuuint32_t)(kByMin + by),
                                           (cuuint32_t)(2 * d + 2)};
                const CUresult r = encode(&out[(bx * kNBY + by) * kDepths + d], type, 3, const_cast<void *>(d_vol), dims,
                                          strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                          CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
                if (r != CUDA_SUCCESS) return cudaErrorInvalidValue;
            }
    return cudaSuccess;
}

// Orders the maps' bytes, written by a copy, before every later launch that
// reads them through the tensor-map proxy: the address may have held another
// handle's maps.  Once a buffer, so that no launch pays for it (a fence for
// every map at the projection's own start: 26 -> 72 us for 16 directions); by
// one block, which every later launch comes after (10 us of a handle's first
// projection; a block an SM 30).
__global__ void __launch_bounds__(1024) fence_maps_kernel(const CUtensorMap *__restrict__ maps, int n)
{
    for (int t = threadIdx.x; t < n; t += blockDim.x)
        asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(maps + t) : "memory");
}

cudaError_t fp_tile_make_maps(const void *d_vol, int V, int P, int prec, void *d_maps, cudaStream_t s)
{
    std::vector<CUtensorMap> m(fp_tile_map_bytes(prec) / sizeof(CUtensorMap));
    cudaError_t e = prec == kF32 ? encode_maps<float>(d_vol, V, P, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, m.data())
                                 : encode_maps<__half>(d_vol, V, P, CU_TENSOR_MAP_DATA_TYPE_UINT16, m.data()); // FP16 and BF16
    if (e != cudaSuccess) return e;
    // on the stream and waited for: a copy from pageable memory may otherwise
    // still be under way when it returns, and streams of other lanes do not
    // wait for it
    e = cudaMemcpyAsync(d_maps, m.data(), m.size() * sizeof(CUtensorMap), cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return e;
    fence_maps_kernel<<<1, 1024, 0, s>>>((const CUtensorMap *)d_maps, (int)m.size());
    count_launches(1);
    e = cudaGetLastError();
    return e != cudaSuccess ? e : cudaStreamSynchronize(s);
}

template <typename TV>
static cudaError_t launch_tile_t(const FpTiles &v, float *d_img, const float *d_ker, const float *d_axes, int n,
                                 const Geom &g, const float *scale, cudaStream_t s, void *d_plans)
{
    const int tilesX = (g.M + kTile - 1) / kTile;
    const long long nItems = (long long)n * tilesX * tilesX;
    if (nItems == 0) return cudaSuccess;
    const size_t smem = TileCfg<TV>::CAP * sizeof(TV) + 16 + sizeof(TileBox) + (size_t)g.ker_size * kTabRep * sizeof(float);
    auto kern = fp_tile_kernel<TV>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int perSm = 0, dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, kern, kTileThreads, smem);
    const long long grid = std::min<long long>(nItems, (long long)std::max(sms, 1) * std::max(perSm, 1));
    // up to four tiles a CTA go without the search for a pitch
    FpPlan *const plans = nItems > 4 * grid ? (FpPlan *)d_plans : nullptr;
    if (plans) {
        fp_plan_kernel<TV><<<(n + 3) / 4, 128, 0, s>>>(d_axes, n, plans);
        count_launches(1);
    }
    kern<<<(unsigned)grid, kTileThreads, smem, s>>>((const TV *)v.vol, g.V, v.pitch, (const CUtensorMap *)v.maps, plans,
                                                    d_img, g.M, d_axes, g.mask_radius, d_ker, g.ker_size, g.ker_hw,
                                                    tilesX, nItems, scale, v.fault);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_forward_project_tiled(const FpTiles &v, float *d_img, const float *d_ker, const float *d_axes, int n,
                                         const Geom &g, const float *scale, cudaStream_t s, void *d_plans)
{
    if (v.prec == kF32) return launch_tile_t<float>(v, d_img, d_ker, d_axes, n, g, scale, s, d_plans);
    if (v.prec == kF16) return launch_tile_t<__half>(v, d_img, d_ker, d_axes, n, g, scale, s, d_plans);
    return launch_tile_t<__nv_bfloat16>(v, d_img, d_ker, d_axes, n, g, scale, s, d_plans);
}

} // namespace gg
