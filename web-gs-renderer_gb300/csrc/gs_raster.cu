// gs_raster.cu -- front-to-back alpha-blending tile rasterizer (src/shaders/raseter.wgsl:35-117).
//
// One thread per pixel; each warp owns an 8x4 block of a tile, a CTA up to 16x16 pixels (a 32x32 tile
// takes four). Every pixel blends the splats of the tile's sorted range in order with the pinned fp32
// semantics:
//   power = fma(-0.5, fma(a*dx, dx, (c*dy)*dy), -((b*dx)*dy)); skip if power > 0
//   alpha = min(0.99, o * exp(power));                         skip if alpha < 1/255
//   testT = T * (1 - alpha);                                   done if testT < 1e-4
//   C += colour * alpha * T (one fma per channel); T = testT
//
// Stage and cull. The CTA takes the range in steps (4 x raster_batch positions, at most 512, one vote per
// step to stop once every pixel is done, raseter.wgsl:54-68): one lane per splat tests the octagon around the
// region where power >= c_o = ln((1/255)/o) - 1e-3 can hold (its half extents come with the record,
// gs_raster_common.cuh) against the CTA's blocks, sends the record to shared memory by asynchronous copies
// if it meets any, and ballots turn the answers into one word per warp and 32 positions. A splat outside a
// block would have been rejected by each of its pixels, so walking only the hits changes no output bit.
// Contributor counts are range positions, so skipping does not change them.
//
// Walk. From there a warp is on its own until the next step: it lists its hits, a lane each lays 32 of
// them out as pairs, and the arithmetic up to the blend (power, exp, alpha, 1 - alpha, colour times alpha)
// runs on two splats at once by packed fp32 operations, which round each half like the scalar ones; only
// the blend itself goes splat by splat, by predicated instructions. Below a power of -20 alpha is formed at
// -20, where every opacity's is under 1/255, so the cut-off need not travel with the hit.
//
// What bounds it: where lists are long, shared-memory reads of the hits' nine values (a 16-byte read
// returns 512 bytes to a warp, four cycles of the SM's 128 bytes), 53% of the time at 1M / 1080p, the fp32
// pipe 56%, issue 72%; where they are short (a dozen splats a tile at 1080p) the chain of loads, tile, index,
// record, that each CTA goes through. So the tile comes with its range (k_tile_place), a record is read once
// per tile, and 40 warps fit an SM (46 to 48 registers, of which the plain 16x16 frame spills one; 34 KB per
// CTA; 48 warps at 8x8 tiles, whose 40 registers spill 16 to 20 bytes). With 32 / 40 / 48 warps: 1M / 1080p
// 306 / 299 / 310 us a frame, 12 views of 300k in 32x32 tiles 745 / 710 / 738, 16 sparse views of 35k at 1080p
// 370 / 339 / 340; steps of 256 cost 1M / 1080p 2%, of 768 gain nothing.
//
// Measured against one CTA per tile that staged 256 splats between two barriers, computed the octagon per
// tile and splat and walked the bits of its ballots at one splat per step (32 registers, 2048 threads per
// SM): 1M / 1080p 189.5 -> 162.4 us (216M -> 143M warp instructions), 3M / 4K 1168 -> 930, 250k / 1237x823 in
// 8x8 tiles 105 -> 70, a close-up of 60k at 1600x900 212 -> 176, 16 views in 32x32 tiles 3906 -> 2167 in
// sum, 50k / 512x512 47.6 -> 41.7, the sixteen sparse views 341 -> 344. Other ways to bring the records
// in: all of a step's, hit or not, 178.3, 1024, 75.3, 182, 2495, 42.7 and 346 us (a list takes its splats by their
// bounding squares, so many of them meet no block); a ring of hits per warp, filled while the hits
// before are blended, between culling steps of 1024, 181.5, 1030, 72.4, 187, 2445, 39.5 and 404 (a record is
// read once per warp that it hits). On the way there, 1M / 1080p: the pairs alone 211 us (3 selects per
// blend instead of predicates, octagons per tile, a barrier per 256 positions), predicates and steps of
// 1024 200, without the cut-off's reads 195.5, half extents from the preprocess and up to 32 hits per step
// 181.8; the packed constants read from constant memory 191.
//
// Tiles start in order[]'s order: by decreasing range length, so the longest tiles
// start first instead of forming the tail of the launch (with tiles in index order the clustered
// scenes left about a third of the launch time to a few long tiles).
#include <algorithm>

#include "gs_kernels.h"
#include "gs_raster_common.cuh"

namespace gs {
namespace {

// Bits of the warps whose 8x4 block of the SUB x SUB pixels at (px0, py0) the octagon of a splat at (x, y)
// with the half extents e (gs_raster_common.cuh) meets; all of them where no bound exists.
template <int SUB>
__device__ __forceinline__ uint32_t block_bits(float x, float y, const float4& e, float px0, float py0) {
    constexpr int WX = SUB / 8, WY = SUB / 4;
    const float x0 = x - e.x, x1 = x + e.x, y0 = y - e.y, y1 = y + e.y;
    const float u = x + y, v = x - y, u0 = u - e.z, u1 = u + e.z, v0 = v - e.w, v1 = v + e.w;
    uint32_t bits = 0;
#pragma unroll
    for (int by = 0; by < WY; ++by)
#pragma unroll
        for (int bx = 0; bx < WX; ++bx) {
            const float rx0 = px0 + 8.0f * bx, rx1 = rx0 + 7.0f, ry0 = py0 + 4.0f * by, ry1 = ry0 + 3.0f;
            const bool meets = (x1 >= rx0) & (x0 <= rx1) & (y1 >= ry0) & (y0 <= ry1) & (u1 >= rx0 + ry0) &
                               (u0 <= rx1 + ry1) & (v1 >= rx0 - ry1) & (v0 <= rx1 - ry0);
            bits |= meets ? 1u << (by * WX + bx) : 0u;
        }
    return e.x < __int_as_float(0x7f800000) ? bits : (1u << (WX * WY)) - 1u;
}

constexpr uint32_t kChunk = 32;   // most hits blended at a time (one lane each lays them out in pairs)
constexpr uint32_t kList = 64;    // hits waiting per warp (room for 32 more at kChunk - 1 pending)

// Shared memory of a warp: its next hits (positions in the step) and the chunk's hits as pairs.
struct RasterWarp {
    float4 pair[kChunk / 2][5];  // (x, x', y, y'), (A, A', -B, -B'), (C, C', o, o'), (r, r', g, g'),
                                 // (b, b', position, position')
    uint32_t list[kList];
};
template <int TILE>
struct RasterShared {
    static constexpr int kSub = TILE < 16 ? TILE : 16;  // a CTA renders kSub x kSub pixels of a tile
    static constexpr int kWarps = kSub * kSub / 32;
    // range positions per step, at most, and CTAs per SM: an 8x8 tile's two warps and short list leave no
    // room for more of either (250k / 1237x823 with 128 positions and 48 warps 133 us a frame, 128 and 40
    // 135, 256 and 32 135)
    static constexpr uint32_t kStage = TILE < 16 ? 128 : 512;
    static constexpr int kCtas = (TILE < 16 ? 48 : 40) / kWarps;
    RasterWarp warp[kWarps];
    float4 a[kStage];  // the step's records: (x, y, conic.x, conic.y)
    float4 b[kStage];  // (conic.z, opacity, r, g)
    float2 c[kStage];  // (b, cut)
    uint32_t masks[kStage / 32][kWarps];  // the step's hits per group of 32 positions and warp
};

// What a raster keeps besides the colours: nothing, the final transmittance, or that and the contributor
// count (and, for a differentiable frame, the hit masks).
constexpr int kKeepNothing = 0, kKeepT = 1, kKeepLast = 2;

// One pixel's blend of one splat given its alpha, 1 - alpha and colour times alpha. No branch: the splat
// counts unless power > 0, power < cut or alpha < 1/255 (a NaN power passes, as in the comparisons' plain
// form), and blends if testT >= 1e-4, by predicated instructions (written out: as selects they cost three
// more). T takes testT either way: once below 1e-4 it stays below, so nothing blends any more (a pixel
// outside the image starts at 0); final_t is the transmittance after the last blend.
template <int KEEP>
__device__ __forceinline__ void blend_one(float power, float alpha, float one_minus, float ra, float ga,
                                          float ba, uint32_t pos, float& T, float& cr, float& cg, float& cb,
                                          float& final_t, uint32_t& last) {
    const float testT = T * one_minus;
#define GS_BLEND(EXTRA, F, L)                                                                                          \
    asm("{\n .reg .pred in, blend;\n"                                                                            \
        " setp.leu.f32 in, %6, 0f00000000;\n"                                                                    \
        " setp.geu.and.f32 in, %7, %8, in;\n"                                                                    \
        " setp.ge.and.f32 blend, %9, %10, in;\n"                                                                 \
        " @blend fma.rn.f32 %1, %11, %0, %1;\n"                                                                  \
        " @blend fma.rn.f32 %2, %12, %0, %2;\n"                                                                  \
        " @blend fma.rn.f32 %3, %13, %0, %3;\n"                                                                  \
        " @in mov.f32 %0, %9;\n" EXTRA "}"                                                                       \
        : "+f"(T), "+f"(cr), "+f"(cg), "+f"(cb), F, L                                                              \
        : "f"(power), "f"(alpha), "f"(kEpsilon), "f"(testT), "f"(kBlendThreshold), "f"(ra), "f"(ga),             \
          "f"(ba), "r"(pos))
    if constexpr (KEEP == kKeepNothing) {
        float none;
        uint32_t unset;
        GS_BLEND("", "=f"(none), "=r"(unset));
    } else if constexpr (KEEP == kKeepT) {
        uint32_t unset;
        GS_BLEND(" @blend mov.f32 %4, %9;\n", "+f"(final_t), "=r"(unset));
    } else {
        GS_BLEND(" @blend mov.f32 %4, %9;\n @blend mov.u32 %5, %14;\n", "+f"(final_t), "+r"(last));
    }
}
#undef GS_BLEND

// One pixel's results.
template <int KEEP>
__device__ __forceinline__ void store_pixel(const RasterOut& out, size_t p, float cr, float cg, float cb, float final_t,
                                            uint32_t last) {
    if (out.rgb) {
        out.rgb[3 * p + 0] = cr;
        out.rgb[3 * p + 1] = cg;
        out.rgb[3 * p + 2] = cb;
    }
    if (KEEP != kKeepNothing && out.final_t) out.final_t[p] = final_t;
    if (KEEP == kKeepLast && out.n_contrib) out.n_contrib[p] = last;
    if (out.rgba8) {
        const uint32_t r8 = (uint32_t)(fminf(fmaxf(cr, 0.0f), 1.0f) * 255.0f + 0.5f);
        const uint32_t g8 = (uint32_t)(fminf(fmaxf(cg, 0.0f), 1.0f) * 255.0f + 0.5f);
        const uint32_t b8 = (uint32_t)(fminf(fmaxf(cb, 0.0f), 1.0f) * 255.0f + 0.5f);
        out.rgba8[p] = r8 | (g8 << 8) | (b8 << 16) | (255u << 24);
    }
}

// CTA `block` of a view: a sub-block of a tile, the longest tiles first.
template <int TILE, int KEEP>
__device__ __forceinline__ void raster_view(const RasterView& view, uint32_t block, uint32_t step) {
    const uint32_t* __restrict__ const vals = view.vals;
    const float4* __restrict__ const rec = view.rec;
    const RasterOut out = view.out;
    const uint32_t n = view.n, width = view.width, height = view.height, tiles_x = view.tiles_x;
    constexpr bool LAST = KEEP == kKeepLast;
    constexpr uint32_t kSub = RasterShared<TILE>::kSub, kWarps = RasterShared<TILE>::kWarps, kThreads = 32u * kWarps;
    constexpr uint32_t kSubs = TILE / kSub;  // CTAs across the tile
    extern __shared__ __align__(16) unsigned char s_raw[];
    RasterShared<TILE>& cta = *reinterpret_cast<RasterShared<TILE>*>(s_raw);

    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint4 place = __ldg(view.order + block / (kSubs * kSubs));
    const uint32_t tile = place.x, start = place.y, end = place.z, sub = block % (kSubs * kSubs);
    const uint32_t px0 = (tile % tiles_x) * TILE + kSub * (sub % kSubs), py0 = (tile / tiles_x) * TILE + kSub * (sub / kSubs);
    RasterWarp& sh = cta.warp[warp];
    const uint32_t bx = 8u * (warp % (kSub / 8u)), by = 4u * (warp / (kSub / 8u));  // the warp's block
    const uint32_t x = px0 + bx + (lane & 7u), y = py0 + by + (lane >> 3);
    // plane of the hit masks: the block's number in the tile, row by row
    const uint32_t plane = ((kSub * (sub / kSubs) + by) / 4u) * (TILE / 8u) + (kSub * (sub % kSubs) + bx) / 8u;
    const bool inside = x < width && y < height;
    const float2 nfx = both(-(float)x), nfy = both(-(float)y);

    float T = inside ? 1.0f : 0.0f, final_t = 1.0f, cr = 0.0f, cg = 0.0f, cb = 0.0f;
    uint32_t last = 0;
    uint32_t head = 0, tail = 0;             // hits blended, listed
    // every pixel of the warp is done, or none is in the image. The same question in two forms: 16x16 tiles with the
    // second lose 0.4% of a frame (1M / 1080p 335.2 -> 336.4 us), 32x32 ones with the first 1.1% (16 views 2433 -> 2460)
    bool over = TILE < 32 ? __all_sync(0xffffffffu, !inside) : __all_sync(0xffffffffu, T == 0.0f);

    // blends the next cnt (at most kChunk) listed hits of the step whose first position is pos0
    auto blend = [&](uint32_t cnt, uint32_t pos0) {
        __syncwarp();  // the list
        {
            float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f), b = a;
            float2 c = make_float2(0.0f, 0.0f);
            float* q = reinterpret_cast<float*>(sh.pair[lane >> 1]) + (lane & 1u);
            // past the hits alpha is 0; so it is below a positive cut-off, where the opacity itself is under 1/255
            uint32_t at = 0;
            if (lane < cnt) {
                at = sh.list[(head + lane) % kList];
                a = cta.a[at];
                b = cta.b[at];
                c = cta.c[at];
            }
            if (c.y > 0.0f) b.y = 0.0f;
            q[0] = a.x; q[2] = a.y; q[4] = a.z; q[6] = -a.w;
            q[8] = b.x; q[10] = b.y; q[12] = b.z; q[14] = b.w;
            q[16] = c.x;
            if (LAST) q[18] = __uint_as_float(pos0 + at + 1u);
        }
        __syncwarp();
        const uint32_t pairs = (cnt + 1u) / 2u;
#pragma unroll 2
        for (uint32_t k = 0; k < pairs; ++k) {
            const float4 p0 = sh.pair[k][0], p1 = sh.pair[k][1], p2 = sh.pair[k][2], p3 = sh.pair[k][3];
            float2 p4, pos = make_float2(0.0f, 0.0f);
            if (LAST) {
                const float4 v = sh.pair[k][4];
                p4 = make_float2(v.x, v.y);
                pos = make_float2(v.z, v.w);
            } else {
                p4 = *reinterpret_cast<const float2*>(&sh.pair[k][4]);
            }
            const float2 dx = __fadd2_rn(make_float2(p0.x, p0.y), nfx), dy = __fadd2_rn(make_float2(p0.z, p0.w), nfy);
            const float2 q = __ffma2_rn(__fmul2_rn(make_float2(p1.x, p1.y), dx), dx,
                                        __fmul2_rn(__fmul2_rn(make_float2(p2.x, p2.y), dy), dy));
            const float2 power = __ffma2_rn(both(-0.5f), q, __fmul2_rn(__fmul2_rn(make_float2(p1.z, p1.w), dx), dy));
            const float2 op = raster_alpha_unclamped2(make_float2(p2.z, p2.w), make_float2(max_nan(power.x, kPowerFloor), max_nan(power.y, kPowerFloor)));
            const float2 alpha = make_float2(fminf(kAlphaClamp, op.x), fminf(kAlphaClamp, op.y));
            const float2 om = __ffma2_rn(alpha, both(-1.0f), both(1.0f));
            const float2 ra = __fmul2_rn(make_float2(p3.x, p3.y), alpha), ga = __fmul2_rn(make_float2(p3.z, p3.w), alpha);
            const float2 ba = __fmul2_rn(p4, alpha);
            blend_one<KEEP>(power.x, alpha.x, om.x, ra.x, ga.x, ba.x, __float_as_uint(pos.x), T, cr, cg, cb, final_t, last);
            blend_one<KEEP>(power.y, alpha.y, om.y, ra.y, ga.y, ba.y, __float_as_uint(pos.y), T, cr, cg, cb, final_t, last);
        }
        head += cnt;
        over = __all_sync(0xffffffffu, T < kBlendThreshold);
        __syncwarp();
    };

    for (uint32_t i = start; i < end; i += step) {
        if (__syncthreads_and(over)) break;
        const uint32_t cnt = min(step, end - i);
        // stage the records and cull: each splat's octagon against the tile's blocks, one word per warp and
        // 32 positions
        for (uint32_t j = threadIdx.x; j < (cnt + 31u & ~31u); j += kThreads) {
            uint32_t bits = 0;
            const uint32_t g = j < cnt ? vals[i + j] : n;
            if (g < n) {  // always, unless the sort timed out
                const float4* r = rec + (size_t)kRecFloat4 * g;
                const float2 c = __ldg(reinterpret_cast<const float2*>(r));
                bits = block_bits<kSub>(c.x, c.y, __ldg(r + 3), (float)px0, (float)py0);
                if (bits) {
                    cp_async16(&cta.a[j], r);
                    cp_async16(&cta.b[j], r + 1);
                    cp_async8(&cta.c[j], r + 2);
                }
            }
            uint32_t word = 0;
#pragma unroll
            for (uint32_t w = 0; w < kWarps; ++w) {
                const uint32_t b = __ballot_sync(0xffffffffu, bits >> w & 1u);
                word = lane == w ? b : word;
            }
            if (lane < kWarps) cta.masks[j >> 5][lane] = word;
        }
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads();
        if (over) continue;
        const uint32_t groups = (cnt + 31u) / 32u;
        const uint32_t words = lane < groups ? cta.masks[lane][warp] : 0u;
        if (LAST && lane < groups && out.hit_masks) {  // the backward visits the same splats
            const size_t at = hit_mask_base(start, tile) + ((i - start) >> 5) + lane;
            if (GS_IN_BOUNDS(at, out.mask_pitch, view.status)) out.hit_masks[plane * out.mask_pitch + at] = words;
        }
        uint32_t any = __ballot_sync(0xffffffffu, words != 0u);
        while (!over && (any != 0u || head < tail)) {
            if (any != 0u && tail - head < kChunk) {
                const uint32_t group = __ffs(any) - 1u, m = __shfl_sync(0xffffffffu, words, group);
                if (m >> lane & 1u) sh.list[(tail + __popc(m & ((1u << lane) - 1u))) % kList] = 32u * group + lane;
                tail += __popc(m);
                any &= any - 1u;
            } else {
                blend(min(kChunk, tail - head), i - start);
            }
        }
    }
    if (inside) store_pixel<KEEP>(out, (size_t)y * width + x, cr, cg, cb, final_t, last);
}

template <int TILE, int KEEP>
__global__ void __launch_bounds__(RasterShared<TILE>::kWarps * 32, RasterShared<TILE>::kCtas)
k_raster(RasterView view, uint32_t step) {
    pdl_wait();
    raster_view<TILE, KEEP>(view, blockIdx.x, step);
}
// Several views: their longest tiles first, view by view, then their next ones.
template <int TILE, int KEEP>
__global__ void __launch_bounds__(RasterShared<TILE>::kWarps * 32, RasterShared<TILE>::kCtas)
k_raster_views(const __grid_constant__ Views<RasterView> views, uint32_t step) {
    pdl_wait();
    constexpr uint32_t kSubs = (TILE / RasterShared<TILE>::kSub) * (TILE / RasterShared<TILE>::kSub);
    const uint32_t unit = blockIdx.x / kSubs, at = unit / views.count;
    const RasterView& view = views.view[unit % views.count];
    if (at >= view.tiles) return;
    raster_view<TILE, KEEP>(view, at * kSubs + blockIdx.x % kSubs, step);
}

template <int TILE>
void launch_tile(const RasterView* views, uint32_t count, uint32_t step, cudaStream_t s) {
    constexpr uint32_t kSubs = TILE / RasterShared<TILE>::kSub;
    uint32_t tiles = 0;
    bool last = false, final_t = false;
    for (uint32_t v = 0; v < count; ++v) {
        tiles = std::max(tiles, views[v].tiles);
        last = last || views[v].out.n_contrib;
        final_t = final_t || views[v].out.final_t;
    }
    const dim3 grid(tiles * count * kSubs * kSubs), block(RasterShared<TILE>::kWarps * 32);
    const size_t smem = sizeof(RasterShared<TILE>);
    auto launch = [&](auto kernel, auto kernel_views) {
        if (count == 1) launch_pdl_smem(kernel, grid, block, smem, s, views[0], step);
        else launch_pdl_smem(kernel_views, grid, block, smem, s, pack_views(views, count), step);
    };
    if (last) launch(k_raster<TILE, kKeepLast>, k_raster_views<TILE, kKeepLast>);
    else if (final_t) launch(k_raster<TILE, kKeepT>, k_raster_views<TILE, kKeepT>);
    else launch(k_raster<TILE, kKeepNothing>, k_raster_views<TILE, kKeepNothing>);
}

template <int TILE>
void configure_tile() {
    auto configure = [](auto kernel) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(RasterShared<TILE>));
        cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    };
    configure(k_raster<TILE, kKeepNothing>);
    configure(k_raster<TILE, kKeepT>);
    configure(k_raster<TILE, kKeepLast>);
    configure(k_raster_views<TILE, kKeepNothing>);
    configure(k_raster_views<TILE, kKeepT>);
    configure(k_raster_views<TILE, kKeepLast>);
}

}  // namespace

void configure_raster_kernels() {
    configure_tile<8>();
    configure_tile<16>();
    configure_tile<32>();
}

// positions per step (a multiple of 32), as far as the stage goes: most tiles need one or two
uint32_t raster_step(uint32_t tile, uint32_t batch) {
    return std::min(4u * batch, tile == 8 ? RasterShared<8>::kStage : RasterShared<16>::kStage);
}

void launch_raster(const RasterView* views, uint32_t count, uint32_t tile, uint32_t batch, cudaStream_t s) {
    const uint32_t step = raster_step(tile, batch);
    if (tile == 8) launch_tile<8>(views, count, step, s);
    else if (tile == 32) launch_tile<32>(views, count, step, s);
    else launch_tile<16>(views, count, step, s);
}

}  // namespace gs
