// gs_backward.cu -- the raster half of the gradients of the splat pipeline (no counterpart in the
// reference, which only renders):
//   k_raster_backward     per 8x4 pixel block, walks the splats that the forward's warp of the block
//                         visited (its hit masks) back to front from the block's last contributor,
//                         recomputing power and alpha bit for bit as the forward did (same pinned
//                         arithmetic), recovering T by division, and accumulating dL/d(pixel.xy, conic,
//                         opacity, colour) per Gaussian: eight hits at a time summed over the block's
//                         pixels, four lanes to a hit, two vector atomics and a scalar one per hit. Up to the pixel's own
//                         chain the arithmetic runs on two hits at once by packed fp32 operations.
// The preprocess half (2D gradients -> the 59 attributes) is in gs_preprocess_backward.cu.
// Conventions: gradients flow through the fp32 RGB before quantization; culled Gaussians, skipped
// pairs and splats after a pixel's termination get none; active clamps (alpha 0.99, colour >= 0)
// pass none; where the frustum guard clamps t.x/t.z (t.y/t.z) no gradient flows through t.x (t.y),
// as in 3DGS.
#include "gs_kernels.h"
#include "gs_raster_common.cuh"

namespace gs {
namespace {

// ---- reduction of a hit's gradients over a block --------------------------------------------------------
// Of a (pixel, splat) pair there are gp = dL/dpower and w = alpha T, its blending weight; the splat's nine
// gradients follow from nine sums over the block's pixels: gp, gp dx, gp dy, gp dx^2, gp dx dy, gp dy^2 and w dC
// (dL/do is the first over o). The pixels leave gp and w of eight hits in shared memory and each hit is then
// summed by four lanes, a row of eight pixels each (dy is the row's), so that a pixel adds two values per hit
// instead of nine and the lanes meet in ten shuffles per eight hits.
//
// All of it is fp32, and dx and dy are the splat's own: sums of gp times powers of the pixel's offset from the
// block's centre, moved to the splat afterwards, cancel where the splat is narrow (at X from the centre of
// the block by X^2 over the mean dx^2), and as products on tf32 matrix instructions, operands split in two
// halves, they keep 22 bits. That form was here before: the scales' gradients of splats about a pixel wide
// were 9.1e-7 off 64 bits instead of 5.8e-7 (colours of splats of two pixels 4.0e-7 instead of 3.4e-7), and it was slower
// (1M / 1080p 283 us, then 260).
constexpr uint32_t kHits = 8;  // hits per flush

// Predicated adds to global memory (no branch around them).
__device__ __forceinline__ void red_add4_if(bool on, float* p, float x, float y, float z, float w) {
    asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %5, 0;\n @q red.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n}"
                 ::"l"(p), "f"(x), "f"(y), "f"(z), "f"(w), "r"((uint32_t)on) : "memory");
}
__device__ __forceinline__ void red_add_if(bool on, float* p, float x) {
    asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %2, 0;\n @q red.global.add.f32 [%0], %1;\n}"
                 ::"l"(p), "f"(x), "r"((uint32_t)on) : "memory");
}

// 1 / x for a normal x (a single instruction: no denormals, so no range handling; 1 ulp).
__device__ __forceinline__ float fast_rcp(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// One pixel's backward state: its last contributor L (1-based position in the tile range), the
// transmittance in front of the splat being visited, its colour gradient dC, and D = dC . S, S being
// the colour the splats behind the visited one added to the pixel (S = sum over them of alpha_j T_j c_j).
struct PixState {
    uint32_t L;
    float fx, fy, T, dr, dg, db;
    float d;
};

__device__ __forceinline__ void pix_load(PixState& p, uint32_t x, uint32_t y, uint32_t width, uint32_t height,
                                         const float* __restrict__ final_t, const uint32_t* __restrict__ n_contrib,
                                         const float* __restrict__ dl_drgb) {
    p.fx = (float)x;
    p.fy = (float)y;
    p.L = 0;
    p.T = 1.0f;
    p.dr = p.dg = p.db = 0.0f;
    p.d = 0.0f;
    if (x < width && y < height) {
        const size_t q = (size_t)y * width + x;
        p.L = n_contrib[q];
        p.T = final_t[q];
        p.dr = dl_drgb[3 * q];
        p.dg = dl_drgb[3 * q + 1];
        p.db = dl_drgb[3 * q + 2];
    }
}

// Visits the splat at 1-based range position pos for one pixel: the same power / exp / alpha
// decisions as the forward (bit for bit); gp = dL/dpower and its blending weight w, zeros if the pixel
// did not blend it. T is recovered by division (the approximate reciprocal, 1 ulp, of 1 - alpha >= 0.01 is
// accurate enough for a gradient). With C = sum_i alpha_i T_i c_i and T_{i+1} = T_i (1 - alpha_i),
// dC/dalpha_i = T_i c_i - S_i / (1 - alpha_i), S_i being the colour added behind splat i, so
// dL/dalpha_i = T_i K_i - D_i / (1 - alpha_i) with K_i = dC . c_i and D_i = dC . S_i, and D grows by
// alpha_i T_i K_i per step. No branch on the rejections: a rejected pixel takes alpha = 0 and K = 0, which
// leaves its state as it is, and gives two zeros, also where D is no longer finite.
__device__ __forceinline__ void pix_step(PixState& p, uint32_t pos, const float4& a, const float4& b,
                                         const float2& c, float& gp, float& w) {
    const float dx = a.x - p.fx, dy = a.y - p.fy;
    const float power = __fmaf_rn(-0.5f, __fmaf_rn(a.z * dx, dx, (b.x * dy) * dy), -((a.w * dx) * dy));
    // the forward's o * exp(power); a positive cut-off: the opacity itself is below 1/255
    const float og = raster_alpha_unclamped(c.y > 0.0f ? 0.0f : b.y, max_nan(power, kPowerFloor));
    float alpha = fminf(kAlphaClamp, og);
    // from here on only gradients are formed: fused multiply-adds are fine (the decisions
    // follow the forward's pinned arithmetic)
    float k = __fmaf_rn(b.z, p.dr, __fmaf_rn(b.w, p.dg, c.x * p.db));  // dC . c
    const bool in = (pos <= p.L) & !(power > 0.0f) & (alpha >= kEpsilon);
    alpha = in ? alpha : 0.0f;
    k = in ? k : 0.0f;
    const float ria = fast_rcp(1.0f - alpha);
    p.T = p.T * ria;  // transmittance in front of this splat
    w = alpha * p.T;
    const float dalpha = __fmaf_rn(p.T, k, -(p.d * ria));
    gp = in & (og <= kAlphaClamp) ? dalpha * alpha : 0.0f;  // a clamped alpha passes no gradient
    p.d = __fmaf_rn(w, k, p.d);
}

// The same for two splats, the one at the higher position first (back to front): what does not depend on the
// pixel's state is formed for both at once by packed operations (each half rounds like the scalar form).
// Pairs as the walk lays them out; opacity 0 stands for one below every cut-off (its alpha is 0).
__device__ __forceinline__ void pix_step2(PixState& p, const float4& p0, const float4& p1, const float4& p2,
                                          const float4& p3, const float4& p4, float2& gp, float2& w) {
    const float2 dx = __fadd2_rn(make_float2(p0.x, p0.y), both(-p.fx)), dy = __fadd2_rn(make_float2(p0.z, p0.w), both(-p.fy));
    const float2 q = __ffma2_rn(__fmul2_rn(make_float2(p1.x, p1.y), dx), dx,
                                __fmul2_rn(__fmul2_rn(make_float2(p2.x, p2.y), dy), dy));
    const float2 power = __ffma2_rn(both(-0.5f), q, __fmul2_rn(__fmul2_rn(make_float2(p1.z, p1.w), dx), dy));
    const float2 og = raster_alpha_unclamped2(make_float2(p2.z, p2.w),
                                              make_float2(max_nan(power.x, kPowerFloor), max_nan(power.y, kPowerFloor)));
    const float2 kk = __ffma2_rn(make_float2(p3.x, p3.y), both(p.dr),
                                 __ffma2_rn(make_float2(p3.z, p3.w), both(p.dg), __fmul2_rn(make_float2(p4.x, p4.y), both(p.db))));
    auto one = [&](float power, float og, float k, uint32_t pos, float& gp, float& w) {
        float alpha = fminf(kAlphaClamp, og);
        const bool in = (pos <= p.L) & !(power > 0.0f) & (alpha >= kEpsilon);
        alpha = in ? alpha : 0.0f;
        k = in ? k : 0.0f;
        const float ria = fast_rcp(1.0f - alpha);
        p.T = p.T * ria;
        w = alpha * p.T;
        const float dalpha = __fmaf_rn(p.T, k, -(p.d * ria));
        gp = in & (og <= kAlphaClamp) ? dalpha * alpha : 0.0f;
        p.d = __fmaf_rn(w, k, p.d);
    };
    one(power.x, og.x, kk.x, __float_as_uint(p4.z), gp.x, w.x);
    one(power.y, og.y, kk.y, __float_as_uint(p4.w), gp.y, w.y);
}

__device__ __forceinline__ bool pix_finite(const PixState& p) {
    return finite_f(p.dr) && finite_f(p.dg) && finite_f(p.db);
}

// The walk of a block with a pixel whose dL/dC is not finite. Such a pixel must not reach the splats that it does
// not blend, where zero times it would be NaN, so the sums over the block take the pixels that blend a splat one
// by one (selects, nine shuffle sums per hit) instead of the flush's plain products. Its own function, so that the
// common walk spends nothing on it: the choice within the flush cost 3% at 1M / 1080p (260 -> 267 us) and 8% at
// 20k / 397x301. Step of an image of NaN at 1M / 1080p 1.04 ms (a finite one 0.33), with one
// such pixel in 1000 0.365; 4.9 and 0.71 when each of them walked its tile's list by itself.
__device__ __noinline__ void walk_not_finite(PixState p, uint32_t wmax, const uint32_t* __restrict__ masks,
                                             const uint32_t* __restrict__ vals, const float4* __restrict__ rec,
                                             uint32_t n, float* __restrict__ grad2d) {
    constexpr uint32_t kAll = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t group = (wmax + 31u) >> 5; group-- > 0u;) {
        uint32_t m = masks[group];
        const uint32_t last = wmax - (group << 5);  // positions of the group that are visited
        if (last < 32u) m &= (1u << last) - 1u;
        if (m == 0u) continue;
        // a lane holds one of the group's splats
        const uint32_t mine = m >> lane & 1u ? vals[(group << 5) + lane] : n;
        float4 ra = make_float4(0.0f, 0.0f, 0.0f, 0.0f), rb = ra, rc = ra;
        if (mine < n) {
            ra = rec[(size_t)kRecFloat4 * mine];
            rb = rec[(size_t)kRecFloat4 * mine + 1];
            rc = rec[(size_t)kRecFloat4 * mine + 2];
        }
        while (m != 0u) {
            const int bit = 31 - __clz(m);
            m &= ~(1u << bit);
            const uint32_t gi = __shfl_sync(kAll, mine, bit);
            if (gi >= n) continue;  // only after a timed-out sort
            auto from = [&](float v) { return __shfl_sync(kAll, v, bit); };
            const float4 a = make_float4(from(ra.x), from(ra.y), from(ra.z), from(ra.w));
            const float4 b = make_float4(from(rb.x), from(rb.y), from(rb.z), from(rb.w));
            const float2 c = make_float2(from(rc.x), from(rc.y));
            float gp, w;
            pix_step(p, (group << 5) + (uint32_t)bit + 1u, a, b, c, gp, w);
            const bool on = w != 0.0f;  // blended (a blended pair's weight is positive)
            if (!__any_sync(kAll, on)) continue;
            const float dx = a.x - p.fx, dy = a.y - p.fy, gx = gp * dx, gy = gp * dy;
            float v[9] = {gp, gx, gy, gx * dx, gx * dy, gy * dy, w * p.dr, w * p.dg, w * p.db};
#pragma unroll
            for (int k = 0; k < 9; ++k) {
                v[k] = on ? v[k] : 0.0f;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(kAll, v[k], o);
            }
            float* q = grad2d + (size_t)8 * gi;
            red_add4_if(lane == 0u, q, -__fmaf_rn(a.z, v[1], a.w * v[2]), -__fmaf_rn(b.x, v[2], a.w * v[1]), v[6], v[7]);
            red_add4_if(lane == 1u, q + 4, -0.5f * v[3], -v[4], -0.5f * v[5], v[8]);
            red_add_if(lane == 2u, grad2d + (size_t)8 * n + gi, v[0] / b.y);
        }
    }
}

constexpr uint32_t kRowPitch = 36;  // floats per row: 32 pixels, padded so that the eight lanes that read
                                    // two rows at once hit distinct banks
constexpr uint32_t kRing = 64;      // staged hits per warp (room for 32 more at two flushes' pending)
constexpr uint32_t kChunk = 32;     // most hits laid out in pairs at once
constexpr uint32_t kBwdWarps = 2;   // warps per CTA; they share nothing

// Shared memory of a warp: a ring of staged hits, and what the pixels add to kHits of them.
struct BwdWarp {
    float4 a[kRing];  // (x, y, conic.x, conic.y)
    float4 b[kRing];  // (conic.z, opacity, r, g)
    float4 c[kRing];  // (b, cut, range position, Gaussian)
    float4 pair[kChunk / 2][5];  // (x, x', y, y'), (A, A', -B, -B'), (C, C', o, o'), (r, r', g, g'),
                                 // (b, b', position, position')
    float gp[kHits][kRowPitch], w[kHits][kRowPitch];
};

// One warp per 8x4 block, one lane per pixel, no barrier between warps. The forward left one word per
// block and 32 range positions with a bit for each splat that its cull let through (hit_masks): the warp
// reads them from the group of its pixels' largest last contributor down, and only the records of those
// splats are staged, 32 positions at a time, by asynchronous copies into the ring while the hits staged
// before are processed, eight at a time and fully unrolled. Against a CTA per tile that staged whole
// batches, computed the cull again and met at two barriers per batch, a hit's bookkeeping (finding the
// next bit, addresses, the counter of the pending rows) is gone.
//
// Bound by instruction issue (76% of slots at 29 warps per SM) and shared-memory reads (74%) where the
// blocks fill the GPU, by the longest list otherwise. Measured against a CTA per tile with shuffle
// reductions and two pixels per lane, mixture scenes: 1M / 1080p 405 -> 260 us; 3M / 1080p (mean of
// eight views) 879 -> 526; 500k / 720p (a list of 2300 splats) 358 -> 130; 20k / 397x301 92 -> 23.4. On the
// way, with the block's sums on matrix instructions (above), 1M / 1080p in thousand cycles, from 839: the chain's divide as one reciprocal and no branch in a hit 693 -> 664;
// predicated atomics 631; hits in pairs on packed operations 577, their loop fully unrolled 560.
template <int TILE>
__global__ void __launch_bounds__(kBwdWarps * 32, 32 / kBwdWarps) k_raster_backward(const uint4* __restrict__ order,
                                                                     const uint32_t* __restrict__ vals,
                                                                     const float4* __restrict__ rec, uint32_t n,
                                                                     uint32_t width, uint32_t height,
                                                                     uint32_t tiles_x, uint32_t tiles,
                                                                     const float* __restrict__ final_t,
                                                                     const uint32_t* __restrict__ n_contrib,
                                                                     const uint32_t* __restrict__ hit_masks,
                                                                     size_t mask_pitch,
                                                                     const float* __restrict__ dl_drgb,
                                                                     float* __restrict__ grad2d) {
    pdl_wait();
    constexpr uint32_t WX = TILE / 8, kTileWarps = TILE * TILE / 32;
    __shared__ BwdWarp s_warp[kBwdWarps];
    BwdWarp& sh = s_warp[threadIdx.x >> 5];

    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t wid = blockIdx.x * kBwdWarps + (threadIdx.x >> 5);
    const uint32_t warp = wid % kTileWarps;
    if (wid / kTileWarps >= tiles) return;
    const uint4 place = __ldg(order + wid / kTileWarps);
    const uint32_t tile = place.x, start = place.y, end = place.z;
    const uint32_t tx = tile % tiles_x, ty = tile / tiles_x;
    const uint32_t bx0 = tx * TILE + 8u * (warp % WX), by0 = ty * TILE + 4u * (warp / WX);
    const uint32_t len = end > start ? end - start : 0u;

    PixState p;
    pix_load(p, bx0 + (lane & 7u), by0 + (lane >> 3), width, height, final_t, n_contrib, dl_drgb);
    const uint32_t wmax = min(__reduce_max_sync(0xffffffffu, p.L), len);
    if (wmax == 0u) return;
    const uint32_t* const masks = hit_masks + (size_t)warp * mask_pitch + hit_mask_base(start, tile);
    if (!__all_sync(0xffffffffu, pix_finite(p))) {
        walk_not_finite(p, wmax, masks, vals + start, rec, n, grad2d);
        return;
    }
    // of a flush a lane sums hit fr over row fc of the block: the row's dL/dC, in pairs of pixels
    const uint32_t fr = lane >> 2, fc = lane & 3u;
    float2 dr[4], dg[4], db[4];
    {
        float* const plane = sh.gp[0];
        plane[lane] = p.dr;
        plane[32u + lane] = p.dg;
        plane[64u + lane] = p.db;
        __syncwarp();
        const float2* const row = reinterpret_cast<const float2*>(plane) + 4u * fc;
#pragma unroll
        for (uint32_t k = 0; k < 4u; ++k) {
            dr[k] = row[k];
            dg[k] = row[16u + k];
            db[k] = row[32u + k];
        }
        __syncwarp();
    }
    const float row_x = (float)bx0, row_y = (float)(by0 + fc);

    // lays the next cnt (at most kChunk) staged hits out as pairs, a lane each
    auto lay_out = [&](uint32_t h0, uint32_t cnt) {
        const uint32_t slot = (h0 + lane) % kRing;
        float4 a = sh.a[slot], b = sh.b[slot], c = sh.c[slot];
        float* q = reinterpret_cast<float*>(sh.pair[lane >> 1]) + (lane & 1u);
        if (c.y > 0.0f) b.y = 0.0f;  // a positive cut-off: the opacity itself is below 1/255
        if (lane >= cnt) {           // past the hits: a position no pixel blends
            a = b = c = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            c.z = __uint_as_float(0xFFFFFFFFu);
        }
        q[0] = a.x; q[2] = a.y; q[4] = a.z; q[6] = -a.w;
        q[8] = b.x; q[10] = b.y; q[12] = b.z; q[14] = b.w;
        q[16] = c.x; q[18] = c.z;
        __syncwarp();
    };
    // visits hits 8 v to 8 v + 7 of those laid out, which are staged from ring slot h0 on, and adds the
    // gradients of the first cnt of them
    auto visit = [&](uint32_t v, uint32_t h0, uint32_t cnt) {
#pragma unroll
        for (uint32_t u = 0; u < kHits / 2u; ++u) {
            const float4* r = sh.pair[4u * v + u];
            float2 gp, w;
            pix_step2(p, r[0], r[1], r[2], r[3], r[4], gp, w);
            sh.gp[2u * u][lane] = gp.x;
            sh.gp[2u * u + 1u][lane] = gp.y;
            sh.w[2u * u][lane] = w.x;
            sh.w[2u * u + 1u][lane] = w.y;
        }
        __syncwarp();
        const uint32_t slot = (h0 + fr) % kRing;
        const float4 a = sh.a[slot];
        const float2 b = *reinterpret_cast<const float2*>(&sh.b[slot]);
        const uint32_t gi = __float_as_uint(sh.c[slot].w);
        const float4 g0 = *reinterpret_cast<const float4*>(&sh.gp[fr][8u * fc]);
        const float4 g1 = *reinterpret_cast<const float4*>(&sh.gp[fr][8u * fc + 4u]);
        const float4 w0 = *reinterpret_cast<const float4*>(&sh.w[fr][8u * fc]);
        const float4 w1 = *reinterpret_cast<const float4*>(&sh.w[fr][8u * fc + 4u]);
        const float2 g[4] = {make_float2(g0.x, g0.y), make_float2(g0.z, g0.w), make_float2(g1.x, g1.y), make_float2(g1.z, g1.w)};
        const float2 wt[4] = {make_float2(w0.x, w0.y), make_float2(w0.z, w0.w), make_float2(w1.x, w1.y), make_float2(w1.z, w1.w)};
        const float x0 = a.x - row_x, dy = a.y - row_y;
        float2 dx = make_float2(x0, x0 - 1.0f);
        float2 t = __fmul2_rn(g[0], dx), s0 = g[0], sx = t, sxx = __fmul2_rn(t, dx);
        float2 r = __fmul2_rn(wt[0], dr[0]), gr = __fmul2_rn(wt[0], dg[0]), bl = __fmul2_rn(wt[0], db[0]);
#pragma unroll
        for (uint32_t k = 1; k < 4u; ++k) {
            dx = __fadd2_rn(dx, both(-2.0f));
            t = __fmul2_rn(g[k], dx);
            s0 = __fadd2_rn(s0, g[k]);
            sx = __fadd2_rn(sx, t);
            sxx = __ffma2_rn(t, dx, sxx);
            r = __ffma2_rn(wt[k], dr[k], r);
            gr = __ffma2_rn(wt[k], dg[k], gr);
            bl = __ffma2_rn(wt[k], db[k], bl);
        }
        // sums over the row: gp, gp dx, gp dy, gp dx^2, gp dx dy, gp dy^2, w dC
        float sum0 = s0.x + s0.y;
        const float rx = sx.x + sx.y, ry = dy * sum0;
        const float even[4] = {rx, ry, r.x + r.y, gr.x + gr.y};
        const float odd[4] = {sxx.x + sxx.y, dy * rx, dy * ry, bl.x + bl.y};
        // and over the four rows: the even lanes of a hit get the first four, the odd ones the others
        const bool first = (fc & 1u) == 0u;
        float v4[4];
#pragma unroll
        for (uint32_t k = 0; k < 4u; ++k) {
            v4[k] = (first ? even[k] : odd[k]) + __shfl_xor_sync(0xffffffffu, first ? odd[k] : even[k], 1);
            v4[k] += __shfl_xor_sync(0xffffffffu, v4[k], 2);
        }
        sum0 += __shfl_xor_sync(0xffffffffu, sum0, 1);
        sum0 += __shfl_xor_sync(0xffffffffu, sum0, 2);
        const bool valid = fr < cnt && gi < n;
        // four zeros (no pixel of the block blended the splat) are not added: times a conic that is not finite they
        // would be NaN
        const bool some = ((__float_as_uint(v4[0]) | __float_as_uint(v4[1]) | __float_as_uint(v4[2]) | __float_as_uint(v4[3])) << 1) != 0u;
        red_add4_if(valid && some && fc < 2u, grad2d + (size_t)8 * gi + 4u * fc,
                    first ? -__fmaf_rn(a.z, v4[0], a.w * v4[1]) : -0.5f * v4[0],
                    first ? -__fmaf_rn(b.x, v4[1], a.w * v4[0]) : -v4[1], first ? v4[2] : -0.5f * v4[2], v4[3]);
        const float ro = fast_rcp(b.y);  // and a Newton step: 1 / o, nearly rounded
        red_add_if(valid && fc == 2u && sum0 != 0.0f, grad2d + (size_t)8 * n + gi, sum0 * __fmaf_rn(ro, __fmaf_rn(-b.y, ro, 1.0f), ro));
        __syncwarp();
    };

    // the groups of 32 positions with hits, from the top down: masks are read 32 groups at a time, and the
    // Gaussian indices of a group are loaded while the group before it is staged
    int32_t group = (int32_t)((wmax - 1u) >> 5) + 1;  // the group staged last
    uint32_t words = 0, left = 0;   // the lane's mask word of the current 32 groups; how many are unread
    uint32_t m = 0, gnext = n;      // the next group's mask and this lane's Gaussian in it
    auto next_group = [&]() {
        m = 0;
        while (m == 0u && group > 0) {
            --group;
            if (left == 0u) {
                left = 32u;
                const int32_t at = group - (int32_t)lane;
                words = at >= 0 ? masks[at] : 0u;
            }
            m = __shfl_sync(0xffffffffu, words, 32u - left);
            --left;
            const uint32_t last = wmax - ((uint32_t)group << 5);  // positions of the group that are visited
            if (last < 32u) m &= (1u << last) - 1u;
        }
        if (m >> lane & 1u) gnext = vals[start + ((uint32_t)group << 5) + lane];
    };

    uint32_t head = 0, ready = 0, tail = 0;  // hits visited, staged for certain, staged or on their way
    auto process = [&](uint32_t cnt) {
        lay_out(head, cnt);
        for (uint32_t v = 0; kHits * v < cnt; ++v) visit(v, head + kHits * v, min(kHits, cnt - kHits * v));
        head += cnt;
    };
    next_group();
    while (true) {
        while (m != 0u && tail - head + __popc(m) <= kRing) {
            if (m >> lane & 1u) {
                const uint32_t slot = (tail + __popc(m >> lane) - 1u) % kRing;  // back to front
                const bool ok = gnext < n;
                const uint32_t g = ok ? gnext : 0u;
                cp_async16(&sh.a[slot], rec + (size_t)kRecFloat4 * g);
                cp_async16(&sh.b[slot], rec + (size_t)kRecFloat4 * g + 1);
                cp_async8(&sh.c[slot], rec + (size_t)kRecFloat4 * g + 2);
                // an index out of range only comes from a timed-out sort: a position no pixel blends
                const uint32_t pos = ok ? ((uint32_t)group << 5) + lane + 1u : 0xFFFFFFFFu;
                reinterpret_cast<uint2*>(&sh.c[slot])[1] = make_uint2(pos, ok ? g : n);
            }
            tail += __popc(m);
            next_group();
        }
        cp_async_commit();
        if (m == 0u) break;
        cp_async_wait<1>();
        __syncwarp();
        if (ready - head >= 2u * kHits) process(min(kChunk, ready - head) & ~(kHits - 1u));
        ready = tail;
    }
    cp_async_wait<0>();
    __syncwarp();
    while (head < tail) process(min(kChunk, tail - head));
}

template <int TILE, typename... Args>
void launch_bwd_tile(uint32_t tiles, cudaStream_t s, Args&&... args) {
    const uint32_t warps = tiles * (TILE * TILE / 32);
    launch_pdl(k_raster_backward<TILE>, dim3((warps + kBwdWarps - 1u) / kBwdWarps), dim3(kBwdWarps * 32), s,
               std::forward<Args>(args)...);
}

}  // namespace

void configure_raster_backward() {
    cudaFuncSetAttribute(k_raster_backward<8>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    cudaFuncSetAttribute(k_raster_backward<16>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    cudaFuncSetAttribute(k_raster_backward<32>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
}

void launch_raster_backward(uint32_t tile, const uint4* order, const uint32_t* vals, const float4* rec, uint32_t n,
                            uint32_t width, uint32_t height, uint32_t tiles_x, uint32_t tiles_y,
                            const float* final_t, const uint32_t* n_contrib, const uint32_t* hit_masks,
                            size_t mask_pitch, const float* dl_drgb, float* grad2d, cudaStream_t s) {
    auto launch = [&](auto bwd) {
        bwd(tiles_x * tiles_y, s, order, vals, rec, n, width, height, tiles_x, tiles_x * tiles_y, final_t, n_contrib,
            hit_masks, mask_pitch, dl_drgb, grad2d);
    };
    if (tile == 8) launch([](auto&&... a) { launch_bwd_tile<8>(a...); });
    else if (tile == 32) launch([](auto&&... a) { launch_bwd_tile<32>(a...); });
    else launch([](auto&&... a) { launch_bwd_tile<16>(a...); });
}

}  // namespace gs
