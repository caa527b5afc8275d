// Conservative pixel boxes of packed 2D records, shared by the rasterizer's
// tile kernels and its VJPs.
#pragma once

#include "common.cuh"

namespace r2s {

// --------------------------------------------------------------------------
// Pixel boxes
// --------------------------------------------------------------------------

// A record's box on one tile, in tile-local pixel indices: column and row bit
// masks, the packed origin and extent (x0 | y0 << 8 | width << 16 |
// height << 24) and ceil(65536 / width), with which (k * magic) >> 16 equals
// k / width for every k < 1024 and width <= 32. An empty box has zero masks
// and extent.
struct alignas(16) TileBox {
    uint32_t cols, rows, packed, magic;
};

__device__ __forceinline__ uint32_t low_bits(uint32_t n) { return n >= 32u ? 0xffffffffu : ((1u << n) - 1u); }

// Clips the inclusive pixel range [x0, x1] x [y0, y1] (indices relative to
// (ox, oy)) to a conservative box of the pixels whose sample can pass the
// contribution test; returns false when no pixel of the range can pass.
//
// Gaussian: a sample counts only if |o mu| exp(-sigma) >= 1e-5, i.e. sigma <=
// s = ln(|o mu| 1e5), with sigma = d^T Q d / 2 and Q = [[a, b], [b, c]]. When Q
// is positive definite with condition number <= (a + c)^2 / det <= 1000, the
// rounded sigma the sample computes is within 8 * 2^-24 * 1000 < 5e-4 of sigma
// relative (each rounding error is relative to |terms| <= cond * sigma), and
// the fast exponential and logarithm add < 1e-5 absolute; so every passing
// pixel lies in the ellipse sigma <= s' = s + 1e-3 |s| + 1e-3, whose bounding
// box has half-widths sqrt(2 s' c / det) and sqrt(2 s' a / det). Those are
// widened by 0.1 % plus 0.01 pixel, and by 1e-6 of the coordinates' magnitude
// for the rounding of the box arithmetic itself.
// Beta: a sample needs d2 = d^T Q d < 1; by the same argument every passing
// pixel has d2 < 1.001.
// Anything outside those conditions (a conic that is not positive definite or
// badly conditioned, non-finite values) falls back to the whole tile, so the
// box never drops a sample the reference would count.
template <typename S, bool kBeta>
__device__ __forceinline__ bool clip_to_record(const Rec2D<S>& r, uint32_t ox, uint32_t oy, uint32_t& x0,
                                               uint32_t& x1, uint32_t& y0, uint32_t& y1, bool& bounded) {
    const S a = r.a, b = r.b, c = r.c;
    const S det = a * c - b * b;
    const S tr = a + c;
    bounded = a > S(0) && c > S(0) && det > S(0) && tr * tr <= S(1000) * det;
    S reach = S(1.001);
    if (!kBeta) {
        const S om = fabs(r.o * r.mu);
        if (bounded && om == S(0)) return false;  // every alpha is zero
        S s = log(om) + S(11.512925464970229);    // ln(1e5)
        s = s + S(1e-3) * fabs(s) + S(1e-3);
        if (bounded && isfinite(s) && s < S(0)) return false;
        bounded = bounded && isfinite(s);
        reach = S(2) * s;
    }
    if (!bounded) return true;
    const S hx = sqrt(reach * c / det) * S(1.001) + S(0.01);
    const S hy = sqrt(reach * a / det) * S(1.001) + S(0.01);
    // Pixel j (centre j + 0.5) can pass only if |j + 0.5 - x| <= hx.
    const S cx = r.x - S(0.5) - static_cast<S>(ox);
    const S cy = r.y - S(0.5) - static_cast<S>(oy);
    const S mx = S(1e-6) * (fabs(r.x) + hx + static_cast<S>(ox));
    const S my = S(1e-6) * (fabs(r.y) + hy + static_cast<S>(oy));
    const S lo_x = ceil(cx - hx - mx), hi_x = floor(cx + hx + mx);
    const S lo_y = ceil(cy - hy - my), hi_y = floor(cy + hy + my);
    if (!(isfinite(lo_x) && isfinite(hi_x) && isfinite(lo_y) && isfinite(hi_y))) return true;
    if (hi_x < static_cast<S>(x0) || lo_x > static_cast<S>(x1) || hi_y < static_cast<S>(y0) ||
        lo_y > static_cast<S>(y1))
        return false;
    if (lo_x > static_cast<S>(x0)) x0 = static_cast<uint32_t>(lo_x);
    if (hi_x < static_cast<S>(x1)) x1 = static_cast<uint32_t>(hi_x);
    if (lo_y > static_cast<S>(y0)) y0 = static_cast<uint32_t>(lo_y);
    if (hi_y < static_cast<S>(y1)) y1 = static_cast<uint32_t>(hi_y);
    return x0 <= x1 && y0 <= y1;
}

template <typename S, bool kBeta>
__device__ __forceinline__ bool clip_to_record(const Rec2D<S>& r, uint32_t ox, uint32_t oy, uint32_t& x0,
                                               uint32_t& x1, uint32_t& y0, uint32_t& y1) {
    bool bounded;
    return clip_to_record<S, kBeta>(r, ox, oy, x0, x1, y0, y1, bounded);
}

// The record's box on the tile with origin (ox, oy) and valid extent vx x vy.
template <typename S, bool kBeta>
__device__ __forceinline__ TileBox record_box(const Rec2D<S>& r, uint32_t ox, uint32_t oy, uint32_t vx, uint32_t vy) {
    uint32_t x0 = 0, x1 = vx - 1, y0 = 0, y1 = vy - 1;
    if (!clip_to_record<S, kBeta>(r, ox, oy, x0, x1, y0, y1)) return TileBox{0u, 0u, 0u, 1u};
    const uint32_t bw = x1 - x0 + 1, bh = y1 - y0 + 1;
    TileBox box;
    box.cols = low_bits(bw) << x0;
    box.rows = low_bits(bh) << y0;
    box.packed = x0 | (y0 << 8) | (bw << 16) | (bh << 24);
    box.magic = (65536u + bw - 1u) / bw;
    return box;
}

// -(log2 e): exp(-s) = 2^(-s log2 e).
constexpr float kNegLog2e = -1.4426950408889634f;

}  // namespace r2s
