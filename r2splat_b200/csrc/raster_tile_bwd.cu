// Tile-parallel VJP of the fp32 Gaussian rasterizer with the variance branch,
// over the forward's sorted lists, one lane per (record, pixel block) pair.
//
// A CTA owns a share of one tile's list. Its warps stage the records in batches
// with the 8x8 pixel blocks of the tile that each record's box meets, list the
// (record, block) pairs block by block, and walk them 32 at a time, one pair
// per lane, all lanes stepping through their block's pixels in lockstep. Every
// lane reads its block's adjoints from shared memory (lanes of one block read
// the same address) and keeps its record's sums serially: no per-record
// stepping, no wrap test, no reduction across lanes, where the record walk of
// raster.cu steps lane groups through each record's box and leaves a third of
// its lanes past a box's end. It evaluates whole blocks, 1.8 times the box's
// samples (565 against 317 a record in the cone-beam scene of 200,000
// primitives and 64 views at 512^2), at less than a third of the instructions.
//
// Each (tile, record) pair's sums go to a slot of its own and a second pass adds
// each record's slots in tile order and applies its constants, so the gradients
// are the same on every run: no atomics.
//
// Measured with the set-up and slot passes (B200): 50,021 primitives, 17 views
// of 333 x 517, 3.76e6 pairs: 1.06 -> 0.57 ms. What bounds it (counters of the
// same walk without the variance terms): the FMA pipe and the special-function
// unit are each busy 53 % of the time, the issue slots 62 %. A packed FMA with
// three distinct register pairs takes 3.4 cycles instead of 2 (register ports),
// and the gathers of a batch's records are exposed at the start of each share.
// Occupancy does not move it: 5, 6, 7 and 8 resident CTAs and 8x4 or 4x8 blocks
// stay within 5 %; a persistent grid drawing shares from a counter was slower.
//
// Without the variance branch the record walk stays: its sums' order is part of
// what a fit step reproduces, since a smooth image adjoint makes the rotation
// gradient cancel by a factor of a hundred.
#include <algorithm>

#include "common.cuh"
#include "raster_box.cuh"

namespace r2s {

namespace {

constexpr int kBlock = 8;  // a pair's pixel block is 8 x 8
constexpr uint32_t kTileBwdWarps = 4;
constexpr uint32_t kTileBwdThreads = kTileBwdWarps * 32u;
constexpr uint32_t kTileBwdBatch = 96;   // records a warp stages at once
constexpr uint32_t kTileBwdBlocksPerSm = 5;  // 96 registers a thread: the walk holds its block's sums without spills

// A slot holds eight values, 32 bytes, one sector: with u = g vis (g: the image
// adjoint plus the variance chain term), sum u {dx, dy, dx^2, dx dy, dy^2},
// sum u and sum v_var vis^2; the last is unused.
constexpr uint32_t kSlotValues = 8;
constexpr uint32_t kSums = 7;

struct TileBwdGeom {
    uint32_t C, N, width, height, tiles_x, n_tiles, log_t, log_blocks;
    int32_t n_isects;
    const int64_t* n_dev;
    uint64_t capacity;
};

// One 32-byte (sector-wide) load or store: a scattered access costs one cache
// lookup instead of two.
struct alignas(32) Float8 {
    float v[8];
};
__device__ __forceinline__ Float8 load_float8(const void* p) {
    Float8 r;
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(r.v[0]), "=f"(r.v[1]), "=f"(r.v[2]), "=f"(r.v[3]), "=f"(r.v[4]), "=f"(r.v[5]), "=f"(r.v[6]), "=f"(r.v[7])
        : "l"(p));
    return r;
}
__device__ __forceinline__ void store_float8(void* p, const Float8& r) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 :: "l"(p), "f"(r.v[0]), "f"(r.v[1]), "f"(r.v[2]), "f"(r.v[3]), "f"(r.v[4]), "f"(r.v[5]), "f"(r.v[6]),
                    "f"(r.v[7])
                 : "memory");
}
__device__ __forceinline__ Rec2D<float> as_record(const Float8& f) {
    return Rec2D<float>{f.v[0], f.v[1], f.v[2], f.v[3], f.v[4], f.v[5], f.v[6], f.v[7]};
}

// What the tile kernel needs of a record besides its values, tabulated once
// per record (a record lies on several tiles: 3.7 at 200,000 primitives and
// 512^2). Its slots are numbered over its tile rectangle, row by row, so the
// slot is an affine function of the tile: base + ty * width + tx (base may be
// negative). The box is clip_to_record's over the whole rectangle, in pixels;
// x0 > x1 marks a record without pixels.
struct alignas(16) RecordMeta {
    int32_t base;
    uint32_t width;  // bit 31: the record's box is an ellipse's (bounded)
    uint32_t xs, ys;  // x0 | x1 << 16, y0 | y1 << 16
};

__global__ void __launch_bounds__(256) record_meta_kernel(const Rec2D<float>* __restrict__ records,
                                                          const ushort4* __restrict__ rects,
                                                          const int64_t* __restrict__ cum, size_t total,
                                                          uint32_t width, uint32_t height, uint32_t T,
                                                          RecordMeta* __restrict__ meta) {
    const size_t r = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (r >= total) return;
    const ushort4 rect = rects[r];
    const uint32_t w = uint32_t(rect.z) - rect.x;
    const int64_t first = r == 0 ? 0 : cum[r - 1];
    RecordMeta m{int32_t(first - int64_t(rect.y) * w - rect.x), w, 1u, 1u};
    uint32_t x0 = rect.x * T, y0 = rect.y * T;
    uint32_t x1 = min(rect.z * T, width), y1 = min(rect.w * T, height);
    if (x0 < x1 && y0 < y1) {
        --x1;
        --y1;
        bool bounded;
        if (clip_to_record<float, false>(as_record(load_float8(records + r)), 0u, 0u, x0, x1, y0, y1, bounded)) {
            m.xs = x0 | (x1 << 16);
            m.ys = y0 | (y1 << 16);
        }
        if (bounded) m.width |= 0x80000000u;
    }
    meta[r] = m;
}

// One lane's walk of an 8x8 pixel block with its first pixel centre at (bx, by),
// column by column. g and gvar hold the block's adjoints by columns. The two
// samples of a packed step are two adjacent rows, so the rows' terms (dy and the
// quadratic form's term in dy) are set up once per block as pairs and a column
// costs one set of terms in dx; the sums are kept per row pair. The samples'
// contribution tests are taken on the same expressions, rounded the same way,
// as the record walk of raster.cu.
//
// kStrict tests sigma >= 0 per sample; a bounded record's sigma cannot round to
// a negative value (the error bound of its box), so a batch of bounded records
// is walked without that test.
template <bool kStrict>
__device__ __forceinline__ void walk_block(const float4 f0, const float4 f1, float bx, float by, const float* g,
                                           const float* gvar, float (&sum)[kSums]) {
    constexpr int kP = kBlock / 2;
    // f0: x, y, a, b; f1: c, o mu, 2 q o mu.
    float2 dy[kP], rc[kP], s0[kP], s1[kP], s2[kP];
    const float2 ny = splat2(-f0.y), py0 = make_float2(by, by + 1.f);
    const float2 qa = splat2(f0.z), qb = splat2(f0.w), qc = splat2(f1.x);
#pragma unroll
    for (int i = 0; i < kP; ++i) {
        dy[i] = add2(add2(py0, splat2(static_cast<float>(2 * i))), ny);
        rc[i] = mul2(mul2(qc, dy[i]), dy[i]);
        s0[i] = s1[i] = s2[i] = splat2(0.f);
    }
    float2 s6 = splat2(0.f);
    const float2 nx = splat2(-f0.x);
    float2 px = splat2(bx);
#pragma unroll
    for (int j = 0; j < kBlock; ++j) {
        const float2 dx = add2(px, nx);
        px = add2(px, splat2(1.f));
        const float2 dxx = mul2(dx, dx);
        float2 col[kP], colv[kP];
#pragma unroll
        for (int i = 0; i < kP; i += 2) {
            const float4 v4 = *reinterpret_cast<const float4*>(g + j * kBlock + 2 * i);
            col[i] = make_float2(v4.x, v4.y);
            col[i + 1] = make_float2(v4.z, v4.w);
            const float4 w4 = *reinterpret_cast<const float4*>(gvar + j * kBlock + 2 * i);
            colv[i] = make_float2(w4.x, w4.y);
            colv[i + 1] = make_float2(w4.z, w4.w);
        }
        // Step by step over the column's row pairs: neighbouring instructions share an operand (dx, qa, dxx),
        // which halves the register reads of the packed operations.
        float2 u[kP];
        const float om = f1.y;
        const float2 uq = splat2(f1.z), adx = mul2(qa, dx), bdx = mul2(qb, dx);
        float2 sigma[kP];
#pragma unroll
        for (int i = 0; i < kP; ++i) sigma[i] = mul2(splat2(0.5f), fma2(adx, dx, rc[i]));
#pragma unroll
        for (int i = 0; i < kP; ++i) sigma[i] = fma2(bdx, dy[i], sigma[i]);
#pragma unroll
        for (int i = 0; i < kP; ++i) {
            const float vx = exp(-sigma[i].x), vy = exp(-sigma[i].y);
            const bool ka = !((kStrict && sigma[i].x < 0.f) || fabs(om * vx) < 1e-5f);
            const bool kb = !((kStrict && sigma[i].y < 0.f) || fabs(om * vy) < 1e-5f);
            const float2 vis = make_float2(ka ? vx : 0.f, kb ? vy : 0.f);
            const float2 vvis = mul2(colv[i], vis);
            s6 = fma2(vvis, vis, s6);
            u[i] = mul2(fma2(uq, vvis, col[i]), vis);
        }
#pragma unroll
        for (int i = 0; i < kP; ++i) s0[i] = add2(s0[i], u[i]);
#pragma unroll
        for (int i = 0; i < kP; ++i) s1[i] = fma2(u[i], dx, s1[i]);
#pragma unroll
        for (int i = 0; i < kP; ++i) s2[i] = fma2(u[i], dxx, s2[i]);
    }
    float2 m0 = s0[0], mx = s1[0], mxx = s2[0], mxy = mul2(s1[0], dy[0]), my = mul2(s0[0], dy[0]);
    float2 myy = mul2(my, dy[0]);
#pragma unroll
    for (int i = 1; i < kP; ++i) {
        const float2 ud = mul2(s0[i], dy[i]);
        m0 = add2(m0, s0[i]);
        mx = add2(mx, s1[i]);
        mxx = add2(mxx, s2[i]);
        mxy = fma2(s1[i], dy[i], mxy);
        my = add2(my, ud);
        myy = fma2(ud, dy[i], myy);
    }
    sum[0] = mx.x + mx.y;
    sum[1] = my.x + my.y;
    sum[2] = mxx.x + mxx.y;
    sum[3] = mxy.x + mxy.y;
    sum[4] = myy.x + myy.y;
    sum[5] = m0.x + m0.y;
    sum[6] = s6.x + s6.y;
}

__global__ void __launch_bounds__(kTileBwdThreads, kTileBwdBlocksPerSm) raster_tile_bwd_kernel(
    const Rec2D<float>* __restrict__ records, const RecordMeta* __restrict__ meta, const float* __restrict__ var_q,
    const int32_t* __restrict__ offsets, const int32_t* __restrict__ flatten_ids, TileBwdGeom g,
    const float* __restrict__ v_render, const float* __restrict__ v_render_var, float* __restrict__ slots) {
    constexpr uint32_t R = kTileBwdBatch, kPer = R / 32u;
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t tile = blockIdx.x, cam = blockIdx.y;
    const uint32_t key = cam * g.n_tiles + tile;
    const int32_t start = offsets[key];
    const int32_t n_total = g.n_dev != nullptr ? int32_t(*g.n_dev) : g.n_isects;
    const int32_t end = (key + 1 == g.C * g.n_tiles) ? n_total : offsets[key + 1];
    const int32_t count = end - start;
    // The warp's share of the list.
    const int32_t shares = int32_t(gridDim.z * kTileBwdWarps);
    const int32_t share = (count + shares - 1) / shares;
    if (int32_t(blockIdx.z * kTileBwdWarps) * share >= count) return;  // block-uniform; empty lists too
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    const int32_t first = start + int32_t(blockIdx.z * kTileBwdWarps + warp) * share;
    const int32_t last = min(end, first + share);
    const uint32_t T = 1u << g.log_t, TT = T << g.log_t;
    const uint32_t ty = tile / g.tiles_x, tx = tile - ty * g.tiles_x;
    const uint32_t ox = tx << g.log_t, oy = ty << g.log_t;

    // Shared memory: the tile's adjoints block by block, then each warp's batch.
    float* s_g = reinterpret_cast<float*>(smem);  // [blocks][8][8], columns of pixels
    float* s_gv = s_g + TT;                       // the same of the variance adjoint
    const uint32_t blocks = 1u << g.log_blocks, log_bx = g.log_t - 3u;
    const size_t per_warp = 2u * R * sizeof(float4) + kSums * R * sizeof(float) + R * sizeof(uint32_t) +
                            (size_t(R) << g.log_blocks) * sizeof(uint16_t);
    float4* s_f0 = reinterpret_cast<float4*>(reinterpret_cast<unsigned char*>(s_gv + TT) +
                                             warp * per_warp);          // [R]
    float4* s_f1 = s_f0 + R;                                            // [R]
    float* s_acc = reinterpret_cast<float*>(s_f1 + R);                  // [kSums][R]
    uint32_t* s_slot = reinterpret_cast<uint32_t*>(s_acc + kSums * R);  // [R]
    uint16_t* s_item = reinterpret_cast<uint16_t*>(s_slot + R);         // [R * blocks]: block << 7 | record

    const size_t cam_base = size_t(cam) * g.height * g.width;
    for (uint32_t p = t; p < TT; p += kTileBwdThreads) {
        const uint32_t y = p >> g.log_t, x = p & (T - 1u);
        const bool ok = ox + x < g.width && oy + y < g.height;
        const size_t pid = cam_base + size_t(oy + y) * g.width + (ox + x);
        const uint32_t at = (((y / kBlock) << log_bx) + x / kBlock) * (kBlock * kBlock) + (x % kBlock) * kBlock + y % kBlock;
        s_g[at] = (ok && v_render != nullptr) ? v_render[pid] : 0.f;
        s_gv[at] = ok ? v_render_var[pid] : 0.f;
    }
    __syncthreads();

    // Equal batches of at most R records.
    const int32_t n_batches = (share + int32_t(R) - 1) / int32_t(R);
    const int32_t batch = (share + n_batches - 1) / n_batches;
    for (int32_t b0 = first; b0 < last; b0 += batch) {
        const int32_t n = min(batch, last - b0);
#pragma unroll
        for (uint32_t i = 0; i < kSums * kPer; ++i) s_acc[i * 32u + lane] = 0.f;
        bool plain = true;
        uint32_t hits[kPer];
#pragma unroll
        for (uint32_t k = 0; k < kPer; ++k) {
            hits[k] = 0u;
            const uint32_t r = k * 32u + lane;
            if (int32_t(r) >= n) continue;
            const int32_t rid = flatten_ids[b0 + int32_t(r)];
            const Rec2D<float> rec = as_record(load_float8(records + rid));
            const RecordMeta m = meta[rid];
            const int32_t slot = m.base + int32_t(ty * (m.width & 0x7fffffffu) + tx);
            s_slot[r] = uint64_t(uint32_t(slot)) < g.capacity ? uint32_t(slot) : 0xffffffffu;
            plain = plain && (m.width >> 31) != 0u;
            const float om = rec.o * rec.mu;
            const float q = var_q != nullptr ? var_q[uint32_t(rid) - cam * g.N] : 0.f;
            s_f0[r] = make_float4(rec.x, rec.y, rec.a, rec.b);
            s_f1[r] = make_float4(rec.c, om, 2.f * q * om, 0.f);
            // The blocks of this tile that the record's box meets.
            const uint32_t x0 = max(m.xs & 0xffffu, ox), x1 = min(m.xs >> 16, ox + T - 1u);
            const uint32_t y0 = max(m.ys & 0xffffu, oy), y1 = min(m.ys >> 16, oy + T - 1u);
            if (x0 <= x1 && y0 <= y1) {
                const uint32_t c0 = (x0 - ox) / kBlock, c1 = (x1 - ox) / kBlock;
                const uint32_t r0 = (y0 - oy) / kBlock, r1 = (y1 - oy) / kBlock;
                const uint32_t row = (2u << c1) - (1u << c0);
                for (uint32_t y = r0; y <= r1; ++y) hits[k] |= row << (y << log_bx);
            }
        }
        plain = __all_sync(0xffffffffu, plain);
        // The pairs, block by block.
        uint32_t n_items = 0u;
        for (uint32_t b = 0; b < blocks; ++b) {
#pragma unroll
            for (uint32_t k = 0; k < kPer; ++k) {
                const bool hit = (hits[k] >> b) & 1u;
                const uint32_t who = __ballot_sync(0xffffffffu, hit);
                if (hit) s_item[n_items + __popc(who & ((1u << lane) - 1u))] = uint16_t((b << 7) | (k * 32u + lane));
                n_items += __popc(who);
            }
        }
        __syncwarp();
        for (uint32_t i0 = 0; i0 < n_items; i0 += 32u) {
            const uint32_t live = min(32u, n_items - i0);
            const uint32_t item = s_item[i0 + min(lane, live - 1u)];
            const uint32_t r = item & 127u, b = item >> 7;
            const uint32_t by = b >> log_bx, bx = b & ((1u << log_bx) - 1u);
            const float wx = static_cast<float>(ox + bx * kBlock) + 0.5f, wy = static_cast<float>(oy + by * kBlock) + 0.5f;
            const uint32_t at = b * uint32_t(kBlock * kBlock);
            float sum[kSums];
            if (!plain)
                walk_block<true>(s_f0[r], s_f1[r], wx, wy, s_g + at, s_gv + at, sum);
            else
                walk_block<false>(s_f0[r], s_f1[r], wx, wy, s_g + at, s_gv + at, sum);
            // A record occurs once per block: block by block the lanes' records are distinct, and a record's
            // blocks are added in order.
            const uint32_t b_last = __shfl_sync(0xffffffffu, b, 31);
            for (uint32_t now = __shfl_sync(0xffffffffu, b, 0); now <= b_last; ++now) {
                if (b == now && lane < live) {
#pragma unroll
                    for (uint32_t s = 0; s < kSums; ++s) s_acc[s * R + r] += sum[s];
                }
                __syncwarp();
            }
        }
#pragma unroll
        for (uint32_t k = 0; k < kPer; ++k) {
            const uint32_t r = k * 32u + lane;
            if (int32_t(r) >= n) continue;
            const uint32_t slot = s_slot[r];
            if (slot == 0xffffffffu) continue;
            Float8 out;
#pragma unroll
            for (uint32_t s = 0; s < kSlotValues; ++s) out.v[s] = s < kSums ? s_acc[s * R + r] : 0.f;
            store_float8(slots + size_t(slot) * kSlotValues, out);
        }
        __syncwarp();  // the batch's shared memory is rewritten
    }
}

// grads[r]: the record's slots added in tile order, its constants applied; one
// thread per record.
__global__ void __launch_bounds__(256) raster_slot_reduce_kernel(const Rec2D<float>* __restrict__ records,
                                                                 const int64_t* __restrict__ cum, size_t total,
                                                                 int64_t capacity, const int64_t* __restrict__ n_dev,
                                                                 const float* __restrict__ slots,
                                                                 Rec2D<float>* __restrict__ grads,
                                                                 float* __restrict__ v_unc) {
    const size_t r = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (r >= total) return;
    // Lists that overflowed are empty (*n_dev is 0): no slot was written, and the gradients are zero.
    if (n_dev != nullptr) capacity = min(capacity, *n_dev);
    const int64_t first = r == 0 ? 0 : min(cum[r - 1], capacity), last = min(cum[r], capacity);
    float s[kSums];
#pragma unroll
    for (uint32_t i = 0; i < kSums; ++i) s[i] = 0.f;
    for (int64_t j = first; j < last; ++j) {
        const Float8 v = load_float8(slots + size_t(j) * kSlotValues);
#pragma unroll
        for (uint32_t i = 0; i < kSums; ++i) s[i] += v.v[i];
    }
    Rec2D<float> out{};
    if (last > first) {
        const Rec2D<float> rec = as_record(load_float8(records + r));
        const float om = rec.o * rec.mu;
        const float sx = -om * s[0], sy = -om * s[1];
        out.x = -(rec.a * sx + rec.b * sy);
        out.y = -(rec.c * sy + rec.b * sx);
        out.a = 0.5f * (-om * s[2]);
        out.b = -om * s[3];
        out.c = 0.5f * (-om * s[4]);
        out.o = rec.mu * s[5];
        out.mu = rec.o * s[5];
        v_unc[r] = om * (om * s[6]);  // om^2 leaves the range of floats from 1.8e19 on
    } else {
        v_unc[r] = 0.f;
    }
    grads[r] = out;
}

int launch_tile_bwd(TileBwdGeom g, const Rec2D<float>* rec, const ushort4* rects, const float* var_q,
                    const int32_t* offsets, const int32_t* ids, const int64_t* cum, const float* v_render,
                    const float* v_render_var, float* slots, Rec2D<float>* grads, float* v_unc, cudaStream_t stream) {
    const size_t total = size_t(g.C) * g.N;
    RecordMeta* meta = reinterpret_cast<RecordMeta*>(grads);  // half of grads' bytes, read before it is written
    record_meta_kernel<<<blocks_for(int64_t(total), 256), 256, 0, stream>>>(rec, rects, cum, total, g.width, g.height,
                                                                            1u << g.log_t, meta);
    R2S_TRY(check_launch("raster_record_meta"));
    const size_t smem = 2 * (sizeof(float) << (2u * g.log_t)) +
                        kTileBwdWarps * kTileBwdBatch * (2 * sizeof(float4) + kSums * sizeof(float) +
                                                         sizeof(uint32_t) + (sizeof(uint16_t) << g.log_blocks));
    R2S_TRY(allow_dynamic_smem(raster_tile_bwd_kernel, smem));
    // A list is shared by several CTAs when there are too few lists to fill the chip: about 8192 CTAs (eleven
    // waves), as far as a warp keeps eight records. Measured on the walk without the variance terms: one view of
    // 100,000 primitives at 512^2 (1024 lists of 360) 0.112, 0.089, 0.063, 0.060 and 0.069 ms with 1, 2, 4, 8 and
    // 16 CTAs a list; 65,536 lists of 720 4.57 ms with one or two and 4.79 ms with four. A few long lists need more:
    // one view at 64^2 (16 lists of 14,000, with the variance) 0.124, 0.068 and 0.062 ms with 16, 64 and 256 CTAs a
    // list, at 100^2 (49 lists of 6,300) 0.155, 0.071 and 0.066 (60 CTAs of 64 records beat 250 of 8 on 16 lists of
    // 2,850: 0.029 / 0.031).
    const uint64_t lists = uint64_t(g.n_tiles) * g.C;
    const uint64_t mean = (g.n_dev != nullptr ? g.capacity : uint64_t(g.n_isects)) / lists;
    const uint64_t fill = (8192 + lists - 1) / lists, records = (mean + 8 * kTileBwdWarps - 1) / (8 * kTileBwdWarps);
    const unsigned split = unsigned(std::min<uint64_t>(64u, std::max<uint64_t>(1u, std::min(fill, records))));
    const dim3 grid(g.n_tiles, g.C, split);
    raster_tile_bwd_kernel<<<grid, kTileBwdThreads, smem, stream>>>(rec, meta, var_q, offsets, ids, g, v_render,
                                                                         v_render_var, slots);
    R2S_TRY(check_launch("raster_tile_bwd"));
    raster_slot_reduce_kernel<<<blocks_for(int64_t(total), 256), 256, 0, stream>>>(
        rec, cum, total, int64_t(g.capacity), g.n_dev, slots, grads, v_unc);
    return check_launch("raster_slot_reduce");
}

}  // namespace

}  // namespace r2s

using namespace r2s;

extern "C" {

int r2s_raster_tile_bwd(const float* records, const uint16_t* rects, const float* uncertainties,
                        int detach_variance, const int32_t* tile_offsets, const int32_t* flatten_ids,
                        uint64_t n_isects, const int64_t* n_used, const int64_t* tile_cum, const float* v_render,
                        const float* v_render_var, uint32_t C, uint32_t N, uint32_t width, uint32_t height,
                        uint32_t tile_size, uint32_t tiles_x, uint32_t tiles_y, float* slots, uint64_t slot_capacity,
                        float* grads, float* v_uncertainties, void* stream) {
    R2S_REQUIRE(tile_size == 8 || tile_size == 16 || tile_size == 32, R2S_ERR_UNSUPPORTED,
                "tile_size must be 8, 16 or 32");
    R2S_REQUIRE(C <= 65535, R2S_ERR_UNSUPPORTED, "camera count exceeds 65535");
    R2S_REQUIRE(uint64_t(C) * N < (uint64_t(1) << 31), R2S_ERR_UNSUPPORTED, "C*N exceeds the int32 range");
    R2S_REQUIRE(uint64_t(C) * tiles_x * tiles_y < (uint64_t(1) << 31), R2S_ERR_UNSUPPORTED, "too many tiles");
    R2S_REQUIRE(n_isects < (uint64_t(1) << 31) && slot_capacity < (uint64_t(1) << 31), R2S_ERR_UNSUPPORTED,
                "n_isects and slot_capacity must be below 2^31");
    R2S_REQUIRE(n_used != nullptr || n_isects <= slot_capacity, R2S_ERR_ARGUMENT,
                "slot_capacity must hold n_isects slots");
    if (uint64_t(C) * N == 0 || uint64_t(tiles_x) * tiles_y == 0) return R2S_OK;
    R2S_REQUIRE(records != nullptr && rects != nullptr && tile_offsets != nullptr && tile_cum != nullptr &&
                    grads != nullptr && (slots != nullptr || slot_capacity == 0) &&
                    (flatten_ids != nullptr || (n_used == nullptr && n_isects == 0)),
                R2S_ERR_ARGUMENT, "records, rects, tile_offsets, flatten_ids, tile_cum, slots and grads must be non-null");
    R2S_REQUIRE(reinterpret_cast<uintptr_t>(slots) % 32 == 0 && reinterpret_cast<uintptr_t>(records) % 32 == 0 &&
                    reinterpret_cast<uintptr_t>(grads) % 32 == 0,
                R2S_ERR_ARGUMENT, "records, slots and grads must be 32-byte aligned");
    R2S_REQUIRE(v_render_var != nullptr && v_uncertainties != nullptr, R2S_ERR_ARGUMENT,
                "v_render_var and v_uncertainties must be non-null");
    R2S_REQUIRE(width < 65536 && height < 65536, R2S_ERR_UNSUPPORTED, "image sides must be below 65536");
    const uint32_t log_t = tile_size == 8 ? 3u : tile_size == 16 ? 4u : 5u;
    const TileBwdGeom g{C, N, width, height, tiles_x, tiles_x * tiles_y, log_t, 2u * (log_t - 3u), int32_t(n_isects),
                        n_used, slot_capacity};
    const auto* rec = reinterpret_cast<const Rec2D<float>*>(records);
    const auto* rc = reinterpret_cast<const ushort4*>(rects);
    auto* out = reinterpret_cast<Rec2D<float>*>(grads);
    const float* q = detach_variance ? nullptr : uncertainties;
    cudaStream_t st = as_stream(stream);
    return launch_tile_bwd(g, rec, rc, q, tile_offsets, flatten_ids, tile_cum, v_render, v_render_var, slots, out,
                           v_uncertainties, st);
}

}  // extern "C"
