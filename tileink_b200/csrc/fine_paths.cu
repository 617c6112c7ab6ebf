// Fine stage of scenes of paths alone: one CTA of 128 threads per 16x16 tile,
// two horizontally adjacent pixels per thread (fine/main.hlsl:23-40,
// fine/interpreter.hlsli:21-219, fine/specialized.hlsli:19-45).
//
// What bounds it is its instructions: HBM is idle, and a tile's records are a
// serial chain that uses two thirds of the issue slots; for the rest the warps wait
// for fixed latencies and at the barriers between staging and compositing. A
// record's dispatch and staging are the same for the two
// pixels of a thread, the pixel arithmetic runs on f32 pairs (f32x2), and
// coverage is evaluated by half rows of fills instead of pixel by pixel.
// Against one pixel per thread with coverage in the record loop: 4.5 G against
// 8.5 G warp instructions on the 2048x2048 / 6,000-path frame, 5.8 against
// 10.1 ms; 4096x4096 / 50,000 paths 122 against 207 ms, 1283x717 / 2,500 paths
// 1.03 against 1.99 ms, 640x360 / 240 fills 0.24 against 0.29 ms.
// Four pixels per thread (64-thread CTAs) took 6.8 ms on the 2048 frame and
// eight (one warp a tile) 11.1: too few warps are in flight, and half-size
// chunks repeat the staging. The loops of the staging are not unrolled and the
// rare records are out of line (opacity groups: in an instance of their own): with
// both inline 2 of 8.9 warps per issue waited for instructions, 0.44 of 10.2 now.
//
// The tile's merged PTCL stream is processed in chunks of up to 32 records
// whose fills together reference at most kSegs tile segments (and at most
// kItems crossings and kBlocks blocks of products, below). Per chunk the CTA
// stages into shared memory:
//   - the records and each fill's solid paint (its draw's PaintInfo, decoded
//     once per upload by k_draw_tables);
//   - the chunk's segments, and for every (segment, row) crossing (dy != 0) an
//     entry with its terms of segment_row_parts (shared/coverage.hlsli:7-24),
//     listed per tile row in segment order;
//   - the partial-area products segment_area_at(x) * dy of an entry's partial
//     pixels, in zero-filled blocks of four, one product per lane;
//   - the segments that touch the tile's left edge: only they add to `base`
//     (the row edges of the others are +-0, which leave the sum unchanged).
// A lane then takes half a row of one fill (a quarter where the chunk has one or two
// fills) and accumulates base, `running` and `partial` of its pixels in segment order over the row's entries exactly as
// fill_alpha_at (shared/coverage.hlsli:34-51) does, so the f32 sums are the
// reference's; the rows are taken in order of their number of entries (2 to 3
// on average, 6 at the longest of 32 rows), so that a warp's lanes end together.
// The alphas go back to shared memory, a byte per pixel, for the record loop.
#include <cuda_runtime.h>

#include "device.cuh"
#include "fine.cuh"
#include "kernels.h"

namespace tk {
namespace {

using namespace tkd;

constexpr uint32_t kThreads = 128, kWarps = kThreads / 32;
// What a chunk holds. 7 CTAs share an SM (28 warps: 72 registers, 29 KB each).
constexpr uint32_t kRecs = 32;    // records: one per lane of the staging warp
constexpr uint32_t kCovers = 16;  // fill-like records with segments
constexpr uint32_t kSegs = 140;   // segments
constexpr uint32_t kItems = 480;  // (segment, row) crossings
constexpr uint32_t kBlocks = 560; // blocks of four partial products (block 0 is zero)
constexpr uint32_t kBuckets = 32; // rows sorted by their number of crossings

// Record classes driving the per-pixel dispatch. kClsCover: a fill-like record
// other than a plain fill, with segments in the tile.
constexpr uint32_t kClsOther = 0, kClsFill = 1, kClsUniform = 2, kClsBatch = 3, kClsEnd = 4, kClsCover = 5;
// Staged record word 0: class | flags | fill << 8 | uniform alpha << 16 | tag << 24.
constexpr uint32_t kHdrClass = 7u, kHdrEvenOdd = 8u, kHdrOpaque = 16u, kHdrGradient = 32u;
constexpr uint32_t kHdrCoverShift = 8u;    // which of the chunk's fills with segments

// A crossing entry: dy, -4 ceil(xmax) (the first pixel past the partial range,
// clamped to [0, 16]), and per group of four pixels the byte offset of its
// products' block (0: the zero block), 16 bits each.
static_assert(kSegs <= 204u && kCovers <= 32u && kItems <= 4095u && kBlocks * 16u <= 65536u, "field widths");
struct FineSmem {
    union {
        struct {  // until the entries are built
            float4 seg[kSegs];      // staged segments: p0x, p0y, p1x, p1y
            float2 sgx[kSegs];      // y_edge, slope = (p1x - p0x) / (p1y - p0y)
            uint32_t rmask[kSegs];  // rows it crosses (dy != 0) | on the left edge << 16 | group boundaries << 17
            uint16_t item[kItems];  // crossings: segment | row << 8
        };
        uint4 alpha[kCovers * TK_TILE_SIZE];  // then: coverage of a fill's row, a byte per pixel
    };
    float2 edge[kSegs];        // segments on the tile's left edge, in order: y_edge, sign
    uint4 pos[kSegs + 1];      // 16 bytes: per row, the crossings of segments before j
    uint32_t pre[kSegs + 1];   // before segment j: crossings | blocks << 12 | left-edge segments << 24
    float4 ent[kItems];        // crossing entries by row, then segment
    float4 prod[kBlocks];
    // the fills' rows by their number of entries: first entry | entries << 12 | row << 20 | fill << 24
    uint32_t rows[kCovers * TK_TILE_SIZE];
    uint32_t bucket[kBuckets];
    uint4 hdr[kRecs];          // word 0 above; positions; backdrop as float; color word
    float4 col[kRecs];         // solid paint channels as floats
    float4 uniform[kRecs];     // segment-free solid fills: the scaled source
    uint32_t seg0[kRecs];      // first segment of the record
    uint32_t off[kRecs + 1];   // staged segments before the record
    uint8_t cover[kCovers];    // the fills' records
    uint32_t n, nblk;
};

// segment_row_parts (shared/coverage.hlsli:7-24) of a segment that crosses
// tile row `row`, with the slope division done once per segment.
__device__ __forceinline__ RowParts crossing_parts(float4 g, float slope, uint32_t row) {
    const float row_y = float(row), local_y = g.y - row_y, far_y = g.w - row_y;
    const float y0 = clampf(local_y, 0.0f, 1.0f), y1 = clampf(far_y, 0.0f, 1.0f);
    const float dy = y0 - y1;
    const bool nearer_p0 = fabsf(local_y - 0.5f) <= fabsf(far_y - 0.5f);
    const float anchor_x = nearer_p0 ? g.x : g.z;
    const float anchor_y = nearer_p0 ? local_y : far_y;
    const float sx0 = mad(y0 - anchor_y, slope, anchor_x);
    const float sx1 = mad(y1 - anchor_y, slope, anchor_x);
    return {0.0f, dy, fminf(sx0, sx1), fmaxf(sx0, sx1)};
}

// Inclusive warp scan of a word (several counters that do not carry into one
// another may share it).
__device__ __forceinline__ uint32_t warp_inclusive(uint32_t v, uint32_t lane) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= uint32_t(d)) v += u;
    }
    return v;
}

// The two pixels of a thread, channel by channel.
struct Pix {
    float2 c[4];
    __device__ __forceinline__ float4 get(int p) const {
        return p ? make_float4(c[0].y, c[1].y, c[2].y, c[3].y) : make_float4(c[0].x, c[1].x, c[2].x, c[3].x);
    }
    __device__ __forceinline__ void set(int p, float4 v) {
        (p ? c[0].y : c[0].x) = v.x;
        (p ? c[1].y : c[1].x) = v.y;
        (p ? c[2].y : c[2].x) = v.z;
        (p ? c[3].y : c[3].x) = v.w;
    }
};

// Pair arithmetic with each operation rounded on its own. A product is a fused
// multiply-add of -0, which leaves its rounding and sign alone; `nz` comes from
// the launch, so that no product is contracted with the sum that follows it.
__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b, float2 nz) { return __ffma2_rn(a, b, nz); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
constexpr float kTwo23 = 8388608.0f;
// floor of values in [0, 2^22] (f2u's truncation, kept as a float)
__device__ __forceinline__ float2 floor2(float2 v) { return add2(__fadd2_rd(v, both(kTwo23)), both(-kTwo23)); }

// coverage_to_alpha of four coverage sums, a byte each. The even-odd fold
// v - 2 round(v / 2) runs for both rules, times `fold` (2, or 0 for nonzero),
// with the rounding by addition of 1.5 * 2^23: exact below 2^22.
__device__ __forceinline__ uint32_t coverage_bytes(const float2 (&v)[2], float fold, float2 nz) {
    uint32_t b[4];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const float2 half = add2(add2(mul2(v[q], both(0.5f), nz), both(1.5f * kTwo23)), both(-1.5f * kTwo23));
        const float2 u = __ffma2_rn(half, both(-fold), v[q]);
        const float2 a = make_float2(fminf(fabsf(u.x), 1.0f), fminf(fabsf(u.y), 1.0f));
        const float2 y = __fadd2_rd(add2(mul2(a, both(255.0f), nz), both(0.5f)), both(kTwo23));
        b[2 * q] = __float_as_uint(y.x);
        b[2 * q + 1] = __float_as_uint(y.y);
    }
    return __byte_perm(__byte_perm(b[0], b[1], 0x0040), __byte_perm(b[2], b[3], 0x0040), 0x5410);
}

// The bucket of a row with c entries: exact up to 16, then in fours.
__device__ __forceinline__ uint32_t bucket_of(uint32_t c) { return c < 16u ? c : min(16u + ((c - 16u) >> 2), kBuckets - 1u); }

// Whether the crossings and blocks of a prefix word fit the shared arrays.
__device__ __forceinline__ bool stage_fits(uint32_t pre) {
    return (pre & 0xFFFu) <= kItems && ((pre >> 12) & 0xFFFu) < kBlocks;
}

// The coverage of the fills' rows, 16 / PARTS pixels per lane. Sliced: those of a single
// record's slice, thread PARTS r + h part h of row r; its sums start from `carry` when carried
// and end there when it is not the last slice (partly).
// Quarter rows spend a quarter more instructions a row than half rows, but one or two
// fills' half rows leave two or three of the four warps idle: with quarters there,
// 2048x2048 / 6,000 paths 6.1 -> 5.8 ms, 640x360 / 240 fills 0.26 -> 0.245, 96x80 / 8 paths
// of 5,000 lines (slices) 2.4 -> 2.1, and 1.78 with the largest slices that fit.
template <uint32_t PARTS>
__device__ __forceinline__ void cover_rows(FineSmem& S, uint32_t fills, uint32_t total, uint32_t first, bool sliced,
                                           bool carried, bool partly, float2 nz, float2 (&carry)[5]) {
    constexpr uint32_t kPairs = TK_TILE_SIZE / PARTS / 2u;  // pixel pairs of a lane
    const uint32_t tid = threadIdx.x;
    const uint32_t rows0 = __shfl_sync(0xffffffffu, first, (tid / PARTS) & 15u);  // the first entry of row tid / PARTS, when sliced
    const unsigned char* prod = reinterpret_cast<const unsigned char*>(S.prod);
#pragma unroll 1
    for (uint32_t ci = tid; ci < fills * TK_TILE_SIZE * PARTS; ci += kThreads) {
        const uint32_t part = ci % PARTS;
        uint32_t w = S.rows[ci / PARTS];
        if (PARTS == 4u && sliced) {
            const unsigned char* at = reinterpret_cast<const unsigned char*>(S.pos) + ci / PARTS;
            w = rows0 | (uint32_t(at[total * TK_TILE_SIZE] - at[0]) << 12) | ((ci / PARTS) << 20);
        }
        const uint32_t f = w >> 24, r = (w >> 20) & 15u;
        const uint4 h = S.hdr[S.cover[f]];
        float base = PARTS == 4u && carried ? carry[4].x : __uint_as_float(h.z);
#pragma unroll 1
        for (uint32_t e = (h.y >> 16) & 255u, e1 = h.y >> 24; e < e1; ++e)
            base += S.edge[e].y * clampf(float(r) - S.edge[e].x + 1.0f, 0.0f, 1.0f);
        float2 running[kPairs], partial[kPairs];
#pragma unroll
        for (uint32_t q = 0; q < kPairs; ++q) {
            running[q] = partial[q] = make_float2(0.0f, 0.0f);
            if (PARTS == 4u && carried) {
                running[q] = carry[q];
                partial[q] = carry[q + 2u];
            }
        }
        const float x4 = 2.0f + float(part) * (64.0f / PARTS);
        const float4* e = S.ent + (w & 0xFFFu);
        const float4* const e1 = e + ((w >> 12) & 255u);
#pragma unroll 1
        for (; e < e1; ++e) {
            const float4 c = *e;
            const uint32_t o = __float_as_uint(part >= PARTS / 2u ? c.w : c.z);
            const float t = c.y + x4;
#pragma unroll
            for (uint32_t q = 0; q < kPairs; ++q) {
                // 1 for pixels x >= phi, else 0: clamp(4 (x - phi) + 2, 0, 1)
                const float2 m = make_float2(__saturatef(t + 8.0f * float(q)), __saturatef(t + (8.0f * float(q) + 4.0f)));
                running[q] = __ffma2_rn(both(c.x), m, running[q]);  // + dy or + 0
            }
#pragma unroll
            for (uint32_t q = 0; q < kPairs; q += 2u) {
                const uint32_t at = PARTS == 4u ? (part & 1u ? o >> 16 : o & 0xFFFFu) : (q ? o >> 16 : o & 0xFFFFu);
                const float4 p = *reinterpret_cast<const float4*>(prod + at);
                partial[q] = add2(partial[q], make_float2(p.x, p.y));
                partial[q + 1u] = add2(partial[q + 1u], make_float2(p.z, p.w));
            }
        }
        if (PARTS == 4u && partly) {
            carry[4].x = base;
#pragma unroll
            for (uint32_t q = 0; q < 2u; ++q) {
                carry[q] = running[q];
                carry[q + 2u] = partial[q];
            }
            continue;
        }
        const bool even_odd = (h.x & kHdrEvenOdd) != 0u;
#pragma unroll
        for (uint32_t g = 0; g < kPairs / 2u; ++g) {
            float2 v[2];
            v[0] = add2(add2(both(base), running[2 * g]), partial[2 * g]);
            v[1] = add2(add2(both(base), running[2 * g + 1]), partial[2 * g + 1]);
            uint32_t word;
            if (even_odd && fabsf(base) > 1.0e6f) {  // windings that coverage_bytes does not fold
                word = coverage_to_alpha(v[0].x, 1u) | (coverage_to_alpha(v[0].y, 1u) << 8) |
                       (coverage_to_alpha(v[1].x, 1u) << 16) | (coverage_to_alpha(v[1].y, 1u) << 24);
            } else {
                word = coverage_bytes(v, even_odd ? 2.0f : 0.0f, nz);
            }
            reinterpret_cast<uint32_t*>(S.alpha)[((f * TK_TILE_SIZE + r) * PARTS + part) * (kPairs / 2u) + g] = word;
        }
    }
}

// Stages the crossing entries and products of the chunk's first n records,
// whose `total` segments are staged, and the coverage alphas of their fills;
// `n` and `total` become the records and segments that the shared arrays hold.
// A single record (n == 1) is taken in as many slices of its segments as it
// needs: `before` are done already and `left` are not, and `carry` holds the sums from
// slice to slice (cover_rows; its alphas count after the last).
__device__ __forceinline__ void stage_coverage(FineSmem& S, uint32_t& n, uint32_t& total, uint32_t before,
                                               uint32_t left, float2 nz, float2 (&carry)[5]) {
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    // Prefixes over the segments: four words of four row counters (bytes), and
    // one of crossings, product blocks (what a segment can need: one per row and
    // one per group boundary it passes) and left-edge segments, dealt out to the
    // warps. A lane takes kPer consecutive segments, so that one warp scan does
    // (a scan for every 32 segments: 6.3 instead of 6.1 ms on the 2048 frame).
    constexpr uint32_t kPer = (kSegs + 31u) / 32u;
#pragma unroll 1
    for (uint32_t t = warp; t < 5u; t += kWarps) {
        uint32_t v[kPer], sum = 0u;
#pragma unroll
        for (uint32_t q = 0; q < kPer; ++q) {
            const uint32_t j = lane * kPer + q, m = j < total ? S.rmask[j] : 0u;
            v[q] = sum;
            sum += t < 4u ? (((m >> (4u * t)) & 15u) * 0x00204081u) & 0x01010101u
                          : uint32_t(__popc(m & 0xFFFFu)) * 0x1001u + ((m >> 17) << 12) + ((m & 0x10000u) << 8);
        }
        const uint32_t before_lane = warp_inclusive(sum, lane) - sum;
#pragma unroll
        for (uint32_t q = 0; q < kPer; ++q) {
            const uint32_t j = lane * kPer + q;
            if (j <= total) {  // the one past the last holds the totals
                if (t < 4u) reinterpret_cast<uint32_t*>(&S.pos[j])[t] = before_lane + v[q];
                else S.pre[j] = before_lane + v[q];
            }
        }
    }
    __syncthreads();
    const unsigned char* pos = reinterpret_cast<const unsigned char*>(S.pos);
    uint32_t fills, first;
    for (;;) {
        // the records whose crossings and blocks fit (their number grows with the record)
        if (n > 1u) {
            const bool fit = lane < n && stage_fits(S.pre[S.off[lane + 1u]]);
            n = max(uint32_t(__popc(__ballot_sync(0xffffffffu, fit))), 1u);
            total = S.off[n];
        }
        // one record: the largest slice whose crossings and blocks fit (one segment's do)
        if (n == 1u && !stage_fits(S.pre[total])) {
            uint32_t fit = 1u;
            while (total - fit > 1u) {
                const uint32_t mid = (fit + total) >> 1;
                if (stage_fits(S.pre[mid])) fit = mid;
                else total = mid;
            }
            total = fit;
        }
        const uint32_t items = S.pre[total] & 0xFFFu;
        const uint32_t count = lane < TK_TILE_SIZE ? pos[total * TK_TILE_SIZE + lane] : 0u;
        first = warp_inclusive(count, lane) - count;  // the first entry of tile row `lane`
#pragma unroll 1
        for (uint32_t j = tid; j < total; j += kThreads) {
            const uint32_t rm = S.rmask[j], pr = S.pre[j];
            uint32_t o = pr & 0xFFFu;
#pragma unroll 1
            for (uint32_t m = rm & 0xFFFFu; m; m &= m - 1u) S.item[o++] = uint16_t(j | ((__ffs(m) - 1) << 8));
            if (rm & 0x10000u) S.edge[pr >> 24] = make_float2(S.sgx[j].x, signum_f32(S.seg[j].z - S.seg[j].x));
        }
        const uint32_t hx = lane < n ? S.hdr[lane].x : 0u, cls = hx & kHdrClass;
        const bool covers = cls == kClsFill || cls == kClsCover;
        fills = __popc(__ballot_sync(0xffffffffu, covers));
        if (tid < 32u && covers) {
            const uint32_t j0 = S.off[tid], j1 = n == 1u ? total : S.off[tid + 1u];
            S.hdr[tid].y = j0 | (j1 << 8) | ((S.pre[j0] >> 24) << 16) | (S.pre[j1] & 0xFF000000u);
            S.cover[(hx >> kHdrCoverShift) & 31u] = uint8_t(tid);
        }
        if (tid < kBuckets) S.bucket[tid] = 0u;
        if (tid == 0) {
            S.nblk = 1u;
            S.prod[0] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        __syncthreads();
#pragma unroll 1
        for (uint32_t it0 = warp * 32u; it0 < items; it0 += kThreads) {
            const uint32_t it = it0 + lane;
            const bool live = it < items;
            const uint32_t word = live ? S.item[it] : 0u;
            const uint32_t j = word & 255u, r = word >> 8;
            const RowParts rp = crossing_parts(S.seg[j], S.sgx[j].y, r);
            const uint32_t plo = uint32_t(min(max(__float2int_rd(rp.xmin), 0), int32_t(TK_TILE_SIZE)));
            const uint32_t phi = uint32_t(min(max(__float2int_ru(rp.xmax), 0), int32_t(TK_TILE_SIZE)));
            const uint32_t span = live && phi > plo ? phi - plo : 0u;
            const uint32_t g0 = plo >> 2, blocks = span ? ((phi - 1u) >> 2) - g0 + 1u : 0u;
            // one pixel, crossed from top to bottom: segment_area_at's second form
            const float x0 = rp.xmin - float(plo), x1 = rp.xmax - float(plo);
            const bool inside = span == 1u && x0 >= 0.0f && x1 <= 1.0f && x1 - x0 != 0.0f;
            const uint32_t dealt = inside ? 0u : span;  // products that the warp deals out below
            // one scan for both: blocks and products
            const uint32_t both = warp_inclusive(blocks | (dealt << 16), lane);
            const uint32_t sums = __shfl_sync(0xffffffffu, both, 31);
            uint32_t base = 0u;
            if (lane == 0) base = atomicAdd(&S.nblk, sums & 0xFFFFu);
            base = __shfl_sync(0xffffffffu, base, 0);
            if (base + (sums & 0xFFFFu) > kBlocks) continue;  // does not fit: the chunk is cut below
            const uint32_t b0 = base + (both & 0xFFFFu) - blocks;
#pragma unroll 1
            for (uint32_t b = 0; b < blocks; ++b) S.prod[b0 + b] = make_float4(0.f, 0.f, 0.f, 0.f);
            float* const prod = reinterpret_cast<float*>(S.prod) + (b0 - g0) * 4u;
            if (inside) prod[plo] = mad(-0.5f, x0 + x1, 1.0f) * rp.dy;
            const uint32_t rfirst = __shfl_sync(0xffffffffu, first, r);
            if (live) {
                // offsets of groups g0 .. g0 + blocks - 1
                const uint32_t o = b0 * 16u;
                uint32_t w0 = 0u, w1 = 0u;
                if (blocks) w0 = o;
                if (blocks > 1u) w0 |= (o + 16u) << 16;
                if (blocks > 2u) w1 = o + 32u;
                if (blocks > 3u) w1 |= (o + 48u) << 16;
                const uint64_t w = (uint64_t(w1) << 32 | w0) << (16u * (g0 & 3u));
                S.ent[rfirst + pos[j * TK_TILE_SIZE + r]] =
                    make_float4(rp.dy, -4.0f * float(phi), __uint_as_float(uint32_t(w)), __uint_as_float(uint32_t(w >> 32)));
            }
            __syncwarp();
            // the round's products, one per lane: lane l owns products [ends(l) - dealt(l), ends(l))
            const uint32_t ends = both >> 16, products = sums >> 16, place = (b0 - g0) * 4u, shift = plo - (ends - dealt);
#pragma unroll 1
            for (uint32_t p0 = 0; p0 < products; p0 += 32u) {
                const uint32_t p = p0 + lane;
                uint32_t l = 0u;  // the first lane with ends > p
#pragma unroll
                for (uint32_t s = 16u; s; s >>= 1) {
                    const uint32_t v = __shfl_sync(0xffffffffu, ends, l + s - 1u);
                    if (v <= p) l += s;
                }
                const float xmin = __shfl_sync(0xffffffffu, rp.xmin, l), xmax = __shfl_sync(0xffffffffu, rp.xmax, l);
                const float dy = __shfl_sync(0xffffffffu, rp.dy, l);
                const uint32_t at = __shfl_sync(0xffffffffu, place, l);
                const uint32_t x = __shfl_sync(0xffffffffu, shift, l) + p;
                if (p < products) reinterpret_cast<float*>(S.prod)[at + x] = segment_area_at(xmin, xmax, x) * dy;
            }
        }
        // the fills' rows, counted by their number of entries
        constexpr uint32_t kPer = (kCovers * TK_TILE_SIZE + kThreads - 1u) / kThreads;
        uint32_t place[kPer], ranked[kPer];
#pragma unroll
        for (uint32_t k = 0; k < kPer; ++k) {
            const uint32_t ci = k * kThreads + tid, f = ci >> 4, r = ci & 15u;
            const uint32_t rfirst = __shfl_sync(0xffffffffu, first, r);
            place[k] = ranked[k] = 0u;
            if (f < fills) {
                const uint32_t y = S.hdr[S.cover[f]].y;
                const uint32_t k0 = pos[(y & 255u) * TK_TILE_SIZE + r], k1 = pos[((y >> 8) & 255u) * TK_TILE_SIZE + r];
                place[k] = (rfirst + k0) | ((k1 - k0) << 12) | (r << 20) | (f << 24);
                ranked[k] = atomicAdd(&S.bucket[bucket_of(k1 - k0)], 1u);
            }
        }
        __syncthreads();
        if (S.nblk <= kBlocks) {
            const uint32_t c = lane < kBuckets ? S.bucket[lane] : 0u;
            const uint32_t start = warp_inclusive(c, lane) - c;
#pragma unroll
            for (uint32_t k = 0; k < kPer; ++k) {
                const uint32_t at = __shfl_sync(0xffffffffu, start, bucket_of((place[k] >> 12) & 255u));
                if (((k * kThreads + tid) >> 4) < fills) S.rows[at + ranked[k]] = place[k];
            }
            break;
        }
        // a crossing rounded into another group than its segment: cut the chunk (a
        // segment alone has at most 16 x 4 blocks)
        if (n == 1u) {
            total >>= 1;
        } else {
            n >>= 1;
            total = S.off[n];
        }
        __syncthreads();
    }
    __syncthreads();
    // fill_alpha_at's coverage sums and coverage_to_alpha: half a fill's row per lane, or a
    // quarter where there are too few fills for the CTA's threads
    const bool partly = n == 1u && total < (before != 0u ? left : S.off[1]), sliced = n == 1u && (partly || before != 0u);
    if (fills > 2u) {
        cover_rows<2>(S, fills, total, first, false, false, false, nz, carry);
    } else {
        cover_rows<4>(S, fills, total, first, sliced, sliced && before != 0u, partly, nz, carry);
    }
    __syncthreads();
}

// Composites two premultiplied colours (channels 0..255 as float pairs) scaled
// by their masked alphas (0..255) over two pixels: scale_premul_u8_to_unorm and
// src_over_premul_unorm (shared/pixel.hlsli). `scale` is alpha / 65025, or
// 1 / 255 where an opaque colour covers the pixel (it then replaces it: the
// weight of px is 0 and the sum exact), or 0 where nothing is drawn.
__device__ __forceinline__ void composite(Pix& px, const float2 (&col)[4], float2 scale, float2 nz) {
    const float2 s3 = mul2(col[3], scale, nz);
    const float2 k = __ffma2_rn(s3, both(-1.0f), both(1.0f));
#pragma unroll
    for (int c = 0; c < 3; ++c) px.c[c] = add2(mul2(col[c], scale, nz), mul2(px.c[c], k, nz));
    px.c[3] = add2(s3, mul2(px.c[3], k, nz));
}

// A solid colour's masked coverage over px (the brush branch of
// fine/interpreter.hlsli's fill handling, fine/draw.hlsli:16-21).
__device__ __forceinline__ void paint_solid(float4 c, bool opaque, float2 alpha, float2 nz, Pix& px) {
    if (c.w == 0.0f) return;
    const float2 col[4] = {both(c.x), both(c.y), both(c.z), both(c.w)};
    float2 scale = mul2(alpha, both(1.0f / 65025.0f), nz);
    if (opaque) {
        if (alpha.x == 255.0f) scale.x = CHANNEL_SCALE;
        if (alpha.y == 255.0f) scale.y = CHANNEL_SCALE;
    }
    composite(px, col, scale, nz);
}

__device__ __forceinline__ float4 channels(uint32_t c) {
    return make_float4(float(c & 255u), float((c >> 8) & 255u), float((c >> 16) & 255u), float(c >> 24));
}
// Byte B of a word as 2^23 + its value.
template <int B>
__device__ __forceinline__ float big_byte(uint32_t w) {
    return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7650u | B));
}

// Pixel by pixel: the brushes that paint_gradient does not evaluate itself.
__device__ __noinline__ void paint_brush(const PaintInfo* pi, const Paint P, float cx, float cy, float2 alpha, Pix& px) {
#pragma unroll 1
    for (int p = 0; p < 2; ++p) {
        const uint32_t masked = uint32_t(p ? alpha.y : alpha.x);
        if (masked == 0u) continue;
        const uint32_t c = gradient_at<false>(pi->g, pi->gk, P, cx + float(p), cy);
        if (masked == 255u && premul_u8_is_opaque(c)) px.set(p, rgba8_to_unorm(c));
        else px.set(p, src_over_premul_unorm(px.get(p), scale_premul_u8_to_unorm(c, masked)));
    }
}

// a / b for two dividends of one divisor
__device__ __forceinline__ float2 divide_both(float2 a, float b, float rcp_b, bool fast, float2 nz) {
    if (fast && dividend_is_plain(a.x) && dividend_is_plain(a.y)) {
        const float2 r = both(rcp_b), m = both(-b);
        float2 q = mul2(a, r, nz);
        q = __ffma2_rn(__ffma2_rn(q, m, a), r, q);
        return __ffma2_rn(__ffma2_rn(q, m, a), r, q);
    }
    return make_float2(a.x / b, a.y / b);
}

// The brush colours of the two pixels over px, painted where alpha is not 0.
// Linear and radial gradients evaluate sample_gradient (fine/paint.hlsli:40-96)
// and the ramp's interpolation (lerp_premul_u8) on the pair, with the channels
// kept as floats.
__device__ __forceinline__ void paint_gradient(const PaintInfo* __restrict__ pi, const Paint& P, float cx, float cy,
                                               float2 alpha, float2 nz, Pix& px) {
    const uint4 k = __ldg(&pi->gk);
    const uint32_t code = k.x & 255u, extend = k.w;
    if (!(k.x & kGradRampOk)) {
        if (code == kGradConst) {
            paint_solid(channels(k.y), premul_u8_is_opaque(k.y), alpha, nz, px);
        } else {
            Pix copy = px;  // the call takes its address
            paint_brush(pi, P, cx, cy, alpha, copy);
            px = copy;
        }
        return;
    }
    if (alpha.x == 0.0f && alpha.y == 0.0f) return;
    const float4* const gv = reinterpret_cast<const float4*>(pi->g);
    const float4 ga = __ldg(gv + 3), gb = __ldg(gv + 4), gc = __ldg(gv + 5);  // g[12..23]
    const uint32_t last = k.z - 1u;
    const float flast = float(last);
    const uint32_t* __restrict__ ramp = P.words + k.y;
    const bool fast = (k.x & kGradFast) != 0u;
    float2 tx = make_float2(cx, cx + 1.0f), ty = both(cy);
    if (!(k.x & kGradIdentity)) {
        const float4 m0 = __ldg(gv), m1 = __ldg(gv + 1), m2 = __ldg(gv + 2);
        const float2 x = __ffma2_rn(both(m0.x), tx, both(mad(m0.z, cy, m1.x)));
        const float2 y = __ffma2_rn(both(m0.y), tx, both(mad(m0.w, cy, m1.y)));
        tx = __ffma2_rn(both(m1.z), x, __ffma2_rn(both(m2.x), y, both(m2.z)));
        ty = __ffma2_rn(both(m1.w), x, __ffma2_rn(both(m2.y), y, both(m2.w)));
    }
    const float2 qx = add2(tx, both(-ga.x)), qy = add2(ty, both(-ga.y));
    float2 t = make_float2(0.0f, 0.0f);
    bool none0 = false, none1 = false;
    if (code == kGradLinear) {
        if (k.x & kGradDenOk)
            t = divide_both(__ffma2_rn(qx, both(ga.z), mul2(qy, both(ga.w), nz)), gb.x, gb.y, fast, nz);
    } else {
        const float2 b = mul2(both(-2.0f), __ffma2_rn(qx, both(ga.z), __ffma2_rn(qy, both(ga.w), both(gb.x))), nz);
        const float2 c = __ffma2_rn(qx, qx, __ffma2_rn(qy, qy, both(gb.y)));
        const float dr = gc.y, sr = gc.z;
        if (k.x & kGradASmall) {
            t = make_float2(-c.x / b.x, -c.y / b.y);
            none0 = !(fabsf(b.x) > RADIAL_QUADRATIC_EPSILON && mad(t.x, dr, sr) >= 0.0f);
            none1 = !(fabsf(b.y) > RADIAL_QUADRATIC_EPSILON && mad(t.y, dr, sr) >= 0.0f);
        } else {
            const float2 disc = __ffma2_rn(b, b, mul2(both(gb.w), c, nz));
            const float2 root = make_float2(sqrtf(disc.x >= 0.0f ? disc.x : 1.0f), sqrtf(disc.y >= 0.0f ? disc.y : 1.0f));
            const float2 mb = make_float2(-b.x, -b.y), mr = make_float2(-root.x, -root.y);
            const float2 t0 = divide_both(add2(mb, mr), gc.x, gc.w, fast, nz);
            const float2 t1 = divide_both(add2(mb, root), gc.x, gc.w, fast, nz);
            const float2 e0 = __ffma2_rn(t0, both(dr), both(sr)), e1 = __ffma2_rn(t1, both(dr), both(sr));
            const bool v00 = e0.x >= 0.0f, v10 = e1.x >= 0.0f, v01 = e0.y >= 0.0f, v11 = e1.y >= 0.0f;
            none0 = !(disc.x >= 0.0f) || !(v00 || v10);
            none1 = !(disc.y >= 0.0f) || !(v01 || v11);
            t.x = v00 ? (v10 ? fmaxf(t0.x, t1.x) : t0.x) : t1.x;
            t.y = v01 ? (v11 ? fmaxf(t0.y, t1.y) : t0.y) : t1.y;
        }
    }
    // sample_ramp (shared/brush/*.hlsli); a coordinate that is not a number stores 0
    float2 ext = make_float2(__saturatef(t.x), __saturatef(t.y));
    if (extend == TK_EXTEND_REPEAT || extend == TK_EXTEND_REFLECT) {
        if (fabsf(t.x) < 4.0e6f && fabsf(t.y) < 4.0e6f) {
            // apply_extend's remainders, the floors by rounding down at 2^23 (halves exact)
            const bool repeat = extend == TK_EXTEND_REPEAT;
            const float2 h = mul2(t, both(repeat ? 1.0f : 0.5f), nz);
            const float2 f = add2(__fadd2_rd(h, both(1.5f * kTwo23)), both(-1.5f * kTwo23));
            ext = __ffma2_rn(f, both(repeat ? -1.0f : -2.0f), t);
            if (!repeat) {
                const float2 back = __ffma2_rn(ext, both(-1.0f), both(2.0f));
                ext = make_float2(fminf(ext.x, back.x), fminf(ext.y, back.y));
            }
        } else {
            ext = make_float2(apply_extend(t.x, extend), apply_extend(t.y, extend));
        }
        none0 = none0 || !(ext.x <= 1.0f);
        none1 = none1 || !(ext.y <= 1.0f);
        if (none0) ext.x = 0.0f;
        if (none1) ext.y = 0.0f;
    }
    // The texel pair (i, i + 1) with i <= last - 1: at the ramp's end the
    // fraction is 1 instead of a next texel's 0. A fraction within 1e-4 of
    // 0 or 1 rounds to that texel, as the reference's test for it does.
    const float2 pos = mul2(ext, both(flast), nz);
    const uint32_t i0 = min(f2u(pos.x), last - 1u), i1 = min(f2u(pos.y), last - 1u);
    const uint32_t l0 = __ldg(ramp + i0), r0 = __ldg(ramp + i0 + 1u);
    const uint32_t l1 = __ldg(ramp + i1), r1 = __ldg(ramp + i1 + 1u);
    const float2 frac = __ffma2_rn(ext, both(flast), make_float2(-float(i0), -float(i1)));
    const auto mix = [&](float la, float lb, float ra, float rb) {
        const float2 l = make_float2(la, lb);  // 2^23 + byte
        const float2 d = __ffma2_rn(l, both(-1.0f), make_float2(ra, rb));
        return floor2(add2(__ffma2_rn(d, frac, add2(l, both(-kTwo23))), both(0.5f)));
    };
    float2 col[4];
    col[0] = mix(big_byte<0>(l0), big_byte<0>(l1), big_byte<0>(r0), big_byte<0>(r1));
    col[1] = mix(big_byte<1>(l0), big_byte<1>(l1), big_byte<1>(r0), big_byte<1>(r1));
    col[2] = mix(big_byte<2>(l0), big_byte<2>(l1), big_byte<2>(r0), big_byte<2>(r1));
    col[3] = mix(big_byte<3>(l0), big_byte<3>(l1), big_byte<3>(r0), big_byte<3>(r1));
    // nothing where the colour's alpha is 0 (else it is 1 or more, and the scale below 1)
    float2 scale = mul2(alpha, both(1.0f / 65025.0f), nz);
    const float2 full = mul2(alpha, col[3], nz);
    scale.x = fminf(full.x == 65025.0f ? CHANNEL_SCALE : scale.x, none0 ? 0.0f : col[3].x);
    scale.y = fminf(full.y == 65025.0f ? CHANNEL_SCALE : scale.y, none1 ? 0.0f : col[3].y);
    composite(px, col, scale, nz);
}

// Stored texels (RGBA8 UNORM: loads are k / 255, stores round to nearest even).
// k / 255 by one correction of k * fl(1/255) (divide_by's step), exact for
// every byte.
__device__ __forceinline__ float2 unorm_of_byte(float2 k, float2 nz) {
    const float2 q = mul2(k, both(CHANNEL_SCALE), nz);
    return __ffma2_rn(__ffma2_rn(q, both(-255.0f), k), both(CHANNEL_SCALE), q);
}
// unorm8_store's byte as 2^23 + its value
__device__ __forceinline__ float2 byte_of_unorm(float2 v, float2 nz) {
    return add2(mul2(make_float2(__saturatef(v.x), __saturatef(v.y)), both(255.0f), nz), both(kTwo23));
}

// combine_alpha of the two bytes of a and b
__device__ __forceinline__ uint32_t combine_bytes(uint32_t a, uint32_t b) {
    return combine_alpha(a & 255u, b & 255u) | (combine_alpha(a >> 8, b >> 8) << 8);
}

struct FineArgs {
    const tk_tile_record* tiles;
    const tk_ptcl_record* ptcl;
    const SegmentRec* segments;
    const PaintInfo* paints;
    const uint32_t* brush;
    uint64_t brush_words;
    uint64_t seg_capacity;
    uint32_t* target;
    uint32_t width, height, tw;
    uint32_t* error;
    const BatchScene* scenes;
    const uint32_t* tile_scene;
    const uint32_t* tile_list;
    float2 nz;  // -0, -0: see mul2
};

// An open opacity group: the two pixels' state before it.
struct Group {
    uint32_t kind, payload, parent_clip, layer_alpha;
    float4 parent[2];
};

// Opacity groups and clipped colours, pixel by pixel. Returns the group depth after the
// record.
template <bool GROUPS>
__device__ __forceinline__ uint32_t rare_record(uint32_t* error, uint32_t tag, uint32_t payload, uint32_t clip,
                                             uint32_t alpha, Group* groups, uint32_t gdepth, Pix& px) {
    if (GROUPS && (tag == TK_PTCL_BEGIN_OPACITY || tag == TK_PTCL_BEGIN_BLEND)) {
        if (gdepth >= kGroupDepth) {
            atomicOr(error, ERR_STACK_DEPTH);
            return gdepth;
        }
        // Parents beyond the local slots are kept as RGBA8
        // (fine/group.hlsli:21-36).
        Group& v = groups[gdepth];
        v.kind = tag;
        v.payload = payload;
        v.parent_clip = clip;
        v.layer_alpha = alpha;
        for (int p = 0; p < 2; ++p) {
            const float4 parent = px.get(p);
            v.parent[p] = gdepth < kGroupLocal ? parent : rgba8_to_unorm(unorm_to_rgba8(parent));
            px.set(p, make_float4(0.f, 0.f, 0.f, 0.f));
        }
        return gdepth + 1u;
    }
    if (GROUPS && (tag == TK_PTCL_END_OPACITY || tag == TK_PTCL_END_BLEND)) {
        if (gdepth == 0u) return 0u;
        const Group& v = groups[--gdepth];
        if (v.kind == TK_PTCL_BEGIN_OPACITY) {
            const uint32_t m = combine_bytes(v.layer_alpha, v.parent_clip);
            for (int p = 0; p < 2; ++p) {
                const uint32_t a = combine_alpha((m >> (8 * p)) & 255u, v.payload);
                px.set(p, src_over_premul_unorm(v.parent[p], scale_premul_u8_to_unorm(unorm_to_rgba8(px.get(p)), a)));
            }
        }
        return gdepth;
    }
    if (tag == TK_PTCL_COLOR) {
        for (int p = 0; p < 2; ++p) {
            const uint32_t m = (clip >> (8 * p)) & 255u;
            if (m == 255u && premul_u8_is_opaque(payload)) px.set(p, rgba8_to_unorm(payload));
            else if (m != 0u) px.set(p, src_over_premul_unorm(px.get(p), scale_premul_u8_to_unorm(payload, m)));
        }
    } else if (tag != TK_PTCL_END && tag < TK_PTCL_BATCH_BEGIN) {
        atomicOr(error, ERR_UNSUPPORTED);  // SDF shapes, images and text take fine.cu's kernel
    }
    return gdepth;
}
__device__ __noinline__ void rare_plain(uint32_t* error, uint32_t tag, uint32_t payload, uint32_t clip, Pix& px) {
    rare_record<false>(error, tag, payload, clip, 0u, nullptr, 0u, px);
}

// GROUPS: the scene has opacity layers. Their records are handled in the loop then: by a
// call, with the pixels and groups through local memory, they took 0.119 ms on 1000x800 /
// 800 blobs in pairs of layers, a pixel per thread 0.105, 0.076 this way. In the loop of
// scenes without them the same code would cost 6% (2048x2048: 5.83 -> 6.2 ms).
template <bool GROUPS>
__global__ void __launch_bounds__(kThreads, 7) k_fine_paths(const FineArgs a) {
    __shared__ FineSmem S;
    const uint32_t tile = a.tile_list ? a.tile_list[blockIdx.x] : blockIdx.x;
    const tk_tile_record rec = a.tiles[tile];
    if (rec.ptcl_start >= rec.ptcl_end) return;
    uint32_t ltile = tile, tw = a.tw, width = a.width, height = a.height;
    uint32_t* target = a.target;
    if (a.scenes) {  // batched pass: this tile's canvas and image
        const BatchScene& sc = a.scenes[a.tile_scene[tile]];
        ltile = tile - sc.tile_base;
        tw = sc.tw;
        width = sc.width;
        height = sc.height;
        target += sc.image_offset;
    }
    const float2 nz = a.nz;
    const uint32_t tid = threadIdx.x;
    const uint32_t column = tid % 8u, row = tid / 8u;  // pixels 2 column and 2 column + 1 of the row
    const uint32_t gx = (ltile % tw) * TK_TILE_SIZE + 2u * column, gy = (ltile / tw) * TK_TILE_SIZE + row;
    const bool in0 = gy < height && gx < width, in1 = gy < height && gx + 1u < width;
    uint32_t* const texel = target + (uint64_t(gy) * width + gx);
    const float cx = float(gx) + 0.5f, cy = float(gy) + 0.5f;
    const Paint P{a.brush, a.brush_words, nullptr};
    Pix px;
    {
        const uint32_t t0 = in0 ? texel[0] : 0u, t1 = in1 ? texel[1] : 0u;
        const float2 m = both(-kTwo23);
        px.c[0] = unorm_of_byte(add2(make_float2(big_byte<0>(t0), big_byte<0>(t1)), m), nz);
        px.c[1] = unorm_of_byte(add2(make_float2(big_byte<1>(t0), big_byte<1>(t1)), m), nz);
        px.c[2] = unorm_of_byte(add2(make_float2(big_byte<2>(t0), big_byte<2>(t1)), m), nz);
        px.c[3] = unorm_of_byte(add2(make_float2(big_byte<3>(t0), big_byte<3>(t1)), m), nz);
    }

    // The clip masks of the two pixels, a byte each. The record stream is the
    // same for all threads, so the depth is too, and depth 0 means 255.
    uint32_t clip = 0xFFFFu, cstack[kClipSpill + 4u];
    uint32_t cdepth = 0u, gdepth = 0u;
    Group groups[GROUPS ? kGroupDepth : 1u];
    uint32_t mode = TK_TILE_KIND_INTERPRETER;
    float2 carry[5];

    uint64_t r = rec.ptcl_start;
    const uint64_t end = rec.ptcl_end;
    bool done = false;
#pragma unroll 1
    while (r < end && !done) {
        // ---- stage a chunk of records ----------------------------------------
        __syncthreads();
        if (tid < 32u) {
            const uint32_t avail = uint32_t(min(uint64_t(kRecs), end - r));
            uint32_t n = 0u;
            if (tid < avail) {
                const uint2* w = reinterpret_cast<const uint2*>(a.ptcl + r + tid);
                const uint2 qa = __ldg(w), qb = __ldg(w + 1), qc = __ldg(w + 2);
                const uint32_t tag = qa.x;
                uint32_t cls = kClsOther, ualpha = 0u, flags = qb.x == 1u ? kHdrEvenOdd : 0u;
                if (tag == TK_PTCL_END) cls = kClsEnd;
                else if (tag == TK_PTCL_BATCH_BEGIN) cls = kClsBatch;
                if (is_fill_like(tag)) {
                    uint32_t s0 = qb.y, s1 = qc.x;
                    if (s1 > a.seg_capacity || s0 > s1) {  // inconsistent scan inputs
                        atomicOr(a.error, ERR_SEGMENT_OVERFLOW);
                        s1 = s0 > a.seg_capacity ? s0 : uint32_t(a.seg_capacity);
                        if (s0 > s1) s1 = s0;
                    }
                    n = s1 - s0;
                    S.seg0[tid] = s0;
                    if (n == 0u) ualpha = coverage_to_alpha(float(int32_t(qa.y)), qb.x);
                    else cls = tag == TK_PTCL_FILL ? kClsFill : kClsCover;
                }
                if (tag == TK_PTCL_FILL) {
                    const uint32_t paint = __ldg(&a.paints[qc.y].paint);
                    if (paint != kGradient) {
                        const bool opaque = premul_u8_is_opaque(paint);
                        if (opaque) flags |= kHdrOpaque;
                        S.col[tid] = channels(paint);
                        if (n == 0u) {
                            // segment-free solid fill: with clip == 255 the source is uniform
                            cls = kClsUniform;
                            S.uniform[tid] = ualpha == 255u && opaque ? rgba8_to_unorm(paint)
                                                                      : scale_premul_u8_to_unorm(paint, ualpha);
                        }
                    } else {
                        flags |= kHdrGradient;
                    }
                }
                S.hdr[tid] = make_uint4(cls | flags | (ualpha << 16) | (tag << 24), 0u,
                                        __float_as_uint(float(int32_t(qa.y))), qc.y);
            }
            const uint32_t incl = warp_inclusive(n, tid);
            S.off[tid + 1u] = incl;
            const uint32_t covers = __ballot_sync(0xffffffffu, n != 0u), slot = __popc(covers & ((1u << tid) - 1u));
            if (n != 0u) S.hdr[tid].x |= (slot & 31u) << kHdrCoverShift;
            // a sum past the budget stays past it: no record holds 2^27 segments of one tile
            const uint32_t nfit = __popc(__ballot_sync(
                0xffffffffu, tid < avail && incl <= kSegs && slot + (n != 0u ? 1u : 0u) <= kCovers));
            if (tid == 0u) {
                S.off[0] = 0u;
                S.n = nfit == 0u ? 1u : nfit;
            }
        }
        __syncthreads();
        uint32_t n = S.n;
        for (uint32_t before = 0u, left = S.off[n]; left != 0u;) {
            uint32_t total = min(left, kSegs);  // more than kSegs: a single record, in slices
#pragma unroll 1
            for (uint32_t sg = tid; sg < total; sg += kThreads) {
                uint32_t lo = 0, hi = n;  // record owning staged segment sg
#pragma unroll 1
                while (hi - lo > 1u) {
                    const uint32_t mid = (lo + hi) >> 1;
                    if (S.off[mid] <= sg) lo = mid;
                    else hi = mid;
                }
                const float4* g = reinterpret_cast<const float4*>(a.segments + S.seg0[lo] + before + (sg - S.off[lo]));
                const float4 q = __ldg(g);
                const float2 e = __ldg(reinterpret_cast<const float2*>(g + 1));  // y_edge, slope
                S.seg[sg] = q;
                S.sgx[sg] = e;
                const uint32_t ga = uint32_t(f2i(fminf(q.x, q.z))) >> 2, gb = uint32_t(f2i(fmaxf(q.x, q.z))) >> 2;
                S.rmask[sg] = crossed_rows(q.y, q.w) | (e.x < 1000000000.0f ? 0x10000u : 0u) | (min(gb - ga, 4u) << 17);
            }
            __syncthreads();
            stage_coverage(S, n, total, before, left, nz, carry);
            if (n > 1u) break;
            if (before == 0u) left = S.off[1];  // the chunk may have been cut to its first record
            before += total;
            left -= total;
        }
        // ---- interpret the chunk -------------------------------------------------
        uint32_t i = 0;
#pragma unroll 1
        while (i < n) {
            const uint4 h = S.hdr[i];
            const uint32_t cls = h.x & kHdrClass;
            uint32_t word;  // the alphas of the record's coverage, a byte per pixel
            if (cls == kClsFill || cls == kClsCover) {
                word = reinterpret_cast<const uint16_t*>(S.alpha + ((h.x >> kHdrCoverShift) & 31u) * TK_TILE_SIZE + row)[column];
            } else {
                if (cls == kClsEnd) {
                    done = true;
                    break;
                }
                if (cls == kClsBatch) {
                    // A new reference batch dispatch: store / reload the target
                    // texel and start from the interpreter's initial state.
#pragma unroll
                    for (int c = 0; c < 4; ++c) px.c[c] = unorm_of_byte(add2(byte_of_unorm(px.c[c], nz), both(-kTwo23)), nz);
                    clip = 0xFFFFu;
                    cdepth = 0u;
                    gdepth = 0u;
                    mode = h.w & TK_TILE_KIND_MASK;
                    i += 1u + (h.w >> TK_TILE_PREFIX_SHIFT);
                    continue;
                }
                // a uniform source over every pixel: colours of color-only tiles
                // (color_only_no_stack_tile_pixel), and without a clip colours and
                // segment-free solid fills
                const bool color_mode = mode == TK_TILE_KIND_COLOR;
                if (color_mode || (cdepth == 0u && (cls == kClsUniform || (h.x >> 24) == TK_PTCL_COLOR))) {
                    const float4 s = color_mode || (cls != kClsUniform && premul_u8_is_opaque(h.w)) ? rgba8_to_unorm(h.w)
                                     : cls == kClsUniform                                           ? S.uniform[i]
                                                          : scale_premul_u8_to_unorm(h.w, 255u);
                    if (s.w > 0.0f) {
                        const float2 k = both(s.w < 1.0f ? 1.0f - s.w : 0.0f);
                        px.c[0] = add2(both(s.x), mul2(px.c[0], k, nz));
                        px.c[1] = add2(both(s.y), mul2(px.c[1], k, nz));
                        px.c[2] = add2(both(s.z), mul2(px.c[2], k, nz));
                        px.c[3] = add2(both(s.w), mul2(px.c[3], k, nz));
                    }
                    ++i;
                    continue;
                }
                word = ((h.x >> 16) & 255u) * 0x0101u;
            }
            const uint32_t tag = h.x >> 24;
            if (tag == TK_PTCL_FILL) {
                if (cdepth != 0u) word = combine_bytes(word, clip);
                if (__any_sync(0xffffffffu, word != 0u)) {
                    const float2 alpha = add2(make_float2(big_byte<0>(word), big_byte<1>(word)), both(-kTwo23));
                    if (h.x & kHdrGradient) paint_gradient(a.paints + h.w, P, cx, cy, alpha, nz, px);
                    else paint_solid(S.col[i], (h.x & kHdrOpaque) != 0u, alpha, nz, px);
                }
            } else if (tag == TK_PTCL_BEGIN_CLIP) {  // push the mask, then narrow it
                if (cdepth < kClipSpill + 4u) {
                    cstack[cdepth] = clip;
                    ++cdepth;
                } else {
                    atomicOr(a.error, ERR_STACK_DEPTH);
                }
                clip = combine_bytes(clip, word);
            } else if (tag == TK_PTCL_END_CLIP) {
                clip = cdepth > 0u ? cstack[cdepth - 1u] : 0xFFFFu;
                if (cdepth > 0u) --cdepth;
            } else {
                if constexpr (GROUPS) {
                    gdepth = rare_record<true>(a.error, tag, h.w, clip, word, groups, gdepth, px);
                } else {
                    Pix copy = px;  // the call takes its address
                    rare_plain(a.error, tag, h.w, clip, copy);
                    px = copy;
                }
            }
            ++i;
        }
        r += i;
    }
    uint32_t w0 = 0u, w1 = 0u;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const float2 b = byte_of_unorm(px.c[c], nz);
        w0 |= (__float_as_uint(b.x) & 255u) << (8 * c);
        w1 |= (__float_as_uint(b.y) & 255u) << (8 * c);
    }
    if (in0) texel[0] = w0;
    if (in1) texel[1] = w1;
}

}  // namespace

void launch_fine_paths(const SceneView& s, const PassView& p, uint32_t* target, uint32_t tiles, cudaStream_t st) {
    const auto kernel = s.groups ? k_fine_paths<true> : k_fine_paths<false>;
    kernel<<<tiles, kThreads, 0, st>>>(
        FineArgs{p.tiles, p.ptcl, s.segments, s.paints, s.brush, s.brush_words, s.segment_capacity, target, s.width,
                 s.height, s.tw, s.error, p.scenes, p.tile_scene, p.tile_list, make_float2(-0.0f, -0.0f)});
}

}  // namespace tk
