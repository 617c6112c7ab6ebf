// Differentiable rendering: a float forward of fine raster, Gaussian blur and
// the group composite, and their hand-written adjoint.
//
// Model (the reference's fine + blur + composite path, fine/interpreter.hlsli,
// shared/coverage.hlsli:7-51, filter/blur.hlsli, without the RGBA8
// quantization between stages so that it is differentiable):
//   coverage  A = signed exact area of the path in the pixel (fill_alpha_at),
//             c = min(|A|, 1) (nonzero)
//   layer     L_i = s_i + L_{i-1} (1 - a_i),  s_i = colp_i c_i,  a_i = alpha_i c_i
//   blur      T1 = Gx L, B = Gy T1, taps w_k = e_k / sum e, e_k = exp(-k^2 / 2 sigma^2),
//             |k| <= r, zero outside the canvas
//   composite I = B + bg (1 - B.a)
//   loss      mean over pixels and channels of (I - target)^2
// Backward: dB from dI; the blur adjoint is the same symmetric blur; the sigma
// gradient uses the tap derivatives w'_k. Fine recomputes coverage per tile
// (forward replay storing A_i and P_i = g . L_{i-1} per pixel), then walks the
// records in reverse with the transmittance T_i = prod_{j>i} (1 - a_j):
//   dL/dc_i = T_i (g . colp_i - alpha_i P_i)
// and turns dL/dA per pixel into line-endpoint gradients by the boundary
// integral of the exact area: for a line P0 -> P1 (d = P1 - P0) and a pixel P,
//   dA_P/dP0 = (int_{u in U_P} (1 - u) du) (d.y, -d.x),
//   dA_P/dP1 = (int_{u in U_P} u du) (d.y, -d.x),
// U_P = the parameters u of the line's points inside P.
#include <cuda_runtime.h>

#include "device.cuh"
#include "kernels.h"

namespace tk {
namespace {

using namespace tkd;

constexpr int kDiffThreads = 256;  // a thread per pixel of a 16x16 tile
constexpr uint32_t kDiffRows = 32;  // segments whose row parts are staged at a time

// A chunk of a tile's records. Both kernels walk the records in chunks of
// kDiffChunk: one round of loads and two barriers per chunk, where a record at a
// time paid a chain of dependent loads and four barriers each (most records of a
// tile have no segment at all, the others a few).
struct DiffChunk {
    float4 colp[kDiffChunk];  // zero: no FILL record
    float base[kDiffChunk];   // the backdrop
    uint32_t color[kDiffChunk];  // TK_INVALID_INDEX: no FILL record
    uint32_t end[kDiffChunk];     // inclusive prefix of the segment counts
    uint32_t offset[kDiffChunk];  // segment index of the chunk's j-th segment: offset + j
    float4 rows[kDiffRows][TK_TILE_SIZE];  // edge, dy, xmin, xmax of a segment in a pixel row
};

// Records [r0, min(r0 + kDiffChunk, r1)) into S (all threads); returns how many.
// Records after END, and those that are no FILL, count as fills of no area.
__device__ uint32_t stage_records(DiffChunk& S, const tk_ptcl_record* __restrict__ ptcl, uint64_t r0, uint64_t r1,
                                  const float4* __restrict__ colp, uint32_t* error) {
    const uint32_t m = uint32_t(min(uint64_t(kDiffChunk), r1 - r0));
    __syncthreads();  // the last chunk's readers
    if (threadIdx.x < 32) {
        const uint32_t lane = threadIdx.x;
        tk_ptcl_record q{};
        q.tag = TK_PTCL_END;
        if (lane < m) q = ptcl[r0 + lane];
        const uint32_t ends = __ballot_sync(0xffffffffu, q.tag == TK_PTCL_END);
        const bool live = !(ends & ((2u << lane) - 1u));
        const bool fill = live && q.tag == TK_PTCL_FILL;
        // occlusion skips come only from opaque solid-rect records, which
        // differentiable scenes do not contain
        if (live && !fill && (q.tag != TK_PTCL_BATCH_BEGIN || (q.color >> TK_TILE_PREFIX_SHIFT)))
            atomicOr(error, ERR_UNSUPPORTED);
        const uint32_t n = fill ? q.segment_end - q.segment_start : 0u;
        uint32_t end = n;
        for (int o = 1; o < int(kDiffChunk); o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, end, o);
            if (lane >= uint32_t(o)) end += v;
        }
        if (lane < kDiffChunk) {
            S.colp[lane] = fill ? colp[q.color] : make_float4(0.f, 0.f, 0.f, 0.f);
            S.base[lane] = fill ? float(q.backdrop) : 0.0f;
            S.color[lane] = fill ? q.color : TK_INVALID_INDEX;
            S.end[lane] = end;
            S.offset[lane] = q.segment_start - (end - n);
        }
    }
    __syncthreads();
    return m;
}

// The record of the chunk's segment j: the first whose end is beyond it.
__device__ __forceinline__ uint32_t record_of(const DiffChunk& S, uint32_t j) {
    uint32_t r = 0;
#pragma unroll
    for (uint32_t o = kDiffChunk / 2; o; o >>= 1)
        if (S.end[r + o - 1] <= j) r += o;
    return r;
}

// on_record(r, A) for the m staged records in order, A the signed area of the
// record in this thread's pixel (fill_alpha_at over its segments, in order). The
// row parts of a segment are the same for a row's 16 pixels: they are computed
// once, a thread per (segment, row).
template <class F>
__device__ __forceinline__ void walk_chunk(DiffChunk& S, uint32_t m, const SegmentRec* __restrict__ segments,
                                           F&& on_record) {
    const uint32_t lx = threadIdx.x & 15u, ly = threadIdx.x >> 4, total = S.end[m - 1];
    const float x = float(lx), x1 = float(lx + 1u);
    uint32_t j = 0, first = 0, staged = 0;
    for (uint32_t r = 0; r < m; ++r) {
        const uint32_t end = S.end[r];
        float base = S.base[r], running = 0.0f, partial = 0.0f;
        while (j < end) {
            if (j == staged) {
                if (staged) __syncthreads();
                first = staged;
                staged = min(first + kDiffRows, total);
                for (uint32_t i = threadIdx.x; i < (staged - first) * TK_TILE_SIZE; i += kDiffThreads) {
                    const uint32_t k = i / TK_TILE_SIZE, row = i % TK_TILE_SIZE;
                    const SegmentRec* seg = segments + uint32_t(S.offset[record_of(S, first + k)] + first + k);
                    const float4 g = __ldg(reinterpret_cast<const float4*>(seg));
                    const RowParts q = segment_row_parts(g.x, g.y, g.z, g.w, __ldg(&seg->y_edge), row);
                    // (a segment that does not reach the row lies right of every pixel)
                    S.rows[k][row] = q.dy != 0.0f ? make_float4(q.edge, q.dy, q.xmin, q.xmax)
                                                  : make_float4(q.edge, 0.0f, 16.0f, 16.0f);
                }
                __syncthreads();
            }
            const uint32_t stop = min(end, staged);
            for (; j < stop; ++j) {
                const float4 q = S.rows[j - first][ly];
                base += q.x;
                if (x >= q.w) running += q.y;
                else if (x1 > q.z) partial += segment_area_at(q.z, q.w, lx) * q.y;
            }
        }
        on_record(r, base + running + partial);
    }
}

__device__ __forceinline__ float dot4(float4 a, float4 b) {
    return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, a.x * b.x)));
}

// Forward: the float layer image of one target pass. 1024x1024, 256 paths of 12
// cubics (87 fill records and 98 segments a tile): 0.41 ms with a record at a time,
// 0.26 in chunks; bound by instruction issue (3.2 a cycle), about 35 per record
// and pixel.
__global__ void __launch_bounds__(kDiffThreads)
    k_diff_fine_fwd(const tk_tile_record* __restrict__ tiles, const tk_ptcl_record* __restrict__ ptcl,
                    const SegmentRec* __restrict__ segments, const float4* __restrict__ colp, float4* layer,
                    uint32_t width, uint32_t height, uint32_t tw, uint32_t* error) {
    __shared__ DiffChunk S;
    const uint32_t tile = blockIdx.x;
    const tk_tile_record rec = tiles[tile];
    const uint32_t gx = (tile % tw) * TK_TILE_SIZE + (threadIdx.x & 15u);
    const uint32_t gy = (tile / tw) * TK_TILE_SIZE + (threadIdx.x >> 4);
    float4 L = make_float4(0.f, 0.f, 0.f, 0.f);
    for (uint64_t r0 = rec.ptcl_start; r0 < rec.ptcl_end; r0 += kDiffChunk) {
        const uint32_t m = stage_records(S, ptcl, r0, rec.ptcl_end, colp, error);
        walk_chunk(S, m, segments, [&](uint32_t r, float A) {
            const float c = fminf(fabsf(A), 1.0f);
            const float4 p = S.colp[r];
            const float k = fmaf(-p.w, c, 1.0f);
            L = make_float4(fmaf(L.x, k, p.x * c), fmaf(L.y, k, p.y * c), fmaf(L.z, k, p.z * c), fmaf(L.w, k, p.w * c));
        });
    }
    if (gx < width && gy < height) layer[uint64_t(gy) * width + gx] = L;
}

// out[p] = sum_k w[k + r] in[p + k * step]; zero outside the canvas.
__device__ __forceinline__ float4 blur_tap(const float4* __restrict__ img, const float* __restrict__ w, int32_t r,
                                           uint32_t width, uint32_t height, int32_t x, int32_t y, int32_t axis) {
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int32_t k = -r; k <= r; ++k) {
        const int32_t sx = axis == 0 ? x + k : x, sy = axis == 0 ? y : y + k;
        if (sx < 0 || sy < 0 || sx >= int32_t(width) || sy >= int32_t(height)) continue;
        const float4 v = img[uint64_t(sy) * width + sx];
        const float wk = w[k + r];
        acc.x += wk * v.x;
        acc.y += wk * v.y;
        acc.z += wk * v.z;
        acc.w += wk * v.w;
    }
    return acc;
}

__global__ void k_diff_blur(const float4* __restrict__ in, float4* out, const float* __restrict__ w, int32_t r,
                            uint32_t width, uint32_t height, int32_t axis) {
    const int32_t x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    if (x >= int32_t(width)) return;
    out[uint64_t(y) * width + x] = blur_tap(in, w, r, width, height, x, y, axis);
}

// I = B + bg (1 - B.a); gI = 2 (I - target) / (4 W H); loss partial sums.
// Only pixels [lo, hi) enter the loss (a row range of a split objective);
// the mean still divides by every pixel, so the row ranges' losses and
// gradients sum to the whole frame's.
__global__ void k_diff_composite(const float4* __restrict__ B, const float4* __restrict__ target, float4 bg,
                                 uint64_t n, uint64_t lo, uint64_t hi, float4* image, float4* gI, double* loss) {
    double acc = 0.0;
    const double inv = 1.0 / (4.0 * double(n));
    for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x) {
        const float4 b = B[i];
        const float k = 1.0f - b.w;
        const float4 I = make_float4(b.x + bg.x * k, b.y + bg.y * k, b.z + bg.z * k, b.w + bg.w * k);
        const float4 t = target[i];
        const float4 d = make_float4(I.x - t.x, I.y - t.y, I.z - t.z, I.w - t.w);
        if (image) image[i] = I;
        if (i < lo || i >= hi) {
            gI[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            continue;
        }
        const float s = float(2.0 * inv);
        gI[i] = make_float4(s * d.x, s * d.y, s * d.z, s * d.w);
        acc += double(d.x) * d.x + double(d.y) * d.y + double(d.z) * d.z + double(d.w) * d.w;
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31u) == 0) atomicAdd(loss, acc * inv);
}

__device__ __forceinline__ float4 composite_adjoint(float4 g, float4 bg) {
    // dI/dB: identity per channel, and -bg on the alpha channel's column.
    return make_float4(g.x, g.y, g.z, g.w - dot4(g, bg));
}

// Blur adjoint along `axis` plus the sigma term <dout, G' in_fwd>:
//   din[p] = sum_k w_k dout[p + k]   (symmetric taps, zero outside)
//   sig   += dout[p] . sum_k w'_k fwd_in[p + k]
// With `from_gI`, dout is the composite adjoint of gI.
__global__ void k_diff_blur_bwd(const float4* __restrict__ dout_src, const float4* __restrict__ fwd_in, float4* din,
                                const float* __restrict__ w, const float* __restrict__ wd, int32_t r, uint32_t width,
                                uint32_t height, int32_t axis, int32_t from_gI, float4 bg, double* sig) {
    const int32_t x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    double part = 0.0;
    if (x < int32_t(width)) {
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f), dacc = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int32_t k = -r; k <= r; ++k) {
            const int32_t sx = axis == 0 ? x + k : x, sy = axis == 0 ? y : y + k;
            if (sx < 0 || sy < 0 || sx >= int32_t(width) || sy >= int32_t(height)) continue;
            const uint64_t q = uint64_t(sy) * width + sx;
            float4 g = dout_src[q];
            if (from_gI) g = composite_adjoint(g, bg);
            const float wk = w[k + r], dk = wd[k + r];
            acc.x += wk * g.x;
            acc.y += wk * g.y;
            acc.z += wk * g.z;
            acc.w += wk * g.w;
            const float4 v = fwd_in[q];
            dacc.x += dk * v.x;
            dacc.y += dk * v.y;
            dacc.z += dk * v.z;
            dacc.w += dk * v.w;
        }
        const uint64_t p = uint64_t(y) * width + x;
        din[p] = acc;
        float4 g = dout_src[p];
        if (from_gI) g = composite_adjoint(g, bg);
        part = double(dot4(g, dacc));
    }
    for (int o = 16; o > 0; o >>= 1) part += __shfl_down_sync(0xffffffffu, part, o);
    if ((threadIdx.x & 31u) == 0 && part != 0.0) atomicAdd(sig, part);
}

// Without blur the layer adjoint is the composite adjoint of gI.
__global__ void k_diff_composite_bwd(const float4* __restrict__ gI, float4 bg, uint64_t n, float4* dL) {
    for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x)
        dL[i] = composite_adjoint(gI[i], bg);
}

// Boundary-integral weights of a tile segment q0 -> q1 (tile-local), part of
// line P0 -> P1 (tile-local), against the per-pixel adjoint gA: returns
// (sum gA int (1-u) du, sum gA int u du) over the cells the segment crosses.
__device__ float2 segment_boundary_sums(const float* __restrict__ gA, float4 q, float2 P0, float2 d) {
    const float dd = d.x * d.x + d.y * d.y;
    if (!(dd > 0.0f)) return make_float2(0.f, 0.f);
    const float u0 = ((q.x - P0.x) * d.x + (q.y - P0.y) * d.y) / dd;
    const float u1 = ((q.z - P0.x) * d.x + (q.w - P0.y) * d.y) / dd;
    const float ex = q.z - q.x, ey = q.w - q.y;
    float vx = 2.0f, vy = 2.0f, stx = 2.0f, sty = 2.0f;
    if (ex > 0.0f) { vx = (floorf(q.x) + 1.0f - q.x) / ex; stx = 1.0f / ex; }
    else if (ex < 0.0f) { vx = (ceilf(q.x) - 1.0f - q.x) / ex; stx = -1.0f / ex; }
    if (ey > 0.0f) { vy = (floorf(q.y) + 1.0f - q.y) / ey; sty = 1.0f / ey; }
    else if (ey < 0.0f) { vy = (ceilf(q.y) - 1.0f - q.y) / ey; sty = -1.0f / ey; }
    float v = 0.0f, s0 = 0.0f, s1 = 0.0f;
    for (int it = 0; it < 2 * int(TK_TILE_SIZE) + 4 && v < 1.0f; ++it) {
        const float vn = fminf(fminf(vx, vy), 1.0f);
        if (vn > v) {
            const float vm = 0.5f * (v + vn);
            const int32_t cx = min(max(int32_t(floorf(q.x + vm * ex)), 0), int32_t(TK_TILE_SIZE) - 1);
            const int32_t cy = min(max(int32_t(floorf(q.y + vm * ey)), 0), int32_t(TK_TILE_SIZE) - 1);
            const float ua = u0 + v * (u1 - u0), ub = u0 + vn * (u1 - u0);
            const float ul = fminf(ua, ub), uh = fmaxf(ua, ub);
            const float sq = 0.5f * (uh * uh - ul * ul);
            const float g = gA[cy * TK_TILE_SIZE + cx];
            s0 += g * ((uh - ul) - sq);
            s1 += g * sq;
        }
        if (vx <= vn) vx += stx;
        if (vy <= vn) vy += sty;
        v = vn;
    }
    return make_float2(s0, s1);
}

constexpr uint32_t kDiffSum = kDiffThreads / 32;  // records whose colour sums are taken at a time, a warp each

struct DiffBack {
    DiffChunk c;
    float A[kDiffChunk][kDiffThreads];  // a record's area per pixel, then dL/dA
    float P[kDiffChunk][kDiffThreads];
    float4 g[kDiffThreads];
};
static_assert(sizeof(DiffChunk::rows) >= kDiffSum * kDiffThreads * sizeof(float), "T c takes the rows' place");

// Sums v[0..4] over the warp: lane 0, 4, 8, 16 and 20 return the sum of v[0], v[1],
// v[2], v[3] and v[4]. Halves exchange the values that the other half keeps: 8
// shuffles, where five trees take 25.
__device__ __forceinline__ float warp_sum5(const float (&v)[5], uint32_t lane) {
    const bool h16 = lane & 16u, h8 = lane & 8u, h4 = lane & 4u;
    const uint32_t all = 0xffffffffu;
    const float a0 = (h16 ? v[3] : v[0]) + __shfl_xor_sync(all, h16 ? v[0] : v[3], 16);
    const float a1 = (h16 ? v[4] : v[1]) + __shfl_xor_sync(all, h16 ? v[1] : v[4], 16);
    const float a2 = (h16 ? 0.0f : v[2]) + __shfl_xor_sync(all, h16 ? v[2] : 0.0f, 16);
    const float b0 = (h8 ? a2 : a0) + __shfl_xor_sync(all, h8 ? a0 : a2, 8);
    const float b1 = (h8 ? 0.0f : a1) + __shfl_xor_sync(all, h8 ? a1 : 0.0f, 8);
    float s = (h4 ? b1 : b0) + __shfl_xor_sync(all, h4 ? b0 : b1, 4);
    s += __shfl_xor_sync(all, s, 2);
    return s + __shfl_xor_sync(all, s, 1);
}

// Backward of fine: per tile, a forward replay that keeps P = g . L per pixel at
// each chunk's start (`scratch`, 256 floats per chunk), then the chunks in reverse,
// A and P of a chunk's records computed again in shared memory: 1 KB of scratch
// per 16 records, where A and P of each record took 32. The segments of a whole
// chunk are dealt out to the threads for the line gradients, and the colour sums of
// 8 records to a warp each. The scene above: 1.65 ms with a record at a time, 0.87
// now (0.93 with the colour sums by shuffles in every record), two thirds of it the
// two replays.
__global__ void __launch_bounds__(kDiffThreads)
    k_diff_fine_bwd(const tk_tile_record* __restrict__ tiles, const tk_ptcl_record* __restrict__ ptcl,
                    const SegmentRec* __restrict__ segments, const uint32_t* __restrict__ seg_line,
                    const tk_line* __restrict__ lines, const float4* __restrict__ colp,
                    const float4* __restrict__ dlayer, float* scratch, float2* line_acc, float* color_acc,
                    uint32_t width, uint32_t height, uint32_t tw, uint32_t* error) {
    __shared__ DiffBack S;
    const uint32_t tile = blockIdx.x;
    const tk_tile_record rec = tiles[tile];
    if (rec.ptcl_start >= rec.ptcl_end) return;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t ox = (tile % tw) * TK_TILE_SIZE, oy = (tile / tw) * TK_TILE_SIZE;
    const uint32_t gx = ox + (tid & 15u), gy = oy + (tid >> 4);
    const bool inside = gx < width && gy < height;
    const float4 g = inside ? dlayer[uint64_t(gy) * width + gx] : make_float4(0.f, 0.f, 0.f, 0.f);
    S.g[tid] = g;
    float(*const tc)[kDiffThreads] = reinterpret_cast<float(*)[kDiffThreads]>(S.c.rows);
    const uint32_t n_chunks = uint32_t((rec.ptcl_end - rec.ptcl_start + kDiffChunk - 1) / kDiffChunk);
    float* const kept = scratch + diff_scratch_at(rec.ptcl_start, tile) + tid;
    uint32_t m = 0;
    auto replay = [&](uint32_t chunk, float P) {
        const uint64_t r0 = rec.ptcl_start + uint64_t(chunk) * kDiffChunk;
        m = stage_records(S.c, ptcl, r0, rec.ptcl_end, colp, error);
        walk_chunk(S.c, m, segments, [&](uint32_t r, float A) {
            const float c = fminf(fabsf(A), 1.0f);
            const float4 p = S.c.colp[r];
            S.A[r][tid] = A;
            S.P[r][tid] = P;
            P = fmaf(dot4(g, p), c, P * fmaf(-p.w, c, 1.0f));
        });
        return P;
    };
    float P = 0.0f;
    for (uint32_t k = 0; k < n_chunks; ++k) {
        kept[uint64_t(k) * kDiffThreads] = P;
        P = replay(k, P);
    }
    float T = 1.0f;
    for (uint32_t k = n_chunks; k-- > 0;) {
        if (k + 1 < n_chunks) replay(k, kept[uint64_t(k) * kDiffThreads]);
        for (uint32_t r0 = (m - 1) / kDiffSum * kDiffSum, r1 = m;; r1 = r0, r0 -= kDiffSum) {
            __syncthreads();  // the readers of rows, or of tc
            for (uint32_t r = r1; r-- > r0;) {
                const float A = S.A[r][tid];
                const float c = inside ? fminf(fabsf(A), 1.0f) : 0.0f;
                const float4 p = S.c.colp[r];
                const float dc = T * fmaf(-p.w, S.P[r][tid], dot4(g, p));
                tc[r - r0][tid] = T * c;
                S.A[r][tid] = (inside && c < 1.0f && A != 0.0f) ? (A > 0.0f ? dc : -dc) : 0.0f;
                T *= fmaf(-p.w, c, 1.0f);
            }
            __syncthreads();
            // colour partials: T g c (4 channels) and -T P c (alpha through 1 - a)
            if (r0 + warp < r1) {
                const uint32_t r = r0 + warp;
                float v[5] = {};
#pragma unroll
                for (uint32_t i = lane; i < kDiffThreads; i += 32) {
                    const float t = tc[warp][i];
                    const float4 gi = S.g[i];
                    v[0] = fmaf(t, gi.x, v[0]);
                    v[1] = fmaf(t, gi.y, v[1]);
                    v[2] = fmaf(t, gi.z, v[2]);
                    v[3] = fmaf(t, gi.w, v[3]);
                    v[4] = fmaf(-t, S.P[r][i], v[4]);
                }
                const float s = warp_sum5(v, lane);
                const uint32_t color = S.c.color[r];
                // (a record that is no FILL sums zeros, or NaN where g is not finite)
                if (s != 0.0f && color != TK_INVALID_INDEX && !(lane & 3u) && lane != 12u && lane < 24u)
                    atomicAdd(color_acc + uint64_t(color) * 5u + (lane >> 2) - (lane > 12u ? 1u : 0u), s);
            }
            if (!r0) break;
        }
        const uint32_t total = S.c.end[m - 1];
        for (uint32_t j = tid; j < total; j += kDiffThreads) {
            const uint32_t r = record_of(S.c, j), at = S.c.offset[r] + j;
            const float4 seg = __ldg(reinterpret_cast<const float4*>(segments + at));
            const uint32_t li = seg_line[at];
            const tk_line ln = lines[li];
            const float2 P0 = make_float2(ln.p0[0] - float(ox), ln.p0[1] - float(oy));
            const float2 d = make_float2(ln.p1[0] - ln.p0[0], ln.p1[1] - ln.p0[1]);
            const float2 s = segment_boundary_sums(S.A[r], seg, P0, d);
            if (s.x != 0.0f) atomicAdd(&line_acc[li].x, s.x);
            if (s.y != 0.0f) atomicAdd(&line_acc[li].y, s.y);
        }
    }
}

// Line-endpoint gradients to control points: each endpoint is
// sum_i w_i C[base + i] (frozen flattening weights).
__global__ void k_diff_lines_to_points(const tk_line* __restrict__ lines, const float2* __restrict__ line_acc,
                                       const uint32_t* __restrict__ ep_base, const float* __restrict__ ep_w,
                                       uint64_t n, float* dpoints) {
    for (uint64_t l = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; l < n; l += uint64_t(gridDim.x) * blockDim.x) {
        const tk_line ln = lines[l];
        const float dx = ln.p1[0] - ln.p0[0], dy = ln.p1[1] - ln.p0[1];
        const float2 s = line_acc[l];
        const float g[2][2] = {{s.x * dy, -s.x * dx}, {s.y * dy, -s.y * dx}};
        for (int e = 0; e < 2; ++e) {
            const uint32_t b = ep_base[2 * l + e];
            for (int i = 0; i < 4; ++i) {
                const float wi = ep_w[8 * l + 4 * e + i];
                if (wi == 0.0f) continue;
                atomicAdd(dpoints + 2u * (b + i), wi * g[e][0]);
                atomicAdd(dpoints + 2u * (b + i) + 1u, wi * g[e][1]);
            }
        }
    }
}

}  // namespace

void launch_diff_fine_fwd(const SceneView& s, const PassView& p, const float4* colp, float4* layer, cudaStream_t st) {
    const uint32_t T = s.tw * s.th;
    if (T == 0) return;
    k_diff_fine_fwd<<<T, kDiffThreads, 0, st>>>(p.tiles, p.ptcl, s.segments, colp, layer, s.width, s.height, s.tw,
                                               s.error);
}

void launch_diff_blur(const float4* in, float4* out, const float* w, int32_t r, uint32_t width, uint32_t height,
                      int32_t axis, cudaStream_t st) {
    dim3 grid((width + 255) / 256, height);
    k_diff_blur<<<grid, 256, 0, st>>>(in, out, w, r, width, height, axis);
}

void launch_diff_composite(const float4* B, const float4* target, float4 bg, uint64_t n, uint64_t lo, uint64_t hi,
                           float4* image, float4* gI, double* loss, cudaStream_t st) {
    k_diff_composite<<<148 * 8, 256, 0, st>>>(B, target, bg, n, lo, hi, image, gI, loss);
}

void launch_diff_blur_bwd(const float4* dout_src, const float4* fwd_in, float4* din, const float* w, const float* wd,
                          int32_t r, uint32_t width, uint32_t height, int32_t axis, bool from_gI, float4 bg,
                          double* sig, cudaStream_t st) {
    dim3 grid((width + 255) / 256, height);
    k_diff_blur_bwd<<<grid, 256, 0, st>>>(dout_src, fwd_in, din, w, wd, r, width, height, axis, from_gI ? 1 : 0, bg,
                                          sig);
}

void launch_diff_composite_bwd(const float4* gI, float4 bg, uint64_t n, float4* dL, cudaStream_t st) {
    k_diff_composite_bwd<<<148 * 8, 256, 0, st>>>(gI, bg, n, dL);
}

void launch_diff_fine_bwd(const SceneView& s, const PassView& p, const uint32_t* seg_line, const float4* colp,
                          const float4* dlayer, float* scratch, float2* line_acc, float* color_acc, cudaStream_t st) {
    const uint32_t T = s.tw * s.th;
    if (T == 0) return;
    k_diff_fine_bwd<<<T, kDiffThreads, 0, st>>>(p.tiles, p.ptcl, s.segments, seg_line, s.lines, colp, dlayer, scratch,
                                               line_acc, color_acc, s.width, s.height, s.tw, s.error);
}

void launch_diff_lines_to_points(const tk_line* lines, const float2* line_acc, const uint32_t* ep_base,
                                 const float* ep_w, uint64_t n, float* dpoints, cudaStream_t st) {
    if (n == 0) return;
    k_diff_lines_to_points<<<148 * 4, 256, 0, st>>>(lines, line_acc, ep_base, ep_w, n, dpoints);
}

}  // namespace tk
