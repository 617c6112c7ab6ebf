// The per-draw table that binning and coarse walk (struct DrawInfo): its bits, and how a
// draw is decoded into it.
#pragma once
#include <cuda_runtime.h>

#include "device.cuh"
#include "kernels.h"

namespace tk {
namespace {

using namespace tkd;

// DrawInfo::meta bits (staged candidates: the batch ordinal in the pass above them, from bit kMetaBatchShift)
constexpr uint32_t kMetaPath = 16u, kMetaSolid = 32u, kMetaSdf = 64u, kMetaSdfSolidClass = 128u, kMetaGlyph = 256u;
constexpr uint32_t kMetaBatchShift = 9u;
// DrawInfo::py bits of an SDF draw (px holds its first SDF word)
constexpr uint32_t kSdfPlain = 256u, kSdfIdentity = 512u, kSdfImage = 1024u;

__device__ __forceinline__ uint32_t tile_min_(int32_t px, uint32_t lim) {
    return px > 0 ? min(uint32_t(px) / TK_TILE_SIZE, lim) : 0u;
}
__device__ __forceinline__ uint32_t tile_max_(int32_t px, uint32_t lim) {
    return px > 0 ? min((uint32_t(px) + TK_TILE_SIZE - 1u) / TK_TILE_SIZE, lim) : 0u;
}

// What the per-draw tables are made from (launch_draw_tables).
struct DrawTables {
    const tk_draw_record* draws;
    uint32_t n;
    const tk_path_record* paths;
    uint32_t path_count;
    const uint32_t* brush;
    uint64_t brush_words;
    const uint32_t* sdf;
    uint32_t sdf_shadow_base;
    const tk_glyph_run* glyph_runs;
    uint32_t glyph_run_count;
    const uint32_t* batch_ids;
    const uint4* images;
    uint32_t image_count;
    PaintInfo* paints;
    DrawInfo* infos;
};

// What binning and the candidate walk need of draw `di`.
__device__ __forceinline__ DrawInfo draw_info(const DrawTables& t, const Paint& P, uint32_t di) {
    const tk_draw_record& d = t.draws[di];
    DrawInfo info{};
    info.batch = t.batch_ids[di];
    info.tx = tile_min_(d.pixel_bounds.x0, 65535u) | (tile_max_(d.pixel_bounds.x1, 65535u) << 16);
    info.ty = tile_min_(d.pixel_bounds.y0, 65535u) | (tile_max_(d.pixel_bounds.y1, 65535u) << 16);
    bool valid_path = d.path_id != TK_INVALID_INDEX && d.tag <= TK_DRAW_PATH_GLYPH && d.path_id < t.path_count;
    if (valid_path) {
        const tk_path_record& p = t.paths[d.path_id];
        info.px = p.tile_x0 | (p.tile_x1 << 16);
        info.py = p.tile_y0 | (p.tile_y1 << 16);
        info.data_offset = p.data_offset;
    }
    bool color_candidate = false;
    info.color = di;
    // nontransparent_solid (coarse/paint.hlsli:13-17)
    const bool solid = d.brush_offset != TK_INVALID_INDEX && P.word(d.brush_offset) == TK_BRUSH_SOLID &&
                       P.word(d.brush_offset + TK_BRUSH_COLOR_WORD) != 0u;
    // a glyph run draw gives a PTCL_GLYPH particle or none
    // (coarse/emit_draw.hlsli:15-22)
    const bool glyph = t.glyph_runs && d.glyph_run_id != TK_INVALID_INDEX;
    const bool has_sdf = !glyph && (d.sdf_offset != TK_INVALID_INDEX || d.sdf_shadow_offset != TK_INVALID_INDEX);
    uint32_t bits = 0u;
    if (glyph) {
        valid_path = false;
        if (d.tag == TK_DRAW_BRUSH && d.glyph_run_id < t.glyph_run_count) {
            const tk_glyph_run run = t.glyph_runs[d.glyph_run_id];
            info.px = run.first;
            info.py = run.count;
            bits |= kMetaGlyph;
        }
    } else if (has_sdf) {
        // draw_has_sdf (shared/draw.hlsli:31): only brush draws give a particle
        valid_path = false;
        const bool plain = d.sdf_offset != TK_INVALID_INDEX;
        info.px = plain ? d.sdf_offset : uint32_t(t.sdf_shadow_base) + d.sdf_shadow_offset;
        const uint32_t kind = __ldg(t.sdf + info.px);
        const bool ident = d.transform.a == 1.0f && d.transform.b == 0.0f && d.transform.c == 0.0f &&
                           d.transform.d == 1.0f;
        // full_tile_image's brush test: an image pattern at full opacity
        const bool image = d.brush_offset != TK_INVALID_INDEX &&
                           P.word(d.brush_offset) == TK_BRUSH_PATTERN_RESOURCE &&
                           P.word(d.brush_offset + TK_BRUSH_IMAGE_ALPHA_WORD) == 255u;
        info.py = (kind & 255u) | (plain ? kSdfPlain : 0u) | (ident ? kSdfIdentity : 0u) | (image ? kSdfImage : 0u);
        if (d.tag == TK_DRAW_BRUSH) bits |= kMetaSdf;
        if (solid) {
            color_candidate = true;
            info.color = P.word(d.brush_offset + TK_BRUSH_COLOR_WORD);
        }
        // solid_supported_sdf (coarse/paint.hlsli:21-25)
        if (solid && plain && (kind == TK_SDF_RECT || kind == TK_SDF_CANDLESTICK || kind == TK_SDF_CHECKERBOARD))
            bits |= kMetaSdfSolidClass;
    } else if (d.tag == TK_DRAW_BRUSH && d.solid_rect != 0u && d.transform.b == 0.0f && d.transform.c == 0.0f && solid) {
        color_candidate = true;
        info.color = P.word(d.brush_offset + TK_BRUSH_COLOR_WORD);
    }
    if (d.tag == TK_DRAW_CLIP) info.color = 0u;
    const uint32_t rule = has_sdf ? 0u : (d.fill_rule & 1u);  // SDF particles carry rule 0
    info.meta = (d.tag & 7u) | (rule << 3) | (valid_path ? kMetaPath : 0u) | (color_candidate ? kMetaSolid : 0u) | bits;
    return info;
}

}  // namespace
}  // namespace tk
