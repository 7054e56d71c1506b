// The launch side of the tensor-core product over affine u4 weights (affine_line.cuh).
#include "affine_line.cuh"

namespace smelt {

namespace {

using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_tiled() {
    static const EncodeTiled fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &found) != cudaSuccess || found != cudaDriverEntryPointSuccess) p = nullptr;
        return reinterpret_cast<EncodeTiled>(p);
    }();
    return fn;
}

// How many CTAs take the line: either a whole number for each tile, or all SMs, whose stretches then begin and end anywhere.  Estimated in us, for
// tiles of up to 32 | 64 | 128 rows of x (fitted to 4,400 timings of 566 shapes, 256 to 12288 rows, 512 to 12288 columns, 33 to 512 rows of x, each
// width both ways; off by 8 % rms):
//   * a launch 1.7 | 1.65 | 3.0 (group sums made in front), a stage 1.0 | 1.55 | 1.6;
//   * a tile that s CTAs share 1.5, in stretches 3.3, and 0.0175 | 0.0125 | 0.016 for each of them and row of x (of 32 at least);
//   * the end of a tile 0.05 for each row of x;
//   * where a row's groups are no multiple of four, scales come two bytes at a time: a launch 0.9 | 0.15 | 0 more, a stage of 128 rows 0.2, and
//     stages beyond those that are fetched ahead 0.45 | 0.1 | 0.3.
// Measured (us, by CTAs of a tile; 148: all SMs): 1024 x 12288, 32 rows: 4 17.3, 8 13.8, 16 15.0, 148 18.5; 4096 x 4096, 32 rows: 2 13.1, 4 10.8,
// 148 12.5; 4096 x 12288, 64 rows: 4 31.1, 148 32.1; gate/up 6144 x 2048, 32 rows: 1 12.1, 148 14.5.
int ctas_for(const Line& p, int sm, int* per_tile, double* cost_us) {
    const long tiles = (long)p.row_tiles * p.col_tiles, units = tiles * p.stages, all = std::min((long)sm, units);
    const bool odd = p.groups % kStageGroups != 0;
    struct { double begin, stage, late, sum; } const width[3] = {{odd ? 2.6 : 1.7, 1.0, odd ? 0.45 : 0.0, 0.0175}, {odd ? 1.8 : 1.65, 1.55, odd ? 0.1 : 0.0, 0.0125}, {3.0, odd ? 1.8 : 1.6, odd ? 0.3 : 0.0, 0.016}};
    const auto& w = width[p.tile_cols <= 32 ? 0 : p.tile_cols <= 64 ? 1 : 2];
    auto cost = [&](long stages, double sharers, double tiles_each, double share) {
        return w.begin + (double)stages * w.stage + (double)std::max(0l, stages - 6) * w.late + (sharers > 1.0 ? share + w.sum * std::max(p.tile_cols, 32) * sharers : 0.0) +
               0.05 * p.tile_cols * tiles_each;
    };
    *per_tile = 0;
    double least = cost((units + all - 1) / all, std::min((double)p.stages, (double)sm / tiles + 1.0), std::max(1.0, (double)tiles / sm), 3.3);
    for (int k = 1; k <= p.stages && tiles * k <= sm; ++k) {
        const double c = cost((p.stages + k - 1) / k, k, 1.0, 1.5);
        if (c < least) { least = c; *per_tile = k; }
    }
    *cost_us = least;
    return (int)(*per_tile ? tiles * *per_tile : all);
}

// How many rows of x a tile has: 32, 64 or 128, whichever ctas_for's estimate says is fastest.  Narrow tiles expand the weights more often, but a small
// matrix has few tiles, SMs idle, and a wide tile's sums take longest to put together.  us, in tiles of 32 | 64 | 128: plain 1024 x 1536, 77 rows
// 8.2 | 10.6 | 15.0, 512 rows 9.9 | 12.8 | 17.4; gate/up 1024 x 2048, 40 rows 9.1 | 11.4, 300 rows 17.1 | 17.8 | 19.9; plain 4096 x 4096, 64 rows
// 14.4 | 15.5, 77 rows 19.0 | 19.3 | 18.6, 128 rows 19.7 | 20.3 | 23.5; gate/up 12288 x 4096, 64 rows 55 | 45, 128 rows 99 | 78 | 57.  Of the 566 shapes the choice
// is 0.3 % slower than the best on average, 15 % at most.
void choose_tile(Line* p, int batch, int max_cols, int sm) {
    Line best = {};
    double least = 0.0;
    for (int cols = 32; cols <= max_cols; cols *= 2) {
        Line q = *p;
        const int wanted = (batch + cols - 1) / cols;
        q.tile_cols = ((batch + wanted - 1) / wanted + 15) & ~15;
        q.col_tiles = (batch + q.tile_cols - 1) / q.tile_cols;
        double cost;
        ctas_for(q, sm, &q.per_tile, &cost);
        if (best.tile_cols == 0 || cost < least) { best = q; least = cost; }
        if (wanted == 1) break;
    }
    *p = best;
}

}  // namespace

bool encode_rows(CUtensorMap* map, CUtensorMapDataType type, int width, const void* base, long rows, long cols, int box_rows) {
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)(cols * width)};
    const cuuint32_t box[2] = {(cuuint32_t)(128 / width), (cuuint32_t)box_rows}, step[2] = {1, 1};
    const EncodeTiled fn = encode_tiled();
    return fn && fn(map, type, 2, const_cast<void*>(base), dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool line_plan(int mode, const AffineArgs& a, int group, int max_cols, int own_cols, LineMaps* maps, Line* line, GroupSums* group_sums, int* grid) {
    if (group != kLineGroup || a.cols % kLineGroup != 0 || a.norm_w) return false;
    if (a.nseg > 1 && affine_stream_passes(mode, a, group) == 0) return false;
    const bool paired = mode == kAffineGateUp || mode == kAffineDual, segs = a.nseg > 1;
    const int sm = a.sm_count > 0 ? a.sm_count : 148;
    if (reinterpret_cast<uintptr_t>(a.x) & 15u) return false;
    *line = {};
    line->groups = a.cols / kLineGroup;
    line->stages = (line->groups + kStageGroups - 1) / kStageGroups;
    line->first1 = line->first2 = INT_MAX;
    for (int s = 0; s < (paired ? 2 : segs ? a.nseg : 1); ++s) {
        const uint8_t* w = segs ? a.seg[s].w : a.w[s];
        const int rows = segs ? a.seg[s].rows : a.rows;
        if ((reinterpret_cast<uintptr_t>(w) & 15u) || !encode_rows(&maps->w[s], CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, w, rows, a.cols / 2, paired ? 64 : kLineRows)) return false;
        if (!paired) {
            if (s == 1) line->first1 = line->row_tiles;
            if (s == 2) line->first2 = line->row_tiles;
            line->row_tiles += (rows + kLineRows - 1) / kLineRows;
        }
    }
    if (paired) line->row_tiles = (a.rows + 63) / 64;
    choose_tile(line, a.batch, max_cols, sm);
    const long tiles = (long)line->row_tiles * line->col_tiles, units = tiles * line->stages;
    if (units >= 1l << 28 || !encode_rows(&maps->x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, a.x, a.batch, a.cols, line->tile_cols)) return false;
    const size_t shared = (size_t)sm * 2 * line->tile_cols * kLineRows;  // two tiles of every CTA
    *group_sums = {nullptr, line->tile_cols > own_cols ? (size_t)a.batch * line->stages * 2 * kStageGroups : 0};
    if (!a.part_scratch || !a.part_counters || (shared + group_sums->floats) * sizeof(float) > a.part_scratch_bytes) return false;
    if (group_sums->floats) {
        group_sums->at = a.part_scratch + shared;
        if (!encode_rows(&maps->sums, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, group_sums->at, a.batch, (long)line->stages * 2 * kStageGroups, line->tile_cols)) return false;
    }
    const bool split = tiles <= 4096;  // a counter each
    line->quantum = split ? 1 : line->stages;
    double cost;
    *grid = split ? ctas_for(*line, sm, &line->per_tile, &cost) : (int)std::min((long)sm, tiles);
    if (!split) line->per_tile = 0;
    line->share = (int)(units / line->quantum / *grid);
    line->extra = (int)(units / line->quantum % *grid);
    return true;
}

}  // namespace smelt
