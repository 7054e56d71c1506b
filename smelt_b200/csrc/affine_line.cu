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

// How many CTAs take the line: either a whole number for each tile, or all SMs, whose stretches then begin and end anywhere.
// Estimated in us.  A group takes a CTA 0.53 us with 32 rows of x, 0.57 with 128 and 0.96 with 256; the CTA that finishes a tile
// needs 0.011 us per column and CTA whose sums it adds, and with stretches anywhere it may finish two, of one CTA more each
// (weighed with 1.5: at 512 rows 4096 x 12288 takes 110.8 by whole numbers and 104.6 by stretches, 6144 x 2048 49.2 and 46.4).
// Measured (us, by CTAs of a tile; 148: all SMs): 1024 x 12288, 32 rows: 4 30.7, 8 19.4, 16 15.6, 148 19.2; 256 rows: 4 63.3,
// 8 51.6, 16 60.2, 148 72.3; 4096 x 4096, 32 rows: 2 22.6, 4 15.5, 148 18.0; 256 rows: 4 36.2, 148 47.7; K | V 1024 x 4096 x 2,
// 32 rows: 4 13.8, 8 11.2, 148 14.7; 512 rows: 4 35.8, 148 47.5; 4096 x 12288, 32 rows: 4 33.7, 148 34.4; gate/up 6144 x 2048,
// 32 rows: 1 22.6, 148 22.3.
long ctas_for(const Line& p, int sm) {
    const long tiles = (long)p.row_tiles * p.col_tiles, quanta = p.groups / p.quantum;
    const double group = p.tile_cols <= 128 ? 0.52 + 0.0004 * p.tile_cols : 0.96, sum = 0.011 * p.tile_cols;
    long best = sm;
    double least = (double)tiles * p.groups / sm * group + 1.5 * sum * ((double)sm / tiles + 1.0);
    for (long k = 1; k <= quanta && tiles * k <= sm; ++k) {
        const double cost = (double)((quanta + k - 1) / k * p.quantum) * group + (k > 1 ? sum * k : 0.0);
        if (cost < least) { least = cost; best = tiles * k; }
    }
    return std::min(best, tiles * quanta);
}

}  // namespace

bool encode_rows(CUtensorMap* map, CUtensorMapDataType type, int width, const void* base, long rows, long cols, int box_rows) {
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)(cols * width)};
    const cuuint32_t box[2] = {(cuuint32_t)(128 / width), (cuuint32_t)box_rows}, step[2] = {1, 1};
    const EncodeTiled fn = encode_tiled();
    return fn && fn(map, type, 2, const_cast<void*>(base), dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool line_plan(int mode, const AffineArgs& a, int group, int max_cols, LineMaps* maps, Line* line, int* grid) {
    if (group != kLineGroup || a.cols % kLineGroup != 0 || a.norm_w) return false;
    if (a.nseg > 1 && affine_stream_passes(mode, a, group) == 0) return false;
    const bool paired = mode == kAffineGateUp || mode == kAffineDual, segs = a.nseg > 1;
    const int sm = a.sm_count > 0 ? a.sm_count : 148;
    if (reinterpret_cast<uintptr_t>(a.x) & 15u) return false;
    *line = {};
    line->groups = a.cols / kLineGroup;
    const int wanted = (a.batch + max_cols - 1) / max_cols;
    line->tile_cols = (a.batch + wanted - 1) / wanted;
    line->tile_cols = line->tile_cols <= 128 ? (line->tile_cols + 15) & ~15 : (line->tile_cols + 31) & ~31;  // above 128 two MMAs share them
    line->col_tiles = (a.batch + line->tile_cols - 1) / line->tile_cols;
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
    const long tiles = (long)line->row_tiles * line->col_tiles, units = tiles * line->groups;
    if (units >= 1l << 30 || !encode_rows(&maps->x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, a.x, a.batch, a.cols, line->tile_cols)) return false;
    const size_t sums = (size_t)sm * 2 * line->tile_cols * kLineRows * sizeof(float);  // two tiles of every CTA
    if (!a.part_scratch || !a.part_counters || sums > a.part_scratch_bytes) return false;
    const bool split = tiles <= 4096;  // a counter each
    line->quantum = !split ? line->groups : line->groups % kStageGroups == 0 ? kStageGroups : 1;
    *grid = (int)(split ? ctas_for(*line, sm) : std::min((long)sm, tiles));
    return true;
}

}  // namespace smelt
