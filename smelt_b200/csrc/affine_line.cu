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

// A row-major matrix read in boxes of box_rows rows x 128 bytes, 128-byte swizzle; beyond its edges: zeros.
bool encode(CUtensorMap* map, CUtensorMapDataType type, int width, const void* base, long rows, long cols, int box_rows) {
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)(cols * width)};
    const cuuint32_t box[2] = {(cuuint32_t)(128 / width), (cuuint32_t)box_rows}, step[2] = {1, 1};
    const EncodeTiled fn = encode_tiled();
    return fn && fn(map, type, 2, const_cast<void*>(base), dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

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
        if ((reinterpret_cast<uintptr_t>(w) & 15u) || !encode(&maps->w[s], CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, w, rows, a.cols / 2, paired ? 64 : kLineRows)) return false;
        if (!paired) {
            if (s == 1) line->first1 = line->row_tiles;
            if (s == 2) line->first2 = line->row_tiles;
            line->row_tiles += (rows + kLineRows - 1) / kLineRows;
        }
    }
    if (paired) line->row_tiles = (a.rows + 63) / 64;
    const long tiles = (long)line->row_tiles * line->col_tiles, units = tiles * line->groups;
    if (units >= 1l << 30 || !encode(&maps->x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, a.x, a.batch, a.cols, line->tile_cols)) return false;
    const size_t sums = (size_t)sm * 2 * line->tile_cols * kLineRows * sizeof(float);  // two tiles of every CTA
    if (!a.part_scratch || !a.part_counters || sums > a.part_scratch_bytes) return false;
    const bool split = tiles <= 4096;  // a counter each
    line->quantum = !split ? line->groups : line->groups % kStageGroups == 0 ? kStageGroups : 1;
    // At most about four CTAs to a tile: each more costs the last one as much time as it saves the others
    // (K | V 1024 x 4096 x 2, 64 rows of x: 30.4 us over 148 CTAs, 17.3 us over 64).
    *grid = (int)std::max(1l, split ? std::min({(long)sm, 4 * tiles, units / kStageGroups}) : std::min((long)sm, tiles));
    return true;
}

}  // namespace smelt
