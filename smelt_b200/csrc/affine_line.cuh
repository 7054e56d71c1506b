// What a tensor-core product over affine u4 weights is cut from (affine_wide.cu): its line of work, bounded waits, the
// feed of scales and biases.
#pragma once
#include <cuda.h>

#include <algorithm>
#include <climits>

#include "affine_matvec.h"
#include "tcgen05.cuh"

namespace smelt {

constexpr int kLineRows = 128, kLineGroup = 64, kStageGroups = 4;     // weight rows of a tile, columns of a group, groups of a stage
constexpr int kRawBytes = kLineRows * kStageGroups * kLineGroup / 2;  // packed weights of a stage: 16 KB

struct LineMaps {
    CUtensorMap w[3], x, sums;  // sums: what group_sums_kernel wrote, where the tile is wide
};

// The work is the line of all (tile, stage) units, tile after tile; a tile is 128 weight rows (64 of each matrix
// in the paired forms) and up to tile_cols rows of x, a stage four groups (a row's last one may have fewer).  Every CTA takes
// an equal stretch of the line, whatever the matrix' shape, so no SM waits for a last wave (192 tiles of gate/up 12288 x 4096
// over 148 SMs would take two waves, the second one third full).  A tile that lies in the stretches of several CTAs is put
// together from fp32 sums in scratch, in column order, by the last of them to finish: results do not depend on timing.
struct Line {
    int row_tiles, col_tiles, tile_cols, groups, stages;
    int first1, first2;  // first row tile of the second and third tensor
    int per_tile;        // CTAs of every tile; 0: equal stretches of the whole line
    int quantum;         // stretches: stages that are never split, one, or a tile's where there is no counter for it
    int share, extra;    // CTAs before `extra` take share + 1 quanta, the others share
};

__device__ __forceinline__ int line_at(const Line& p, int c) {  // where CTA c begins, in stages
    return p.per_tile ? c / p.per_tile * p.stages + c % p.per_tile * p.stages / p.per_tile : (c * p.share + min(c, p.extra)) * p.quantum;
}

// One tile's part of a stretch.
struct Part {
    int tile, s0, s1, row_tile, col_tile, col0, live;  // stages [s0, s1); first row of x and how many
};
__device__ __forceinline__ void part_rows(const Line& p, Part& t, int batch) {
    t.col0 = t.col_tile * p.tile_cols;
    t.live = min(p.tile_cols, batch - t.col0);
}
__device__ __forceinline__ Part part_at(const Line& p, int u, int end, int batch) {
    Part t;
    t.tile = u / p.stages;
    t.s0 = u - t.tile * p.stages;
    t.s1 = min(p.stages, t.s0 + (end - u));
    t.row_tile = t.tile / p.col_tiles;
    t.col_tile = t.tile - t.row_tile * p.col_tiles;
    part_rows(p, t, batch);
    return t;
}
// The next tile's part, from stage u of the line on (roles walk the line with this: a division each would be code in front of every loop).
__device__ __forceinline__ void next_part(const Line& p, Part& t, int u, int end, int batch) {
    ++t.tile;
    t.s0 = 0;
    t.s1 = min(p.stages, end - u);
    if (++t.col_tile == p.col_tiles) { t.col_tile = 0; ++t.row_tile; }
    part_rows(p, t, batch);
}
__device__ __forceinline__ int stage_groups(const Line& p, int stage) { return min(kStageGroups, p.groups - stage * kStageGroups); }

// Where row r of a tile lies: matrix row, its scales and biases, its output.
struct LineRow {
    int row, rows;
    const __half *s, *b;
    __half* y;
};
template <int MODE>
__device__ __forceinline__ LineRow line_row(const AffineArgs& a, const Line& p, int row_tile, int r) {
    LineRow o;
    if (MODE == kAffineGateUp || MODE == kAffineDual) {
        const int mat = r >> 6;
        o.row = row_tile * 64 + (r & 63);
        o.rows = a.rows;
        o.s = a.s[mat]; o.b = a.b[mat];
        o.y = MODE == kAffineDual && mat ? a.y2 : a.y;
    } else {
        const int seg = (row_tile >= p.first1) + (row_tile >= p.first2);
        o.row = (row_tile - (seg == 0 ? 0 : seg == 1 ? p.first1 : p.first2)) * kLineRows + r;
        const bool one = a.nseg <= 1;
        o.rows = one ? a.rows : a.seg[seg].rows;
        o.s = one ? a.s[0] : a.seg[seg].s; o.b = one ? a.b[0] : a.seg[seg].b;
        o.y = one ? a.y : a.seg[seg].y;
    }
    o.s += (size_t)o.row * p.groups;
    o.b += (size_t)o.row * p.groups;
    return o;
}

// Packed weights of one stage of the tile's rows.
template <int MODE>
__device__ __forceinline__ void request_weights(const LineMaps& maps, const Line& p, int row_tile, int stage, uint32_t dst, uint32_t bar) {
    if (MODE == kAffineGateUp || MODE == kAffineDual) {
        tma_load_2d_at(dst, &maps.w[0], stage * 128, row_tile * 64, bar);
        tma_load_2d_at(dst + kRawBytes / 2, &maps.w[1], stage * 128, row_tile * 64, bar);
    } else {
        const int seg = (row_tile >= p.first1) + (row_tile >= p.first2);
        tma_load_2d_at(dst, &maps.w[seg], stage * 128, (row_tile - (seg == 0 ? 0 : seg == 1 ? p.first1 : p.first2)) * kLineRows, bar);
    }
}

// Waits by a whole warp, all of it or none, and by one thread: bar and dead are addresses of shared memory; the word at dead is set when a
// wait gives up.
__device__ __forceinline__ uint32_t lds_word(uint32_t a) {
    uint32_t v;
    asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ bool wait_one(uint32_t bar, uint32_t parity, uint32_t dead) { return wait_alive_short(bar, parity, dead); }
__device__ __forceinline__ bool wait_warp(uint32_t bar, uint32_t parity, uint32_t dead) { return __all_sync(0xffffffffu, wait_one(bar, parity, dead)); }
__device__ __forceinline__ Part uniform(const Part& t) {
    return {uniform(t.tile), uniform(t.s0), uniform(t.s1), uniform(t.row_tile), uniform(t.col_tile), uniform(t.col0), uniform(t.live)};
}
__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}

// Scales and biases of a stage on their way to shared memory, by a warp that has little else to do, as many stages ahead as there are
// slots: a lane takes rows `row + 32 i` of the tile; dst(stage, i, which) is where the four values of such a row go, after
// wait(stage, part, stage of the part).  Every lane arrives at full(stage) when its copies have.
template <int MODE, typename Wait, typename Dst, typename Full>
__device__ __forceinline__ void feed_scales(const AffineArgs& a, const Line& p, Part t, int u0, int u1, int row, Wait wait, Dst dst, Full full) {
    constexpr int kRows = 4;
    uint32_t it = 0;
#pragma unroll 1
    for (int u = u0; u < u1; next_part(p, t, u, u1, a.batch)) {
        // Rows 64 apart may lie in two matrices; those 32 apart are in one.
        const LineRow o0 = line_row<MODE>(a, p, t.row_tile, row), o1 = line_row<MODE>(a, p, t.row_tile, row + 64);
        const __half* from[4] = {o0.s, o0.b, o1.s, o1.b};
        const int live[2] = {o0.rows - o0.row, o1.rows - o1.row}, step = 32 * p.groups;
        bool async = (p.groups & 3) == 0;  // eight bytes at a time
#pragma unroll
        for (int i = 0; i < 4; ++i) async = async && (reinterpret_cast<uintptr_t>(from[i]) & 7u) == 0;
        if (!async) {  // two bytes at a time: one stage's are on their way while the one before is stored, out of L2
#pragma unroll
            for (int i = 0; i < 2 * kRows; ++i)
                if (live[i >> 2] > (i >> 1 & 1) * 32)
#pragma unroll 1
                    for (int g = t.s0 * kStageGroups; g < min(p.groups, t.s1 * kStageGroups); g += 16) asm volatile("prefetch.global.L2 [%0];" ::"l"(from[(i >> 2) * 2 + (i & 1)] + (i >> 1 & 1) * step + g));
        }
        uint2 ahead[2 * kRows];
        auto load = [&](int st) {
            const int g = st * kStageGroups, n = stage_groups(p, st);
#pragma unroll
            for (int i = 0; i < 2 * kRows; ++i) {
                const __half* q = from[(i >> 2) * 2 + (i & 1)] + (i >> 1 & 1) * step + g;
                const bool ok = live[i >> 2] > (i >> 1 & 1) * 32;
                uint32_t h[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) h[j] = ok && j < n ? (uint32_t)__half_as_ushort(__ldg(q + j)) : 0u;
                ahead[i] = make_uint2(h[0] | h[1] << 16, h[2] | h[3] << 16);
            }
        };
        if (!async) load(t.s0);
#pragma unroll 1
        for (int st = t.s0; st < t.s1; ++st, ++it) {
            if (!wait(it, t, st)) { cp_async_wait<0>(); return; }
            const int g = st * kStageGroups;
#pragma unroll
            for (int i = 0; i < 2 * kRows; ++i) {
                const uint32_t to = dst(it, i >> 1, i & 1);
                if (!async) {
                    asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(to), "r"(ahead[i].x), "r"(ahead[i].y) : "memory");
                } else if (live[i >> 2] > (i >> 1 & 1) * 32) {
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(to), "l"(from[(i >> 2) * 2 + (i & 1)] + (i >> 1 & 1) * step + g) : "memory");
                }
            }
            if (async) asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(full(it)) : "memory");
            else {
                arrive_at(full(it));
                if (st + 1 < t.s1) load(st + 1);
            }
        }
        u += t.s1 - t.s0;
    }
    cp_async_wait<0>();
}

// A tile that several CTAs share: CTA first holds its first group, CTA last its last; a CTA has at most two such tiles, its
// first (slot 2 cta) and its last (slot 2 cta + 1), and of a tile's CTAs only the first can have another one in front of it.
struct Sharers {
    int first, last, first_slot;
    __device__ __forceinline__ int slot(int cta) const { return cta == first ? first_slot : 2 * cta; }
};
__device__ __forceinline__ Sharers sharers(const Line& p, int tile) {
    Sharers s;
    if (p.per_tile) {
        s.first = tile * p.per_tile;
        s.last = s.first + p.per_tile - 1;
    } else {
        const int start = tile * p.stages, end = start + p.stages - 1, longer = p.extra * (p.share + 1);
        s.first = start < longer ? start / (p.share + 1) : p.extra + (start - longer) / p.share;
        s.last = end < longer ? end / (p.share + 1) : p.extra + (end - longer) / p.share;
    }
    s.first_slot = 2 * s.first + (line_at(p, s.first) < tile * p.stages ? 1 : 0);
    return s;
}

constexpr int kSumWindow = 4;  // stages whose group sums of x lie in one 128-byte row of the tile that the biases multiply
// Sums of x by group as two tf32 values each, behind the shared tiles in scratch: per row of x and stage {hi of four groups, lo of four groups}.
struct GroupSums {
    float* at;  // null: the product sums for itself
    size_t floats;
};

// Whether the product takes the launch (group 64, 16-byte aligned weights and activations, no folded norm; several
// tensors where the streaming kernel takes them), and if so its maps and its line, in tiles of up to max_cols rows of x; tiles of more
// than own_cols have their group sums made in front.
bool line_plan(int mode, const AffineArgs& a, int group, int max_cols, int own_cols, LineMaps* maps, Line* line, GroupSums* sums, int* grid);

}  // namespace smelt
