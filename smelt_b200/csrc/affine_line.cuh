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
    CUtensorMap w[3], x;
};

// The work is the line of all (tile, group) units, tile after tile; a tile is 128 weight rows (64 of each matrix
// in the paired forms) and up to tile_cols rows of x.  Every CTA takes an equal stretch of the line, whatever the
// matrix' shape, so no SM waits for a last wave (192 tiles of gate/up 12288 x 4096 over 148 SMs would take two
// waves, the second one third full).  A tile that lies in the stretches of several CTAs is put together from
// fp32 sums in scratch, in column order, by the last of them to finish: results do not depend on timing.
struct Line {
    int row_tiles, col_tiles, tile_cols, groups;
    int first1, first2;  // first row tile of the second and third tensor
    int quantum;         // groups that are never split: a stage's where the row is whole stages, a tile's where there is no scratch
};

__host__ __device__ inline int line_at(const Line& p, int c, int n) {  // where CTA c of n begins
    return (int)((long)c * (p.row_tiles * p.col_tiles * p.groups / p.quantum) / n) * p.quantum;
}

// One tile's part of a stretch.
struct Part {
    int tile, g0, g1, row_tile, col0, live;  // groups [g0, g1); first row of x and how many
};
__device__ __forceinline__ Part part_at(const Line& p, int u, int end, int batch) {
    Part t;
    t.tile = u / p.groups;
    t.g0 = u - t.tile * p.groups;
    t.g1 = min(p.groups, t.g0 + (end - u));
    t.row_tile = t.tile / p.col_tiles;
    t.col0 = (t.tile - t.row_tile * p.col_tiles) * p.tile_cols;
    t.live = min(p.tile_cols, batch - t.col0);
    return t;
}

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

// Packed weights of one stage: groups g .. g + 3 of the tile's rows.
template <int MODE>
__device__ __forceinline__ void request_weights(const LineMaps& maps, const Line& p, int row_tile, int g, uint8_t* dst, uint64_t* bar) {
    if (MODE == kAffineGateUp || MODE == kAffineDual) {
        tma_load_2d(dst, &maps.w[0], g * (kLineGroup / 2), row_tile * 64, bar);
        tma_load_2d(dst + kRawBytes / 2, &maps.w[1], g * (kLineGroup / 2), row_tile * 64, bar);
    } else {
        const int seg = (row_tile >= p.first1) + (row_tile >= p.first2);
        tma_load_2d(dst, &maps.w[seg], g * (kLineGroup / 2), (row_tile - (seg == 0 ? 0 : seg == 1 ? p.first1 : p.first2)) * kLineRows, bar);
    }
}

__device__ __forceinline__ bool wait_warp(uint64_t* bar, uint32_t parity, volatile uint32_t* dead) { return __all_sync(0xffffffffu, wait_alive(bar, parity, dead)); }
// Whether a phase has completed, without waiting: several are asked at once and only what is missing is waited for.
__device__ __forceinline__ bool peek(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
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
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}

// Scales and biases of a stage on their way to shared memory, by a warp of its own: a thread that fetched its own row's
// beside its other work waited for them.  A lane takes rows `row + 32 i` of the tile; store(stage, i, group of the stage,
// {scale, bias}) is called after wait(stage), done(stage) behind it.
template <int MODE, typename Wait, typename Store, typename Done>
__device__ __forceinline__ void feed_scales(const AffineArgs& a, const Line& p, int u0, int u1, int row, Wait wait, Store store, Done done) {
    constexpr int kRows = 4;
    const bool vec = (p.quantum & 3) == 0 && (p.groups & 3) == 0;  // every stage begins at a multiple of four groups
    auto four = [&](const __half* q, int n) {
        if (vec && (reinterpret_cast<uintptr_t>(q) & 7u) == 0) return __ldg(reinterpret_cast<const uint2*>(q));
        uint32_t h[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) h[j] = j < n ? (uint32_t)__half_as_ushort(__ldg(q + j)) : 0u;
        return make_uint2(h[0] | h[1] << 16, h[2] | h[3] << 16);
    };
    uint32_t stage = 0;
    for (int u = u0; u < u1;) {
        const Part t = part_at(p, u, u1, a.batch);
#pragma unroll 1
        for (int i = 0; i < kRows; ++i) {
            const LineRow o = line_row<MODE>(a, p, t.row_tile, row + 32 * i);
            if (o.row < o.rows)
                for (int g = t.g0; g < t.g1; g += 16) {
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(o.s + g));
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(o.b + g));
                }
        }
        for (int g = t.g0; g < t.g1; g += kStageGroups, ++stage) {
            const int n = min(kStageGroups, t.g1 - g);
            uint2 s[kRows], b[kRows];
#pragma unroll
            for (int i = 0; i < kRows; ++i) {
                const LineRow o = line_row<MODE>(a, p, t.row_tile, row + 32 * i);
                const bool ok = o.row < o.rows;
                s[i] = ok ? four(o.s + g, n) : make_uint2(0, 0);
                b[i] = ok ? four(o.b + g, n) : make_uint2(0, 0);
            }
            if (!wait(stage)) return;
#pragma unroll
            for (int i = 0; i < kRows; ++i) {
                const uint32_t sw[2] = {s[i].x, s[i].y}, bw[2] = {b[i].x, b[i].y};
#pragma unroll
                for (int j = 0; j < 4; ++j) store(stage, i, j, __byte_perm(sw[j >> 1], bw[j >> 1], (j & 1) ? 0x7632 : 0x5410));
            }
            __syncwarp();
            done(stage);
        }
        u += t.g1 - t.g0;
    }
}

// A tile that several CTAs share: CTA first holds its first group, CTA last its last; a CTA has at most two such tiles, its
// first (slot 2 cta) and its last (slot 2 cta + 1), and of a tile's CTAs only the first can have another one in front of it.
struct Sharers {
    int first, last, first_slot;
    __device__ __forceinline__ int slot(int cta) const { return cta == first ? first_slot : 2 * cta; }
};
__device__ __forceinline__ Sharers sharers(const Line& p, int tile, int n) {
    const int total = p.row_tiles * p.col_tiles * p.groups / p.quantum, tile_q = p.groups / p.quantum, start = tile * tile_q;
    Sharers s;
    s.first = (int)(((start + 1l) * n - 1) / total);
    s.last = (int)(((long)(start + tile_q) * n - 1) / total);
    s.first_slot = 2 * s.first + (line_at(p, s.first, n) < tile * p.groups ? 1 : 0);
    return s;
}

// Whether the product takes the launch (group 64, 16-byte aligned weights and activations, no folded norm; several
// tensors where the streaming kernel takes them), and if so its maps and its line, in tiles of up to max_cols rows of x.
bool line_plan(int mode, const AffineArgs& a, int group, int max_cols, LineMaps* maps, Line* line, int* grid);

}  // namespace smelt
