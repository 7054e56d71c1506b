// Quantised matrix product for many rows of x (prompt chunks, decode of many sequences):
// Y[M, R] = X[M, K] . W[R, K]^T with W affine u4, group 64, on the fifth-generation tensor cores.
//
// Replaces agent_affine_qmm_fixed_batched_full and its fused gate/up form (Resources/Shaders/agent_affine_qmm.h:107-316,
// :360-742; wrappers Resources/Shaders/lut_matvec.metal:6519-6545, :6615-6635).  The tensor core multiplies the
// dequantised weight w = scale * q + bias, evaluated in fp32 with one FMA, as TWO fp16 operands: hi = half(w) and
// lo = half(w - hi).  The weights of a row in two groups are first brought near the top of fp16's range by a power of two of
// their own, so that hi + lo carries 22 significant bits of the largest of them whatever the scales are, and no weight is too
// large; the sums are multiplied by its inverse.
//
// The tensor core truncates every sum it adds to.  Over all of K in one accumulator that made 0.5 to 7 % of the fp16 results
// another value than the correctly rounded one, and all of them a little small; so an accumulator holds the products of two
// groups, the small ones first, and its contents are added in fp32 registers: 0.1 to 0.2 % of the results differ, as many as of
// the matvec family's (4096 x 4096, 32 rows: 0.12 %, exact nibbles with scale and bias applied group by group 0.12 %, all of K
// 0.53 %; 4096 x 12288: 0.12, 0.14, 1.4 %; gate and up 12288 x 4096: 0.20, 0.21, 2.6 %).
//
// Mapping.  One CTA an SM takes an equal stretch of the launch's line of work (affine_line.cuh); a tile is 128 weight
// rows, the MMA's M, by up to 256 rows of x, its N.  The roles, each on warps of its own, each a ring ahead of the next:
//   * weights: TMA, 128 rows x 256 columns of packed nibbles a stage, requested before the wait for the launch in front;
//   * activations: TMA, two 64-column groups a stage, 128-byte swizzled: the MMA's B operand as it is;
//   * scales and biases, one warp;
//   * expansion: a thread owns a weight row and turns its 64 nibbles of a group into hi and lo, in pairs, straight into
//     tensor memory, from where the MMA takes its A operand.  (An A tile in shared memory is written once and read once per
//     256 rows of x, which with the B tile's two reads and its write is more than the SM's 128 bytes a clock.)
//   * issue: sixteen K = 16 MMAs a turn of two groups, in a loop of four (unrolled, its code was fetched from beyond the
//     instruction cache every turn: 89 clocks an MMA, of 16 with 32 rows of x and 64 with 128 that it takes alone);
//   * sums and epilogue: plain, + residual, SwiGLU of gate and up, dual.
// What bounds it: up to 128 rows the expansion, about 370 instructions per row and group; with 256 the tensor pipe, which does
// the work twice, and the ends of tiles, which it waits for.  Against the form that expanded through shared memory and drained
// or staged by the same threads (us; gate/up 12288 x 4096 x 2 | 4096 x 12288 | 4096 x 4096): 32 rows 77.8 -> 57.7 | 43.9 ->
// 33.7 | 17.0 -> 15.5; 128 rows 190 -> 74.3 | 78.4 -> 41.2 | 34.4 -> 22.4; 512 rows 347 -> 226 | 164 -> 105 | 77.8 -> 52.4.
// A launch in front may take longer than a wait may (its waits on a peer are as long): every role waits for it before the first
// wait that depends on the activations, and only what needs none of them goes ahead.
// Every wait is bounded: on expiry the CTA sets bit 10 of the error word, its roles stop, copies and MMAs in flight are
// waited for (bounded too) and the tensor memory is freed.
#include "affine_line.cuh"

namespace smelt {

namespace {

constexpr int kThreads = 640, kEpilogueWarp = 4, kEpilogueWarps = 8, kExpandWarp = 12, kExpandWarps = 8;
constexpr int kEpilogueThreads = kEpilogueWarps * 32;
constexpr int kASlots = 2;     // hi | lo of two groups: 128 columns of tensor memory each
constexpr int kDone = 16;      // barriers that units' completion goes through, one after the other: no role is that far behind another
constexpr int kPowers = 16;    // turns whose powers of two are kept: two in the A slots, up to eight in accumulators

template <int N>
struct WideCfg {
    static constexpr int kHalves = N == 256 ? 2 : 1, kMma = N / kHalves;  // an MMA takes up to 128 rows of x, so that one half is drained while the other is multiplied
    static constexpr int kSlots = 256 / kMma;                             // accumulators
    static constexpr int kSums = N / 2;                                   // of a thread: two sets of epilogue warps share the columns
    static constexpr int kXBytes = N * kLineGroup * 2, kXStages = N == 256 ? 2 : 4, kRawStages = N <= 64 ? 6 : 4;  // a stage of x is two groups
    static constexpr uint32_t kSmem = kRawStages * kRawBytes + kXStages * 2 * kXBytes + 1024;
    static_assert(kSmem + 30 * 1024 <= 227u * 1024u, "shared memory");
    static_assert(kPowers >= kASlots + kSlots / kHalves, "powers");
};

// D[128 x N] (+)= A[128 x 64] . B[N x 64]^T, A from tensor memory (lane = row, two fp16 a column), as four MMAs of 16 columns: eight
// columns of tensor memory, 32 bytes in the descriptor's address field.  A whole warp calls it, one lane issues: the operands stay in
// the uniform registers that the instruction reads.
__device__ __forceinline__ void umma_f16_group(uint32_t d, uint32_t a, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q, t;\n\t.reg .b32 a1, a2, a3;\n\t.reg .b64 b1, b2, b3;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.eq.b32 t, 0, 0;\n\t"
        "add.u32 a1, %1, 8;\n\tadd.u32 a2, %1, 16;\n\tadd.u32 a3, %1, 24;\n\t"
        "add.u64 b1, %2, 2;\n\tadd.u64 b2, %2, 4;\n\tadd.u64 b3, %2, 6;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], b1, %3, t;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], b2, %3, t;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a3], b3, %3, t;\n\t}"
        ::"r"(d), "r"(a), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t t, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(t), "r"(v[0]), "r"(v[1]), "r"(v[2]),
                 "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
                 : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t t, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(t), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
// Eight nibbles -> four pairs of adjacent columns, hi and lo; s2, b2: scale and bias, twice.
__device__ __forceinline__ void expand_hi_lo(uint32_t word, uint64_t s2, uint64_t b2, uint32_t* hi, uint32_t* lo) {
    const uint64_t minus = pack2(-8388608.f, -8388608.f), neg = pack2(-1.f, -1.f);
    const uint32_t even = word & 0x0F0F0F0Fu, odd = (word >> 4) & 0x0F0F0F0Fu;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        const uint32_t sel = 0x7440u + b;  // the byte under the exponent of 2^23
        const uint64_t q = add2(pack2(__uint_as_float(__byte_perm(even, 0x4B000000u, sel)), __uint_as_float(__byte_perm(odd, 0x4B000000u, sel))), minus);
        const uint64_t w = fma2(q, s2, b2);
        const float2 wf = unpack2(w);
        const __half2 h = __floats2half2_rn(wf.x, wf.y);
        const float2 hf = __half22float2(h);
        const float2 rest = unpack2(fma2(pack2(hf.x, hf.y), neg, w));
        hi[b] = h2_as_u32(h);
        lo[b] = h2_as_u32(__floats2half2_rn(rest.x, rest.y));
    }
}

// Exponent field of the largest weight that {scale, bias} can give: |w| <= max(|bias|, |15 scale + bias|) < 2^(top - 126).
__device__ __forceinline__ uint32_t top_of(float2 f) {
    return max(__float_as_uint(fmaxf(fabsf(f.y), fabsf(fmaf(15.f, f.x, f.y)))) >> 23, 64u);
}
__device__ __forceinline__ float power_up(uint32_t top) { return __uint_as_float((268u - top) << 23); }    // 2^14 / 2^(top - 127)
__device__ __forceinline__ float power_down(uint32_t top) { return __uint_as_float((top - 14u) << 23); }  // its inverse

template <int REGS>
__device__ __forceinline__ void registers_up() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS)); }
template <int REGS>
__device__ __forceinline__ void registers_down() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS)); }

// silu(gate) * up in fp32
__device__ __forceinline__ __half swiglu_f32(float gate, float up) { return __float2half_rn(gate / (1.0f + expf(-gate)) * up); }

template <int MODE, int N>
__global__ void __launch_bounds__(kThreads, 1) affine_wide_kernel(const __grid_constant__ LineMaps maps, const AffineArgs a, const Line line) {
    using C = WideCfg<N>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* raw = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* x_tiles = raw + C::kRawStages * kRawBytes;
    __shared__ uint64_t raw_full[C::kRawStages], raw_empty[C::kRawStages], scale_full[C::kRawStages], x_full[C::kXStages], a_full[kASlots], done[kDone], acc_empty[C::kSlots];
    __shared__ uint32_t scales[C::kRawStages][kStageGroups][kLineRows];  // {scale, bias}
    __shared__ float powers[kPowers][kLineRows];                         // what the products of two groups are to be multiplied by
    __shared__ uint32_t s_tmem, s_dead, s_ticket, s_go;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    pdl_trigger();
    if (tid == 0) {
        for (int i = 0; i < C::kRawStages; ++i) { mbar_init(&raw_full[i], 1); mbar_init(&raw_empty[i], kExpandWarps); mbar_init(&scale_full[i], 1); }
        for (int i = 0; i < C::kXStages; ++i) mbar_init(&x_full[i], 1);
        for (int i = 0; i < kASlots; ++i) mbar_init(&a_full[i], 4);
        for (int i = 0; i < kDone; ++i) mbar_init(&done[i], 2);
        for (int i = 0; i < C::kSlots; ++i) mbar_init(&acc_empty[i], kEpilogueWarps);
        s_dead = 0u;
        mbar_fence_init();
        fence_async_smem();
    }
    if (warp == 2) tmem_alloc(&s_tmem, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem, tmem_a = tmem + 256;
    volatile uint32_t* dead = &s_dead;
    const int u0 = line_at(line, blockIdx.x, gridDim.x), u1 = line_at(line, blockIdx.x + 1, gridDim.x);
    const int mma_cols = line.tile_cols / C::kHalves;
    // A turn is two groups, or the last one of a part that has an odd number; a unit is a turn's MMAs into one accumulator.
    auto turn_done = [&](uint32_t turn, auto wait) {  // all of the turn's MMAs
        const uint32_t unit = turn * C::kHalves + C::kHalves - 1;
        return wait(&done[unit % kDone], (unit / kDone) & 1, dead);
    };
    // Weight row (of the tile as the weights arrive) that tensor-memory lane r stands for: gate and up rows of one result 16 lanes apart
    auto tile_row = [](int r) { return MODE == kAffineGateUp ? (r & 16) * 4 + (r >> 5) * 16 + (r & 15) : r; };
    // The sums of many rows of x take up to 128 registers of an epilogue thread: 128 roles + 256 epilogue + 256 expand <= 640 x 96, the launch's.
    if (warp < kEpilogueWarp) {
    if (N >= 128) registers_down<N == 256 ? 48 : 64>();
    if (warp == 0) {
        // ── packed weights ──
        if (lane == 0) {
            uint32_t it = 0;
            bool alive = true;
            for (int u = u0; u < u1 && alive;) {
                const Part t = part_at(line, u, u1, a.batch);
                for (int g = t.g0; g < t.g1; g += kStageGroups, ++it) {
                    const uint32_t s = it % C::kRawStages, use = it / C::kRawStages;
                    if (it == C::kRawStages) pdl_wait();
                    if (use > 0 && !(alive = wait_alive(&raw_empty[s], (use - 1) & 1, dead))) break;
                    mbar_arrive_expect_tx(&raw_full[s], kRawBytes);
                    request_weights<MODE>(maps, line, t.row_tile, g, raw + s * kRawBytes, &raw_full[s]);
                }
                u += t.g1 - t.g0;
            }
            for (uint32_t i = it > C::kRawStages ? it - C::kRawStages : 0; i < it; ++i) mbar_poll_bounded(&raw_full[i % C::kRawStages], (i / C::kRawStages) & 1);  // no copy may land after the CTA has left
        }
    } else if (warp == 1) {
        // ── activations ──
        if (lane == 0) {
            pdl_wait();
            const bool skip = dyn_skip(a.dyn);
            if (skip) *dead = 2u;  // a guarded launch that is not to run: the other roles stop at their next wait
            uint32_t it = 0;
            bool alive = !skip;
            const uint32_t bytes = (uint32_t)line.tile_cols * kLineGroup * 2;
            for (int u = u0; u < u1 && alive;) {
                const Part t = part_at(line, u, u1, a.batch);
                for (int g = t.g0; g < t.g1; g += 2, ++it) {
                    const uint32_t s = it % C::kXStages;
                    if (it >= C::kXStages && !(alive = turn_done(it - C::kXStages, wait_alive))) break;
                    const int n = min(2, t.g1 - g);
                    mbar_arrive_expect_tx(&x_full[s], bytes * n);
                    for (int i = 0; i < n; ++i) tma_load_2d(x_tiles + (2 * s + i) * C::kXBytes, &maps.x, (g + i) * kLineGroup, t.col0, &x_full[s]);
                }
                u += t.g1 - t.g0;
            }
            for (uint32_t i = it > C::kXStages ? it - C::kXStages : 0; i < it; ++i) mbar_poll_bounded(&x_full[i % C::kXStages], (i / C::kXStages) & 1);
        }
    } else if (warp == 2) {
        // ── issue ──
        const uint32_t idesc = (1u << 4) | ((uint32_t)(mma_cols >> 3) << 17) | ((uint32_t)(kLineRows >> 4) << 24);  // f32 += f16 x f16, K-major both
        const uint32_t x_base = smem_u32(x_tiles);
        pdl_wait();
        uint32_t turn = 0, unit = 0;
        bool alive = true;
        for (int u = u0; u < u1 && alive;) {
            const Part t = part_at(line, u, u1, a.batch);
            for (int g = t.g0; g < t.g1 && alive; g += 2, ++turn) {
                const uint32_t as = turn % kASlots, xs = turn % C::kXStages, ap = (turn / kASlots) & 1, xp = (turn / C::kXStages) & 1;
                const bool two = t.g1 - g > 1, b0 = peek(&x_full[xs], xp), b1 = peek(&a_full[as], ap);
                if (!__all_sync(0xffffffffu, b0 && b1)) alive = wait_warp(&x_full[xs], xp, dead) && wait_warp(&a_full[as], ap, dead);
#pragma unroll 1
                for (int h = 0; h < C::kHalves && alive; ++h) {
                    const uint32_t slot = unit % C::kSlots, use = unit / C::kSlots;
                    if (use > 0 && !(alive = wait_warp(&acc_empty[slot], (use - 1) & 1, dead))) break;
                    tc_fence_after();
                    const uint64_t b = smem_desc_sw128(x_base + 2 * xs * C::kXBytes + h * mma_cols * 128);
#pragma unroll 1
                    for (int j = two ? 0 : 2; j < 4; ++j) {  // lo and lo, hi and hi: the small products first, what is cut off their sums is small too
                        const int i = two ? j & 1 : 0, lo = two ? j < 2 : j == 2;
                        umma_f16_group(tmem + slot * C::kMma, tmem_a + as * 128 + i * 64 + lo * 32, b + i * (C::kXBytes / 16), idesc, j > 0 && (two || j > 2) ? 1u : 0u);
                    }
                    if (elect_one()) {
                        umma_commit(&done[unit % kDone]);
                        mbar_arrive(&done[unit % kDone]);  // hands the power on, which this warp has seen with a_full
                    }
                    __syncwarp();
                    ++unit;
                }
            }
            u += t.g1 - t.g0;
        }
        if (unit > 0) mbar_poll_bounded(&done[(unit - 1) % kDone], ((unit - 1) / kDone) & 1);  // the MMAs in flight read shared memory and write tensor memory
    } else if (warp == 3) {
        // ── scales and biases ──
        feed_scales<MODE>(a, line, u0, u1, lane,
            [&](uint32_t it) {
                if (it == C::kRawStages) pdl_wait();
                return it < C::kRawStages || wait_warp(&raw_empty[it % C::kRawStages], (it / C::kRawStages - 1) & 1, dead);
            },
            [&](uint32_t it, int i, int j, uint32_t sb) { scales[it % C::kRawStages][j][lane + 32 * i] = sb; },
            [&](uint32_t it) { if (lane == 0) mbar_arrive(&scale_full[it % C::kRawStages]); });
    }
    } else if (warp < kExpandWarp) {
        if (N >= 128) registers_up<N == 256 ? 160 : 120>();
        // ── sums and epilogue: two sets of four warps, each half of an accumulator's columns ──
        const int set = (warp - kEpilogueWarp) >> 2, quad = warp & 3, r = quad * 32 + lane;
        const uint32_t lane_base = tmem + ((uint32_t)(quad * 32) << 16);
        const bool leader = tid == kEpilogueWarp * 32;
        const int set_cols = mma_cols / 2;  // a multiple of eight
        auto all_sync = [] { asm volatile("bar.sync 1, %0;" ::"n"(kEpilogueThreads) : "memory"); };
        uint32_t unit = 0, turns = 0;
        pdl_wait();
        for (int u = u0; u < u1;) {
            const Part t = part_at(line, u, u1, a.batch);
            uint64_t sums[C::kSums / 2];
#pragma unroll
            for (int j = 0; j < C::kSums / 2; ++j) sums[j] = 0;
            bool alive = true;
            for (int g = t.g0; g < t.g1 && alive; g += 2, ++turns) {
#pragma unroll
                for (int h = 0; h < C::kHalves; ++h, ++unit) {
                    const uint32_t slot = unit % C::kSlots, src = lane_base + slot * C::kMma + set * set_cols;
                    if (!(alive = wait_warp(&done[unit % kDone], (unit / kDone) & 1, dead))) break;
                    tc_fence_after();
                    const float power = powers[turns % kPowers][r];
                    const uint64_t power2 = pack2(power, power);
                    // sixteen columns on their way while the sixteen before them are added, where the registers allow it
                    constexpr int kBatches = C::kMma / 32, kAhead = N == 256 ? 0 : 1;
                    uint32_t v[1 + kAhead][16];
                    tmem_ld16(src, v[0]);
#pragma unroll
                    for (int i = 0; i < kBatches; ++i) {
                        if (i > 0 && 16 * i >= set_cols) break;
                        const bool more = i + 1 < kBatches && 16 * (i + 1) < set_cols;
                        tmem_wait_ld16(v[i & kAhead]);
                        if (kAhead && more) tmem_ld16(src + 16 * (i + 1), v[(i + 1) & kAhead]);
                        if (!more) {
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive(&acc_empty[slot]);
                        }
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            uint64_t& s = sums[h * (C::kMma / 4) + 8 * i + j];
                            s = fma2(pack2(__uint_as_float(v[i & kAhead][2 * j]), __uint_as_float(v[i & kAhead][2 * j + 1])), power2, s);
                        }
                        if (!kAhead && more) tmem_ld16(src + 16 * (i + 1), v[0]);
                    }
                }
            }
            if (!alive && *dead == 0u) *dead = 1u;
            all_sync();  // the eight warps go on together or not at all
            if (leader) s_go = *dead == 0u ? 1u : 0u;
            all_sync();
            if (s_go == 0u) break;
            // The sums go through scratch, a tile's alone as well: what comes then is a short loop (unrolled over the registers, its
            // code came from beyond the instruction cache: a tile of gate and up cost 52,000 clocks).
            const size_t part = (size_t)line.tile_cols * kLineRows;
            const bool shared = t.g0 != 0 || t.g1 != line.groups;
            Sharers sh = {(int)blockIdx.x, (int)blockIdx.x, 2 * (int)blockIdx.x + 1};  // a slot that this CTA's last tile has, if it is shared
            if (shared) sh = sharers(line, t.tile, gridDim.x);
            float4* mine = reinterpret_cast<float4*>(a.part_scratch + (size_t)sh.slot(blockIdx.x) * part) + set * set_cols / 4 * kLineRows + r;  // [four columns][row]
#pragma unroll
            for (int h = 0; h < C::kHalves; ++h)
#pragma unroll
                for (int c0 = 0; c0 < C::kMma / 2; c0 += 4)
                    if (c0 < set_cols) {
                        const float2 lo = unpack2(sums[(h * (C::kMma / 2) + c0) / 2]), hi = unpack2(sums[(h * (C::kMma / 2) + c0) / 2 + 1]);
                        __stcg(mine + (h * mma_cols + c0) / 4 * kLineRows, make_float4(lo.x, lo.y, hi.x, hi.y));
                    }
            bool finish = true;
            if (shared) {
                __threadfence();
                all_sync();
                if (leader) s_ticket = (uint32_t)atomicAdd(a.part_counters + t.tile, 1);
                all_sync();
                finish = s_ticket == (uint32_t)(sh.last - sh.first);
                if (finish) {
                    __threadfence();
                    if (leader) a.part_counters[t.tile] = 0;  // the next launch finds every counter at zero
                }
            }
            if (finish) {
                const LineRow o = line_row<MODE>(a, line, t.row_tile, tile_row(r));
                const bool row_ok = o.row < o.rows;
                auto write = [&](int c, float (&v)[8]) {  // eight columns of the tile from c on
                    const int n = t.live - c;
                    if (MODE == kAffineGateUp) {
                        // lanes 16 apart have gate and up of one row of the result: the gate's takes the first four columns, the up's the others
                        const bool up = r & 16;
                        __half* y = o.y + (size_t)(t.col0 + c + (up ? 4 : 0)) * o.rows + o.row;
#pragma unroll 1
                        for (int j = 0; j < 4; ++j, y += o.rows) {
                            const float other = __shfl_xor_sync(0xffffffffu, up ? v[0] : v[4], 16);
                            const __half z = swiglu_f32(up ? other : v[0], up ? v[4] : other);  // lut_matvec.metal:2228
                            if (row_ok && j + (up ? 4 : 0) < n) *y = z;
#pragma unroll
                            for (int i = 0; i < 7; ++i) v[i] = v[i + 1];
                        }
                    } else if (row_ok) {
                        const size_t at = (size_t)(t.col0 + c) * o.rows + o.row;
                        __half res[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            if (MODE == kAffineAdd) res[j] = j < n ? a.residual[at + (size_t)j * o.rows] : __half(0.f);
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            if (j < n) o.y[at + (size_t)j * o.rows] = MODE == kAffineAdd ? __hadd(__float2half_rn(v[j]), res[j]) : __float2half_rn(v[j]);  // lut_matvec.metal:1802-1803
                    }
                };
                // A step: eight columns of four CTAs' sums; the next step's are on their way while these are added (one after the
                // other a step cost 1 us, most of it latency).
                const int chunks = set_cols / 8, rounds = (sh.last - sh.first + 4) / 4, steps = C::kHalves * chunks * rounds;
                float4 f[4][2];
                auto request = [&](int step) {
                    const int c = sh.first + step % rounds * 4, i = step / rounds, col = i / chunks * mma_cols + set * set_cols + i % chunks * 8;
#pragma unroll
                    for (int z = 0; z < 4; ++z) {
                        const float4* q = reinterpret_cast<const float4*>(a.part_scratch + (size_t)sh.slot(min(c + z, sh.last)) * part) + col / 4 * kLineRows + r;
#pragma unroll
                        for (int j = 0; j < 2; ++j) f[z][j] = c + z <= sh.last ? __ldcg(q + j * kLineRows) : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
                };
                float v[8];
                request(0);
#pragma unroll 1
                for (int step = 0; step < steps; ++step) {
                    if (step % rounds == 0)
#pragma unroll
                        for (int j = 0; j < 8; ++j) v[j] = 0.f;
#pragma unroll
                    for (int z = 0; z < 4; ++z)
#pragma unroll
                        for (int j = 0; j < 2; ++j) { v[4 * j] += f[z][j].x; v[4 * j + 1] += f[z][j].y; v[4 * j + 2] += f[z][j].z; v[4 * j + 3] += f[z][j].w; }
                    if (step + 1 < steps) request(step + 1);
                    const int i = step / rounds, col = i / chunks * mma_cols + set * set_cols + i % chunks * 8;
                    if (step % rounds == rounds - 1 && col < t.live) write(col, v);
                }
            }
            __syncwarp();  // the next tensor-memory load needs the whole warp
            u += t.g1 - t.g0;
        }
    } else {
        if (N >= 128) registers_down<N == 256 ? 56 : 88>();
        // ── expansion: two sets of four warps take turns ──
        const int set = (warp - kExpandWarp) >> 2, quad = warp & 3, r = quad * 32 + lane, row = tile_row(r);
        const uint32_t dst = tmem_a + ((uint32_t)(quad * 32) << 16), raw_a = smem_u32(raw);
        uint32_t turn = 0, stage = 0;
        bool alive = true;
        for (int u = u0; u < u1 && alive;) {
            const Part t = part_at(line, u, u1, a.batch);
            for (int g = t.g0; g < t.g1 && alive; g += kStageGroups, ++stage) {
                const uint32_t s = stage % C::kRawStages, ph = (stage / C::kRawStages) & 1;
                const bool b0 = peek(&raw_full[s], ph), b1 = peek(&scale_full[s], ph);
                if ((!__all_sync(0xffffffffu, b0) && !wait_warp(&raw_full[s], ph, dead)) || (!__all_sync(0xffffffffu, b1) && !wait_warp(&scale_full[s], ph, dead))) { alive = false; break; }
                const uint32_t src = raw_a + s * kRawBytes + row * 128;
                const int n = min(kStageGroups, t.g1 - g);
                for (int k = 0; 2 * k < n; ++k, ++turn) {
                    const uint32_t as = turn % kASlots;
                    if ((int)as != set) continue;
                    if (turn >= kASlots && turn < 2 * kASlots) pdl_wait();
                    if (turn >= kASlots && !turn_done(turn - kASlots, wait_warp)) { alive = false; break; }
                    tc_fence_after();
                    const int last = min(n - 1, 2 * k + 1);
                    const uint32_t top = max(top_of(__half22float2(u32_as_h2(scales[s][2 * k][row]))), top_of(__half22float2(u32_as_h2(scales[s][last][row]))));
                    const float up = power_up(top);
                    powers[turn % kPowers][r] = power_down(top);
#pragma unroll 1
                    for (int i = 2 * k; i <= last; ++i) {
                        const float2 f = __half22float2(u32_as_h2(scales[s][i][row]));
                        const uint64_t s2 = pack2(f.x * up, f.x * up), b2 = pack2(f.y * up, f.y * up);
#pragma unroll
                        for (int p = 0; p < 2; ++p) {
                            const uint4 v = lds128(src + (((2 * i + p) ^ (row & 7)) << 4));
                            const uint32_t word[4] = {v.x, v.y, v.z, v.w}, to = dst + as * 128 + (i & 1) * 64 + p * 16;
                            if constexpr (N == 256) {  // few registers
#pragma unroll
                                for (int q = 0; q < 4; q += 2) {
                                    uint32_t hi[8], lo[8];
                                    expand_hi_lo(word[q], s2, b2, hi, lo);
                                    expand_hi_lo(word[q + 1], s2, b2, hi + 4, lo + 4);
                                    tmem_st8(to + 4 * q, hi);
                                    tmem_st8(to + 32 + 4 * q, lo);
                                }
                            } else {
                                uint32_t hi[16], lo[16];
#pragma unroll
                                for (int q = 0; q < 4; ++q) expand_hi_lo(word[q], s2, b2, hi + 4 * q, lo + 4 * q);
                                tmem_st16(to, hi);
                                tmem_st16(to + 32, lo);
                            }
                        }
                    }
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&a_full[as]);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&raw_empty[s]);
            }
            u += t.g1 - t.g0;
        }
    }
    __syncthreads();
    if (tid == 0 && a.err && *dead == 1u) atomicOr(a.err, 0x400u);
    tc_fence_before();
    __syncthreads();
    if (warp == 2) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

template <int MODE, int N>
cudaError_t launch_wide_t(const Launch& l, AffineArgs a, const LineMaps& maps, const Line& line, int grid) {
    auto kern = affine_wide_kernel<MODE, N>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WideCfg<N>::kSmem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = WideCfg<N>::kSmem;
    cfg.stream = l.stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = l.pdl ? 1 : 0;
    prefer_max_shared(kern);
    a.dyn = dev_dyn(l);
    return cudaLaunchKernelEx(&cfg, kern, maps, a, line);
}

template <int MODE>
cudaError_t launch_wide(const Launch& l, const AffineArgs& a, const LineMaps& maps, const Line& line, int grid) {
    if (line.tile_cols <= 32) return launch_wide_t<MODE, 32>(l, a, maps, line, grid);
    if (line.tile_cols <= 64) return launch_wide_t<MODE, 64>(l, a, maps, line, grid);
    return line.tile_cols <= 128 ? launch_wide_t<MODE, 128>(l, a, maps, line, grid) : launch_wide_t<MODE, 256>(l, a, maps, line, grid);
}

}  // namespace

cudaError_t launch_affine_wide(const Launch& l, int mode, const AffineArgs& a, int group, bool* handled) {
    LineMaps maps = {};
    Line line;
    int grid = 0;
    *handled = line_plan(mode, a, group, 256, &maps, &line, &grid);
    if (!*handled) return cudaSuccess;
    switch (mode) {
        case kAffinePlain: return launch_wide<kAffinePlain>(l, a, maps, line, grid);
        case kAffineAdd: return launch_wide<kAffineAdd>(l, a, maps, line, grid);
        case kAffineGateUp: return launch_wide<kAffineGateUp>(l, a, maps, line, grid);
        case kAffineDual: return launch_wide<kAffineDual>(l, a, maps, line, grid);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace smelt
