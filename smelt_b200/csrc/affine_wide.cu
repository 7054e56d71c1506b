// Quantised matrix product for many rows of x (prompt chunks, decode of many sequences):
// Y[M, R] = X[M, K] . W[R, K]^T with W affine u4, group 64, on the fifth-generation tensor cores.
//
// Replaces agent_affine_qmm_fixed_batched_full and its fused gate/up form (Resources/Shaders/agent_affine_qmm.h:107-316,
// :360-742; wrappers Resources/Shaders/lut_matvec.metal:6519-6545, :6615-6635), in their factored form: per group
// y += scale * sum(q x) + bias * sum(x).  The tensor core multiplies the nibbles (exact in fp16) by x, one accumulator a group;
// epilogue warps multiply what they drain by the scale and add it to fp32 registers.  The nibbles are centred (q - c, c = 8 up to 32 rows) and
// the bias is bias + c scale, so that neither sum is much larger than the result.  The tensor core truncates what it adds to, here four
// K = 16 products at a time.  Share of fp16 results that are not the correctly rounded ones, against two fp16 operands per
// dequantised weight summed over two groups (before -> now): 4096 x 4096, 32 rows 0.11 -> 0.07 %, 512 rows 0.11 -> 0.08; gate and
// up 12288 x 4096, 32 rows 0.19 -> 0.10, 512 rows 0.19 -> 0.14.  Up to 32 rows the four groups of a turn are added up before they meet the
// running sum, which rounds once for them: with two roundings a group, 5120 x 17408 had 0.16 % at 8 rows and 0.17 at 32, where the kernels
// in front have 0.09 and 0.14; now 0.09 and 0.09 (4096 x 12288 + residual, 9 rows: 0.024, in front 0.020, now 0.009).  It costs nothing.
//
// bias * sum(x).  Tiles of up to 64 rows of x: four warps sum x from shared memory.  More: the sums are made once in front
// (group_sums_kernel), as they would cost every CTA four warps' issue slots.  Tiles of up to 32 rows: the epilogue adds the products in fp32.
// More: the sums are kept as two tf32 values each, and the biases of up to sixteen groups multiply them on the tensor core as one
// more turn; c is chosen for each group, to the nearest eighth, so that these operands are small (tf32_bias).  With c = 8, x of mean 0.5 and biases
// of -7.5 scales, 0.24 % of the results of 4096 columns were misrounded (before the tensor core had the biases: 0.11 %), now 0.07; it costs
// 1 % of the time.
// (When that was decided: the epilogue's way with 64 rows of gate/up 12288 x 4096 50.2 us instead of 44.7; the tensor core's with 32 rows, a turn
// more for each of a CTA's short stretches, a step of 32 sequences 3.88 ms instead of 3.75.)
//
// Mapping.  One CTA an SM takes a stretch of the launch's line of work (affine_line.cuh); a tile is 128 weight
// rows, the MMA's M, by up to 128 rows of x, its N.  The roles, each on warps of its own, each a ring ahead of the next:
//   * weights, TMA, 128 rows x 256 columns of packed nibbles a stage, and their scales and biases, cp.async: requested before the
//     wait for the launch in front;
//   * activations: TMA, 128-byte swizzled: the MMA's B operand as it is;
//   * expansion: a thread owns a weight row and turns its nibbles of a group into fp16 pairs straight in tensor memory, from where
//     the MMA takes its A operand: 11 instructions for eight nibbles;
//   * issue: two warps take turns;
//   * sums and epilogue, eight warps: plain, + residual, SwiGLU of gate and up, dual.  A turn is 128 columns of tensor memory: four
//     groups of 32 rows of x, two of 64, one of 128.
// What bounds it: instruction issue (gate/up 12288 x 4096 with 32 | 64 | 512 rows: 0.60 | 0.66 | 0.72 an SM quarter and clock; the tensor pipe is
// active 10 | 14 | 29 % of the cycles, DRAM 19 | 14 | 5) and the handing over between the roles.  What cost most on the way here: code
// beyond what the instruction cache holds (wait loops unrolled by the compiler), spilled registers (the shared memory leaves no first-level
// cache: a reload is an L2 round trip), waits with a time hint (a timed loop each), shared addresses made anew at every use, packed
// FMAs (a move each).
// us, graph replay over distinct weights, before -> now (gate/up 12288 x 4096 x 2 | 4096 x 12288 | 4096 x 4096): 32 rows
// 58.4 -> 30.7 | 34.5 -> 18.4 | 15.6 -> 10.7; 64 rows 63.8 -> 44.4 | 38.3 -> 27.4 | 18.4 -> 14.0; 128 rows 74.4 -> 55.9 |
// 41.4 -> 37.3 | 22.5 -> 19.0; 512 rows 243 -> 181 | 105 -> 84 | 51.5 -> 35.1.
// A launch in front may take longer than a wait may (its waits on a peer are as long): every role waits for it before the first
// wait that depends on the activations, and only what needs none of them goes ahead.
// Every wait is bounded: on expiry the CTA sets bit 10 of the error word, its roles stop, copies and MMAs in flight are
// waited for (bounded too) and the tensor memory is freed.
#include "affine_line.cuh"

namespace smelt {

namespace {

constexpr int kEpilogueWarp = 4, kEpilogueWarps = 8, kExpandWarp = 12, kExpandWarps = 8, kSumWarp = 20, kSumWarps = 4;
constexpr int kEpilogueThreads = kEpilogueWarps * 32;
constexpr int kDone = 16;      // barriers that units' completion goes through, one after the other: no role is that far behind another
constexpr int kOwnCols = 64;   // up to so many rows of x a tile's CTAs make the group sums themselves
constexpr float kNibble = 512.f;  // the tensor core gets nibbles as 2^-9 of their value

// A position in a ring of barriers and the parity of its present use.
template <int N>
struct Ring {
    uint32_t i = 0, phase = 0;
    __device__ __forceinline__ void next(uint32_t steps = 1) {
        if ((i += steps) >= N) { i -= N; phase ^= 1u; }
    }
};

// Whether a wait of an issuing warp can be taken for one of an earlier use of its barrier: a parity tells a phase only from the one next to it, and
// each of the two warps waits on its own turns, every second one, only.  When a warp comes to turn t it knows of a use in turn `before` if that
// was its own, or if the accumulator of its turn in front, t - 2, was only free once that turn had been drained.  Walks tiles of rows of up to 20
// groups from every stage on, short last stages among them.
constexpr bool issue_waits_hold(int turn_groups, int slots, int x_stages, int a_slots, int windows, bool folded) {
    for (int groups = 1; groups <= 20; ++groups) {
        const int stages = (groups + kStageGroups - 1) / kStageGroups;
        for (int first = 0; first < stages; ++first) {
            int x_used[8] = {}, a_used[8] = {}, window_used[4] = {};  // turn + 1 of a position's latest use
            int t = 0, x = 0, window = 0;
            auto known = [&](int before) { return before == 0 || ((before - 1) ^ t) % 2 == 0 || before - 1 <= t - 2 - slots; };
            for (int tile = 0; tile < 4; ++tile)
                for (int st = tile ? 0 : first, held = 1; st < stages; ++st, ++held) {
                    const int n = groups - st * kStageGroups < kStageGroups ? groups - st * kStageGroups : kStageGroups;
                    for (int k = 0; k < n; k += turn_groups, ++t, ++x) {
                        if (!known(x_used[x % x_stages]) || !known(a_used[t % a_slots])) return false;
                        x_used[x % x_stages] = a_used[t % a_slots] = t + 1;
                    }
                    if (folded || (held % kSumWindow != 0 && st + 1 != stages)) continue;
                    if (!known(window_used[window % windows]) || !known(a_used[t % a_slots])) return false;
                    window_used[window % windows] = a_used[t % a_slots] = t + 1;
                    ++window;
                    ++t;
                }
        }
    }
    return true;
}

template <int N>
struct WideCfg {
    static constexpr bool kOwn = N <= kOwnCols;    // the CTA sums x itself
    static constexpr bool kFolded = N <= 32;       // and the epilogue adds bias * sum in fp32: no turn for the biases
    static constexpr int kThreads = kOwn ? 768 : 640;
    // Registers of the roles in front, the epilogue, and the others; together no more than the launch's.
    static constexpr int kFront = 48, kDrain = N == 128 ? 160 : 128, kBehind = 56;
    static constexpr int kTurn = N <= 32 ? 4 : N <= 64 ? 2 : 1;           // groups of a turn: multiplied into accumulators side by side
    static constexpr int kSlots = kOwn ? 2 : 3;                           // of accumulators: 128 columns of tensor memory each
    static constexpr int kASlots = kOwn ? 256 / (32 * kTurn) : 4, kACol = kSlots * 128;
    static constexpr int kXBytes = N * kLineGroup * 2, kXStages = N == 128 ? 5 : 4, kRawStages = N == 128 ? 4 : 6;  // a stage of x is a turn's
    static constexpr int kScaleStages = kFolded ? 8 : 12;
    // Group sums of kSumWindow stages.  Two: with one, a window of one short last stage begins three turns after the window in front, which
    // the other issuing warp took and this one has not seen arrive.
    static constexpr int kWindows = 2, kWindow = kFolded ? 0 : N * 128;
    static constexpr int kFoldedSlots = 4;                                // turns whose sums are kept for the epilogue
    static constexpr uint32_t kSmem = kRawStages * kRawBytes + kXStages * kTurn * kXBytes + kWindows * kWindow + 1024;
    static_assert(kSmem + 28 * 1024 <= 227u * 1024u, "shared memory");
    static_assert(kACol + kASlots * kTurn * 32 <= 512 && kTurn * N <= 128, "tensor memory");
    static_assert(kScaleStages >= 2 * kSumWindow, "the biases of a window wait for it");
    static_assert(issue_waits_hold(kTurn, kSlots, kXStages, kASlots, kWindows, kFolded), "an issuing warp could take a barrier's earlier use for this one");
    // Barriers, by the address of the first one of a kind.
    static constexpr int kRawFull = 0, kRawEmpty = kRawFull + kRawStages, kScaleFull = kRawEmpty + kRawStages, kScaleEmpty = kScaleFull + kScaleStages, kXFull = kScaleEmpty + kScaleStages,
                         kXEmpty = kXFull + kXStages, kAFull = kXEmpty + kXStages, kTurnDone = kAFull + kASlots, kAccEmpty = kTurnDone + kDone, kWindowFull = kAccEmpty + kSlots,
                         kWindowEmpty = kWindowFull + kWindows, kSumFull = kWindowEmpty + kWindows, kSumEmpty = kSumFull + kFoldedSlots, kBarriers = kSumEmpty + kFoldedSlots;
    static_assert(128 * kFront + kEpilogueThreads * kDrain + (kThreads - 128 - kEpilogueThreads) * kBehind <= kThreads * (65536 / kThreads / 8 * 8), "registers");
};

template <int N>
struct WideShared {
    using C = WideCfg<N>;
    uint64_t bars[C::kBarriers];
    uint2 scales[C::kScaleStages][2][kLineRows];                                    // four scales and four biases of a row
    alignas(16) float folded[C::kFolded ? C::kFoldedSlots : 1][C::kTurn][C::kFolded ? N : 4];  // sums of x by group
    uint32_t x_turns[C::kXStages];                                                  // the turn that reads a stage of x
    uint32_t tmem, dead, ticket, go;
    int u0, u1;
    Part first;
};

// D[128 x N] = A[128 x 64] . B[N x 64]^T, A from tensor memory (lane = row, two fp16 a column), as four MMAs of 16 columns: eight
// columns of tensor memory, 32 bytes in the descriptor's address field.  A whole warp calls it, one lane issues: the operands stay in
// the uniform registers that the instruction reads.
__device__ __forceinline__ void umma_f16_group(uint32_t d, uint32_t a, uint64_t b_desc, uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .pred p, q, t;\n\t.reg .b32 a1, a2, a3;\n\t.reg .b64 b1, b2, b3;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "setp.ne.b32 p, 0, 0;\n\tsetp.eq.b32 t, 0, 0;\n\t"
        "add.u32 a1, %1, 8;\n\tadd.u32 a2, %1, 16;\n\tadd.u32 a3, %1, 24;\n\t"
        "add.u64 b1, %2, 2;\n\tadd.u64 b2, %2, 4;\n\tadd.u64 b3, %2, 6;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], b1, %3, t;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], b2, %3, t;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a3], b3, %3, t;\n\t}"
        ::"r"(d), "r"(a), "l"(b_desc), "r"(idesc)
        : "memory");
}
// D (+)= A[128 x 8] . B[N x 8]^T in tf32, likewise.
__device__ __forceinline__ void umma_tf32_step(uint32_t d, uint32_t a, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}"
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
// What a group's sum of x is multiplied by when its nibbles go to the tensor core as q - c: bias + c scale, with c the multiple of 1/8 that makes
// it smallest.  The tensor core truncates the sum of these products too, over up to sixteen groups, where x has a mean that is far from
// small beside the result.  q - c is exact in fp16 up to |c| = 240; bias + c scale, at most a sixteenth of the scale, has no more than
// eleven bits, so that a tf32 operand holds it.  Else (a scale of zero, a bias beyond 240 scales) c is 0.  minus: -c / 512 twice.
__device__ __forceinline__ float tf32_bias(float s, float b, uint32_t* minus) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(s));
    const float k = __fadd_rn(fmaf(-8.f * b, r, 12582912.f), -12582912.f), t = fmaf(0.125f * k, s, b);  // k: to the nearest whole number
    const bool centred = fabsf(k) <= 1920.f && (__float_as_uint(t) & 0x1FFFu) == 0u;
    *minus = centred ? h2_as_u32(__float2half2_rn(k * (-1.f / 4096.f))) : 0u;
    return centred ? t : b;
}
// Eight nibbles -> four pairs of adjacent columns: a byte that holds a nibble is an fp16 of 2^-24 of its value, brought to 2^-9 of it (and
// centred) by one packed FMA.  (The tensor core takes the subnormals exactly too, but aligns their products by an exponent that is up to ten
// bits too high: four times as many results were misrounded.)
__device__ __forceinline__ void expand_nibbles(uint32_t word, uint32_t minus, uint32_t* pair) {
    const uint32_t even = word & 0x0F0F0F0Fu, odd = (word >> 4) & 0x0F0F0F0Fu;
    // 8 and C: the sign of such a byte, zero
    asm("prmt.b32 %0, %4, %5, 0xC480;\n\tprmt.b32 %1, %4, %5, 0xD591;\n\tprmt.b32 %2, %4, %5, 0xE6A2;\n\tprmt.b32 %3, %4, %5, 0xF7B3;"
        : "=&r"(pair[0]), "=&r"(pair[1]), "=&r"(pair[2]), "=&r"(pair[3])
        : "r"(even), "r"(odd));
#pragma unroll
    for (int b = 0; b < 4; ++b) asm("fma.rn.f16x2 %0, %0, %1, %2;" : "+r"(pair[b]) : "r"(0x78007800u), "r"(minus));  // 2^15
}
__device__ __forceinline__ uint32_t lds_u16(uint32_t a) {
    uint16_t h;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(h) : "r"(a));
    return h;
}
__device__ __forceinline__ void sts_word(uint32_t a, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory"); }
__device__ __forceinline__ float tf32_of(float v) {
    uint32_t u;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(u) : "f"(v));
    return __uint_as_float(u);
}

template <int REGS>
__device__ __forceinline__ void registers_up() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS)); }
template <int REGS>
__device__ __forceinline__ void registers_down() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS)); }

// silu(gate) * up in fp32
__device__ __forceinline__ __half swiglu_f32(float gate, float up) { return __float2half_rn(gate / (1.0f + expf(-gate)) * up); }

// Sums of x by group for tiles of many rows, as hi + lo of eleven bits each (what a tf32 operand holds): a warp takes four groups of a row.
__global__ void __launch_bounds__(256) group_sums_kernel(const __half* __restrict__ x, float* __restrict__ out, int batch, int cols, int stages) {
    pdl_trigger();
    pdl_wait();
    const int lane = threadIdx.x & 31, row = blockIdx.x;
    for (int st = blockIdx.y * 8 + (threadIdx.x >> 5); st < stages; st += gridDim.y * 8) {
        const int c = st * (kStageGroups * kLineGroup) + lane * 8;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (c < cols) v = *reinterpret_cast<const uint4*>(x + (size_t)row * cols + c);
        const float2 f0 = __half22float2(u32_as_h2(v.x)), f1 = __half22float2(u32_as_h2(v.y)), f2 = __half22float2(u32_as_h2(v.z)), f3 = __half22float2(u32_as_h2(v.w));
        float sum = ((f0.x + f0.y) + (f1.x + f1.y)) + ((f2.x + f2.y) + (f3.x + f3.y));
#pragma unroll
        for (int o = 1; o < 8; o *= 2) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        sum = __shfl_sync(0xffffffffu, sum, (lane & 3) * 8);
        const float hi = tf32_of(sum);
        if (lane < 8) out[((size_t)row * stages + st) * 8 + lane] = lane < 4 ? hi : tf32_of(sum - hi);
    }
}

template <int MODE, int N>
__global__ void __launch_bounds__(WideCfg<N>::kThreads, 1) affine_wide_kernel(const __grid_constant__ LineMaps maps, const AffineArgs a, const Line line) {
    using C = WideCfg<N>;
    extern __shared__ uint8_t smem_raw[];
    __shared__ WideShared<N> sh;
    const uint32_t raw = kept((smem_u32(smem_raw) + 1023u) & ~1023u), shared = kept(smem_u32(&sh));
    const uint32_t x_tiles = raw + C::kRawStages * kRawBytes, window = x_tiles + C::kXStages * C::kTurn * C::kXBytes;
    const uint32_t scales = shared + (uint32_t)offsetof(WideShared<N>, scales), folded = shared + (uint32_t)offsetof(WideShared<N>, folded), dead = shared + (uint32_t)offsetof(WideShared<N>, dead);
    auto bar = [&](int kind, uint32_t i = 0) { return shared + 8u * (kind + i); };
    const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;

    pdl_trigger();
    if (tid == 0) {
        auto init = [&](int kind, int n, int count) {
            for (int i = 0; i < n; ++i) mbar_init(&sh.bars[kind + i], count);
        };
        init(C::kRawFull, C::kRawStages, 1);
        init(C::kRawEmpty, C::kRawStages, C::kTurn == kStageGroups ? 4 : kExpandWarps);
        init(C::kScaleFull, C::kScaleStages, 32);
        init(C::kScaleEmpty, C::kScaleStages, kEpilogueWarps);
        init(C::kXFull, C::kXStages, 1);
        init(C::kXEmpty, C::kXStages, kSumWarps);
        init(C::kAFull, C::kASlots, 4);
        init(C::kTurnDone, kDone, 1);
        init(C::kAccEmpty, C::kSlots, kEpilogueWarps);
        init(C::kWindowFull, C::kWindows, C::kOwn ? kSumWarps : 1);
        init(C::kWindowEmpty, C::kWindows, 1);
        init(C::kSumFull, C::kFoldedSlots, kSumWarps);
        init(C::kSumEmpty, C::kFoldedSlots, kEpilogueWarps);
        sh.dead = 0u;
        mbar_fence_init();
        fence_async_smem();
    }
    if (tid == 32) {  // where the roles begin: read by each when it does, not held in registers until then
        sh.u0 = line_at(line, blockIdx.x);
        sh.u1 = line_at(line, blockIdx.x + 1);
        sh.first = part_at(line, sh.u0, sh.u1, a.batch);
    }
    if (warp == 2) tmem_alloc(&sh.tmem, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = (uint32_t)uniform((int)sh.tmem), tmem_a = tmem + C::kACol;
    // A turn is up to kTurn groups of a stage, each into an accumulator of its own; unless the epilogue adds the biases, one more after the
    // last group of a window (four stages of a part) multiplies the window's.
    // What comes after this needs the launch in front; true where a guarded launch is not to run.
    auto started = [&] {
        pdl_wait();
        return dyn_skip(a.dyn);
    };
    auto window_ends = [&](const Part& t, int st) { return !C::kFolded && (((st - t.s0) & (kSumWindow - 1)) == kSumWindow - 1 || st + 1 == t.s1); };
    // Weight row (of the tile as the weights arrive) that tensor-memory lane r stands for: gate and up rows of one result 16 lanes apart
    auto tile_row = [](int r) { return MODE == kAffineGateUp ? (r & 16) * 4 + (r >> 5) * 16 + (r & 15) : r; };
    if (warp < kEpilogueWarp) {
    registers_down<C::kFront>();
    if (warp == 0) {
        // ── packed weights, scales and biases ──
        uint32_t requested = 0;
        Ring<C::kRawStages> rs;
        Ring<C::kScaleStages> ss;
        uint32_t stage_scales = 0, stage_full = 0;
        feed_scales<MODE>(a, line, sh.first, sh.u0, sh.u1, lane,
            [&](uint32_t it, const Part& t, int st) {
                if (it == C::kRawStages && started()) return false;
                if (!wait_warp(bar(C::kRawEmpty, rs.i), rs.phase ^ 1u, dead)) return false;
                if (lane == 0) {
                    arrive_expect_at(bar(C::kRawFull, rs.i), kRawBytes);
                    request_weights<MODE>(maps, line, t.row_tile, st, raw + rs.i * kRawBytes, bar(C::kRawFull, rs.i));
                }
                requested = it + 1;
                rs.next();
                if (!wait_warp(bar(C::kScaleEmpty, ss.i), ss.phase ^ 1u, dead)) return false;
                stage_scales = scales + ss.i * (2 * kLineRows * 8) + lane * 8;
                stage_full = bar(C::kScaleFull, ss.i);
                ss.next();
                return true;
            },
            [&](uint32_t, int i, int which) { return stage_scales + which * (kLineRows * 8) + i * 256; }, [&](uint32_t) { return stage_full; });
        if (lane == 0)
#pragma unroll 1
            for (uint32_t i = requested > C::kRawStages ? requested - C::kRawStages : 0; i < requested; ++i) mbar_poll_bounded(&sh.bars[C::kRawFull + i % C::kRawStages], (i / C::kRawStages) & 1);  // no copy may land after the CTA has left
    } else if (warp == 1) {
        // ── activations, and their group sums where they were made in front ──
        if (lane == 0) {
            uint32_t it = 0, windows = 0, turn = 0;
            Ring<C::kXStages> xs;
            Ring<C::kWindows> ws;
            bool alive = !started();
            const uint32_t bytes = (uint32_t)line.tile_cols * kLineGroup * 2;
            const int u1 = sh.u1;
            Part t = sh.first;
#pragma unroll 1
            for (int u = sh.u0; u < u1 && alive; next_part(line, t, u, u1, a.batch)) {
#pragma unroll 1
                for (int st = t.s0; st < t.s1 && alive; ++st) {
                    const int n = stage_groups(line, st);
#pragma unroll 1
                    for (int j = 0; j < n; j += C::kTurn, ++it) {
                        if (it >= C::kXStages) {
                            const uint32_t last = sh.x_turns[xs.i];
                            if (!(alive = wait_one(bar(C::kTurnDone, last % kDone), (last / kDone) & 1, dead) && (!C::kOwn || wait_one(bar(C::kXEmpty, xs.i), xs.phase ^ 1u, dead)))) break;
                        }
                        sh.x_turns[xs.i] = turn++;
                        const int m = min(C::kTurn, n - j);
                        arrive_expect_at(bar(C::kXFull, xs.i), bytes * m);
#pragma unroll 1
                        for (int i = 0; i < m; ++i) tma_load_2d_at(x_tiles + (C::kTurn * xs.i + i) * C::kXBytes, &maps.x, (st * kStageGroups + j + i) * kLineGroup, t.col0, bar(C::kXFull, xs.i));
                        xs.next();
                    }
                    if (alive && window_ends(t, st)) {
                        if (!C::kOwn) {
                            if (!(alive = wait_one(bar(C::kWindowEmpty, ws.i), ws.phase ^ 1u, dead))) break;
                            const int first = st - ((st - t.s0) & (kSumWindow - 1));
                            arrive_expect_at(bar(C::kWindowFull, ws.i), (uint32_t)line.tile_cols * 128);
                            tma_load_2d_at(window + ws.i * C::kWindow, &maps.sums, first * 2 * kStageGroups, t.col0, bar(C::kWindowFull, ws.i));
                            ws.next();
                            ++windows;
                        }
                        ++turn;
                    }
                }
                u += t.s1 - t.s0;
            }
#pragma unroll 1
            for (uint32_t i = it > C::kXStages ? it - C::kXStages : 0; i < it; ++i) mbar_poll_bounded(&sh.bars[C::kXFull + i % C::kXStages], (i / C::kXStages) & 1);
#pragma unroll 1
            for (uint32_t i = windows > C::kWindows ? windows - C::kWindows : 0; i < windows; ++i) mbar_poll_bounded(&sh.bars[C::kWindowFull + i % C::kWindows], (i / C::kWindows) & 1);
        }
    } else {
        // ── issue: two warps, each every second turn; a warp's chain from one turn to the next is longer than the MMAs ──
        const int who = warp - 2;
        const uint32_t shape = (1u << 4) | ((uint32_t)(line.tile_cols >> 3) << 17) | ((uint32_t)(kLineRows >> 4) << 24);  // f32 += f16 x f16, K-major both
        const uint32_t tf32 = shape | (2u << 7) | (2u << 10);
        const uint64_t x_desc = smem_desc_sw128(x_tiles), window_desc = smem_desc_sw128(window);
        Ring<C::kASlots> as;
        Ring<C::kXStages> xs;
        Ring<C::kSlots> slot;
        Ring<kDone> end;
        Ring<C::kWindows> ws;
        slot.next(who);
        end.next(who);
        uint32_t turn = 0, units = 0, last = 0, last_window = 2;
        bool alive = !started();
        auto ready = [&](uint32_t b_full, uint32_t b_phase) {
            const bool ok = wait_warp(b_full, b_phase, dead) && wait_warp(bar(C::kAFull, as.i), as.phase, dead) && wait_warp(bar(C::kAccEmpty, slot.i), slot.phase ^ 1u, dead);
            tc_fence_after();
            return ok;
        };
        auto issued = [&] {
            commit_elected(bar(C::kTurnDone, end.i));
            last = end.i | end.phase << 16;
            slot.next(2);
            end.next(2);
            ++units;
        };
        const int u1 = uniform(sh.u1);
        Part t = uniform(sh.first);
#pragma unroll 1
        for (int u = uniform(sh.u0); u < u1 && alive; next_part(line, t, u, u1, a.batch)) {
#pragma unroll 1
            for (int st = t.s0; st < t.s1 && alive; ++st) {
                const int n = stage_groups(line, st);
#pragma unroll 1
                for (int k = 0; k < n; k += C::kTurn, ++turn, as.next(), xs.next()) {
                    if ((int)(turn & 1) != who) continue;
                    if (!(alive = ready(bar(C::kXFull, xs.i), xs.phase))) break;
                    uint32_t d = tmem + slot.i * 128, at = tmem_a + as.i * (C::kTurn * 32);
                    uint64_t b = x_desc + xs.i * (C::kTurn * C::kXBytes / 16);
#pragma unroll 1
                    for (int i = min(C::kTurn, n - k); i > 0; --i, d += N, at += 32, b += C::kXBytes / 16) umma_f16_group(d, at, b, shape);
                    issued();
                }
                if (alive && window_ends(t, st)) {
                    if ((int)(turn & 1) == who) {
                        if (!(alive = ready(bar(C::kWindowFull, ws.i), ws.phase))) break;
                        const int steps = ((st - t.s0) & (kSumWindow - 1)) + 1;
#pragma unroll 1
                        for (int i = 0; i < steps; ++i) umma_tf32_step(tmem + slot.i * 128, tmem_a + as.i * (C::kTurn * 32) + 8 * i, window_desc + ws.i * (C::kWindow / 16) + 2 * i, tf32, i > 0);
                        commit_elected(bar(C::kWindowEmpty, ws.i));
                        issued();
                    }
                    last_window = ws.i | ws.phase << 16;  // whichever warp issued it: a barrier's parity tells only its latest phase
                    ++turn;
                    as.next();
                    ws.next();
                }
            }
            u += t.s1 - t.s0;
        }
        // the MMAs in flight read shared memory and write tensor memory
        if (units > 0) mbar_poll_bounded(&sh.bars[C::kTurnDone + (last & 0xffff)], last >> 16);
        if (last_window != 2) mbar_poll_bounded(&sh.bars[C::kWindowEmpty + (last_window & 0xffff)], last_window >> 16);
    }
    } else if (warp < kExpandWarp) {
        registers_up<C::kDrain>();
        // ── sums and epilogue: two sets of four warps, each half of the tile's columns; a turn is 64 values of a thread, fetched at once ──
        const int set = (warp - kEpilogueWarp) >> 2, quad = warp & 3, r = quad * 32 + lane, row = tile_row(r);
        const int eights = line.tile_cols / 16, from = set * eights * 8;  // of a set
        const uint32_t lane_base = tmem + ((uint32_t)(quad * 32) << 16) + from;
        const bool leader = tid == kEpilogueWarp * 32;
        auto all_sync = [] { asm volatile("bar.sync 1, %0;" ::"n"(kEpilogueThreads) : "memory"); };
        Ring<C::kScaleStages> ss;
        Ring<C::kSlots> slot;
        Ring<kDone> end;
        Ring<C::kFoldedSlots> sum;
        const int u1 = started() ? sh.u0 : sh.u1;
        Part t = sh.first;
#pragma unroll 1
        for (int u = sh.u0; u < u1; next_part(line, t, u, u1, a.batch)) {
            constexpr int kSums = N / 2, kChunks = kSums / 16;  // chunks of sixteen columns of a group
            float sums[kSums];
#pragma unroll
            for (int j = 0; j < kSums; ++j) sums[j] = 0.f;
            bool alive = true;
            uint32_t held = 0;  // stages whose scales this window has used
#pragma unroll 1
            for (int st = t.s0; st < t.s1 && alive; ++st) {
                if (!(alive = wait_warp(bar(C::kScaleFull, ss.i), ss.phase, dead))) break;
                const uint32_t row_scales = scales + ss.i * (2 * kLineRows * 8) + row * 8;
                const int n = stage_groups(line, st), groups = C::kTurn == kStageGroups ? 1 : (n + C::kTurn - 1) / C::kTurn, all = groups + window_ends(t, st);
                uint2 sv = lds64(row_scales), bv = C::kFolded ? lds64(row_scales + kLineRows * 8) : make_uint2(0, 0);
#pragma unroll 1
                for (int k = 0; k < all; ++k) {
                    float s1[C::kTurn], b1[C::kTurn];
#pragma unroll
                    for (int i = 0; i < C::kTurn; ++i) {
                        const float si = __low2float(u32_as_h2(sv.x));
                        s1[i] = C::kFolded || k < groups ? si * kNibble : 1.f;
                        b1[i] = C::kFolded ? fmaf(8.f, si, __low2float(u32_as_h2(bv.x))) : 0.f;  // the nibbles are centred
                        sv = make_uint2(__funnelshift_r(sv.x, sv.y, 16), sv.y >> 16);
                        bv = make_uint2(__funnelshift_r(bv.x, bv.y, 16), bv.y >> 16);
                    }
                    const int m = k < groups ? min(C::kTurn, n - k * C::kTurn) : 1;
                    if (!(alive = wait_warp(bar(C::kTurnDone, end.i), end.phase, dead) && (!C::kFolded || wait_warp(bar(C::kSumFull, sum.i), sum.phase, dead)))) break;
                    tc_fence_after();
                    uint32_t v[4][16];
#pragma unroll
                    for (int q = 0; q < 4; ++q) tmem_ld16(lane_base + slot.i * 128 + q / kChunks * N + q % kChunks * 16, v[q]);
                    float part[C::kFolded ? 16 : 1];  // of this turn: the running sums, much larger, round once a turn and not twice a group
                    const uint32_t x_sums = folded + sum.i * (C::kTurn * N * 4) + from * 4;
                    auto add_biases = [&](int q) {
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const uint4 xs = lds128(x_sums + q * (N * 4) + 16 * j);
                            float* to = part + 4 * j;
                            to[0] = q == 0 ? __uint_as_float(xs.x) * b1[0] : fmaf(__uint_as_float(xs.x), b1[q], to[0]);
                            to[1] = q == 0 ? __uint_as_float(xs.y) * b1[0] : fmaf(__uint_as_float(xs.y), b1[q], to[1]);
                            to[2] = q == 0 ? __uint_as_float(xs.z) * b1[0] : fmaf(__uint_as_float(xs.z), b1[q], to[2]);
                            to[3] = q == 0 ? __uint_as_float(xs.w) * b1[0] : fmaf(__uint_as_float(xs.w), b1[q], to[3]);
                        }
                    };
                    if constexpr (C::kFolded) add_biases(0);  // while the accumulators are on their way: two groups ahead are slower, four spill
#pragma unroll
                    for (int q = 0; q < 4; ++q) tmem_wait_ld16(v[q]);
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) arrive_at(bar(C::kAccEmpty, slot.i));
                    slot.next();
                    end.next();
                    if constexpr (C::kFolded) {
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            if (q < m) {
#pragma unroll
                                for (int j = 0; j < 16; ++j) part[j] = fmaf(__uint_as_float(v[q][j]), s1[q], part[j]);
                            }
#pragma unroll
                        for (int q = 1; q < 4; ++q)
                            if (q < m) add_biases(q);
                        __syncwarp();
                        if (lane == 0) arrive_at(bar(C::kSumEmpty, sum.i));
                        sum.next();
#pragma unroll
                        for (int j = 0; j < 16; ++j) sums[j] += part[j];
                    } else {
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            if (q / kChunks < m) {
#pragma unroll
                                for (int j = 0; j < 16; ++j) sums[q % kChunks * 16 + j] = fmaf(__uint_as_float(v[q][j]), s1[q / kChunks], sums[q % kChunks * 16 + j]);
                            }
                    }
                }
                if (!alive) break;
                if (C::kFolded) {
                    if (lane == 0) arrive_at(bar(C::kScaleEmpty, ss.i));
                } else {
                    ++held;
                    if (window_ends(t, st)) {  // the expansion has read the biases of the window's stages too
                        if (lane == 0)
#pragma unroll 1
                            for (uint32_t i = 0; i < held; ++i) arrive_at(bar(C::kScaleEmpty, ss.i >= i ? ss.i - i : ss.i + C::kScaleStages - i));
                        held = 0;
                    }
                }
                ss.next();
            }
            all_sync();  // the eight warps go on together or not at all: one that gave up has set the word
            if (leader) sh.go = lds_word(dead) == 0u ? 1u : 0u;
            all_sync();
            if (sh.go == 0u) break;
            // The end of a tile.  A CTA that shares it leaves its sums in scratch; the last to arrive adds them in the order of the CTAs.
            const size_t part = (size_t)line.tile_cols * kLineRows;
            constexpr int kEights = N / 16;
            auto column = [&](int i) { return from + 8 * i; };
            const bool together = t.s0 != 0 || t.s1 != line.stages;
            Sharers sharing = {(int)blockIdx.x, (int)blockIdx.x, 2 * (int)blockIdx.x + 1};
            if (together) sharing = sharers(line, t.tile);
            float4* const mine = reinterpret_cast<float4*>(a.part_scratch + (size_t)sharing.slot(blockIdx.x) * part) + r;  // [four columns][row]
            bool finish = true, left = false;  // left: this CTA's sums are in scratch
            if (together) {
                if (leader) sh.ticket = *(volatile int*)(a.part_counters + t.tile) == sharing.last - sharing.first ? 1u : 0u;
                all_sync();
                left = sh.ticket == 0u;  // else all others have arrived: this one is the last, and its sums need not go through scratch
                if (left) {
#pragma unroll
                    for (int i = 0; i < kEights; ++i)
                        if (i < eights) {
                            __stcg(mine + column(i) / 4 * kLineRows, make_float4(sums[8 * i], sums[8 * i + 1], sums[8 * i + 2], sums[8 * i + 3]));
                            __stcg(mine + (column(i) / 4 + 1) * kLineRows, make_float4(sums[8 * i + 4], sums[8 * i + 5], sums[8 * i + 6], sums[8 * i + 7]));
                        }
                    __threadfence();
                }
                all_sync();
                if (leader) sh.ticket = (uint32_t)atomicAdd(a.part_counters + t.tile, 1);
                all_sync();
                finish = sh.ticket == (uint32_t)(sharing.last - sharing.first);
                if (finish) {
                    __threadfence();
                    if (leader) a.part_counters[t.tile] = 0;  // the next launch finds every counter at zero
                }
            }
            if (finish) {
                const LineRow o = line_row<MODE>(a, line, t.row_tile, row);
                const bool row_ok = o.row < o.rows;
                auto write = [&](int c, float (&v)[8]) {  // eight columns of the tile from c on
                    const int n = t.live - c;
                    if (MODE == kAffineGateUp) {
                        // lanes 16 apart have gate and up of one row of the result: the gate's takes the first four columns, the up's the others
                        const bool up = r & 16;
                        __half* y = o.y + (size_t)(t.col0 + c + (up ? 4 : 0)) * o.rows + o.row;
#pragma unroll
                        for (int j = 0; j < 4; ++j, y += o.rows) {
                            const float other = __shfl_xor_sync(0xffffffffu, up ? v[j] : v[4 + j], 16);
                            const __half z = swiglu_f32(up ? other : v[j], up ? v[4 + j] : other);  // lut_matvec.metal:2228
                            if (row_ok && j + (up ? 4 : 0) < n) *y = z;
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
                // A step: eight columns of some CTAs' sums; the next step's are on their way while these are added.  A short loop that picks its
                // own sums from the registers by a jump: unrolled, the code would come from beyond the instruction cache.
                constexpr int kAtOnce = 2;
                const int rounds = (sharing.last - sharing.first + kAtOnce) / kAtOnce, steps = eights * rounds;
                float4 f[kAtOnce][2];
                auto request = [&](int i, int c) {
#pragma unroll
                    for (int z = 0; z < kAtOnce; ++z) {
                        const float4* q = reinterpret_cast<const float4*>(a.part_scratch + (size_t)sharing.slot(min(c + z, sharing.last)) * part) + column(i) / 4 * kLineRows + r;
                        const bool there = c + z <= sharing.last && c + z != (int)blockIdx.x;
#pragma unroll
                        for (int j = 0; j < 2; ++j) f[z][j] = there ? __ldcg(q + j * kLineRows) : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
                };
                float v[8];
                request(0, sharing.first);
#pragma unroll 1
                for (int i = 0, c = sharing.first, left_steps = steps; left_steps > 0; --left_steps) {
                    if (c == sharing.first)
#pragma unroll
                        for (int j = 0; j < 8; ++j) v[j] = 0.f;
                    const int me = (int)blockIdx.x - c;
                    if (me >= 0 && me < kAtOnce) {
                        float own_v[8];
                        switch (i) {
#define PICK(n)                                                    \
    case n:                                                        \
        if constexpr (n < kEights)                                 \
            for (int j = 0; j < 8; ++j) own_v[j] = sums[8 * n + j];      \
        break;
                            PICK(0) PICK(1) PICK(2) PICK(3) PICK(4) PICK(5) PICK(6) PICK(7)
#undef PICK
                        }
#pragma unroll
                        for (int z = 0; z < kAtOnce; ++z)
                            if (z == me) { f[z][0] = make_float4(own_v[0], own_v[1], own_v[2], own_v[3]); f[z][1] = make_float4(own_v[4], own_v[5], own_v[6], own_v[7]); }
                    }
#pragma unroll
                    for (int z = 0; z < kAtOnce; ++z)
#pragma unroll
                        for (int j = 0; j < 2; ++j) { v[4 * j] += f[z][j].x; v[4 * j + 1] += f[z][j].y; v[4 * j + 2] += f[z][j].z; v[4 * j + 3] += f[z][j].w; }
                    const int col = column(i);
                    const bool summed = c + kAtOnce > sharing.last;
                    if (summed) { ++i; c = sharing.first; } else c += kAtOnce;
                    if (left_steps > 1) request(i, c);
                    if (summed && col < t.live) write(col, v);
                }
            }
            __syncwarp();  // the next tensor-memory load needs the whole warp
            u += t.s1 - t.s0;
        }
    } else if (warp < kSumWarp) {
        registers_down<C::kBehind>();
        // ── expansion: sets of four warps take turns ──
        const int set = (warp - kExpandWarp) >> 2, quad = warp & 3, r = quad * 32 + lane, row = tile_row(r);
        const uint32_t dst = tmem_a + ((uint32_t)(quad * 32) << 16);
        uint32_t turn = 0;
        Ring<C::kRawStages> rs;
        Ring<C::kScaleStages> ss;
        Ring<C::kASlots> as;
        bool alive = true;
        auto slot_free = [&] {
            if (turn >= C::kASlots && turn < C::kASlots + 2 && started()) return false;
            if (turn >= C::kASlots) {
                const uint32_t last = turn - C::kASlots;
                if (!wait_warp(bar(C::kTurnDone, last % kDone), (last / kDone) & 1, dead)) return false;
            }
            tc_fence_after();
            return true;
        };
        auto written = [&] {
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) arrive_at(bar(C::kAFull, as.i));
        };
        const int u1 = sh.u1;
        Part t = sh.first;
#pragma unroll 1
        for (int u = sh.u0; u < u1 && alive; next_part(line, t, u, u1, a.batch)) {
#pragma unroll 1
            for (int st = t.s0; st < t.s1 && alive; ++st) {
                const int n = stage_groups(line, st);
                const bool mine = C::kTurn < kStageGroups || (int)(turn & 1) == set;
                if (mine && !(alive = wait_warp(bar(C::kRawFull, rs.i), rs.phase, dead) && (C::kFolded || wait_warp(bar(C::kScaleFull, ss.i), ss.phase, dead)))) break;
                const uint32_t src = raw + rs.i * kRawBytes + row * 128, row_scales = scales + ss.i * (2 * kLineRows * 8) + row * 8;
#pragma unroll 1
                for (int k = 0; k < n; k += C::kTurn, ++turn, as.next()) {
                    if ((int)(turn & 1) != set) continue;
                    uint2 sv = make_uint2(0, 0), bv = make_uint2(0, 0);
                    if (C::kFolded) {
                    } else if (C::kTurn == 1) {
                        sv = make_uint2(lds_u16(row_scales + 2 * k), 0u);
                        bv = make_uint2(lds_u16(row_scales + kLineRows * 8 + 2 * k), 0u);
                    } else {
                        sv = lds64(row_scales);
                        bv = lds64(row_scales + kLineRows * 8);
                        if (k > 0) { sv.x = sv.y; bv.x = bv.y; }
                    }
                    if (!(alive = slot_free())) break;
                    const uint32_t to = dst + as.i * (C::kTurn * 32);
                    const int halves = 2 * min(C::kTurn, n - k);
#pragma unroll 1
                    for (int i = 0; i < halves; i += 2) {  // a group
                        uint32_t minus = 0xA400A400u;  // -8 x 2^-9: in fp32 every bias is exact enough
                        if (!C::kFolded) tf32_bias(__low2float(u32_as_h2(sv.x)), __low2float(u32_as_h2(bv.x)), &minus);
                        sv = make_uint2(__funnelshift_r(sv.x, sv.y, 16), sv.y >> 16);
                        bv = make_uint2(__funnelshift_r(bv.x, bv.y, 16), bv.y >> 16);
                        const uint4 v0 = lds128(src + (((2 * k + i) ^ (row & 7)) << 4)), v1 = lds128(src + (((2 * k + i + 1) ^ (row & 7)) << 4));
                        uint32_t pair[16], more[16];
                        expand_nibbles(v0.x, minus, pair);
                        expand_nibbles(v0.y, minus, pair + 4);
                        expand_nibbles(v0.z, minus, pair + 8);
                        expand_nibbles(v0.w, minus, pair + 12);
                        expand_nibbles(v1.x, minus, more);
                        expand_nibbles(v1.y, minus, more + 4);
                        expand_nibbles(v1.z, minus, more + 8);
                        expand_nibbles(v1.w, minus, more + 12);
                        tmem_st16(to + i * 16, pair);
                        tmem_st16(to + i * 16 + 16, more);
                    }
                    written();
                }
                if (!alive) break;
                if (mine) {
                    __syncwarp();
                    if (lane == 0) arrive_at(bar(C::kRawEmpty, rs.i));
                }
                if (window_ends(t, st)) {  // biases, twice each: they meet hi and lo of the group sums
                    if ((int)(turn & 1) == set) {
                        if (!(alive = slot_free())) break;
                        const uint32_t last = (st - t.s0) & (kSumWindow - 1);
#pragma unroll 1
                        for (uint32_t i = 0; i <= last; ++i) {
                            const uint32_t back = last - i, stage = ss.i >= back ? ss.i - back : ss.i + C::kScaleStages - back, at = scales + stage * (2 * kLineRows * 8) + row * 8;
                            uint32_t v[8];
                            uint32_t minus;
                            uint2 sv = lds64(at), bv = lds64(at + kLineRows * 8);
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                v[j] = v[4 + j] = __float_as_uint(tf32_bias(__low2float(u32_as_h2(sv.x)), __low2float(u32_as_h2(bv.x)), &minus));
                                sv = make_uint2(__funnelshift_r(sv.x, sv.y, 16), sv.y >> 16);
                                bv = make_uint2(__funnelshift_r(bv.x, bv.y, 16), bv.y >> 16);
                            }
                            tmem_st8(dst + as.i * (C::kTurn * 32) + 8 * i, v);
                        }
                        written();
                    }
                    ++turn;
                    as.next();
                }
                rs.next();
                ss.next();
            }
            u += t.s1 - t.s0;
        }
    } else if constexpr (C::kOwn) {
        registers_down<C::kBehind>();
        // ── group sums of x: a thread sums the 64 columns of one row ──
        constexpr int kRowWarps = kSumWarps / C::kTurn;  // warps that share a group's rows
        const int i = (warp - kSumWarp) / kRowWarps, col = (warp - kSumWarp) % kRowWarps * 32 + lane;
        Ring<C::kXStages> xs;
        Ring<C::kWindows> ws;
        Ring<C::kFoldedSlots> slot;
        bool alive = !started();
        const int u1 = sh.u1;
        Part t = sh.first;
#pragma unroll 1
        for (int u = sh.u0; u < u1 && alive; next_part(line, t, u, u1, a.batch)) {
#pragma unroll 1
            for (int st = t.s0; st < t.s1 && alive; ++st) {
                const int n = stage_groups(line, st), at = (st - t.s0) & (kSumWindow - 1);
                if (!C::kFolded && at == 0 && !(alive = wait_warp(bar(C::kWindowEmpty, ws.i), ws.phase ^ 1u, dead))) break;
                // where this row's sums of the stage lie: hi of four groups and lo of four, 16 bytes each, swizzled as the MMA reads them
                const uint32_t row_at = window + ws.i * C::kWindow + col * 128, hi_at = row_at + ((2 * at ^ (col & 7)) << 4), lo_at = row_at + (((2 * at + 1) ^ (col & 7)) << 4);
#pragma unroll 1
                for (int k = 0; k < n; k += C::kTurn) {
                    if (!(alive = wait_warp(bar(C::kXFull, xs.i), xs.phase, dead))) break;
                    float total = 0.f;
                    if (k + i < n && col < line.tile_cols) {
                        uint64_t sum[4] = {0, 0, 0, 0};
                        const uint32_t src = x_tiles + (C::kTurn * xs.i + i) * C::kXBytes + col * 128;
#pragma unroll 2
                        for (int c = 0; c < 8; ++c) {
                            const uint4 v = lds128(src + ((c ^ (col & 7)) << 4));
                            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                const float2 f = __half22float2(u32_as_h2(w[j]));
                                sum[j] = add2(sum[j], pack2(f.x, f.y));
                            }
                        }
                        const float2 f = unpack2(add2(add2(sum[0], sum[1]), add2(sum[2], sum[3])));
                        total = f.x + f.y;
                    }
                    __syncwarp();
                    if (lane == 0) arrive_at(bar(C::kXEmpty, xs.i));
                    if (C::kFolded) {
                        if (!(alive = wait_warp(bar(C::kSumEmpty, slot.i), slot.phase ^ 1u, dead))) break;
                        sts_word(folded + slot.i * (C::kTurn * N * 4) + (i * N + col) * 4, total);
                        __syncwarp();
                        if (lane == 0) arrive_at(bar(C::kSumFull, slot.i));
                        slot.next();
                        xs.next();
                        continue;
                    }
                    const float hi = tf32_of(total), lo = tf32_of(total - hi);
                    sts_word(hi_at + 4 * (k + i), hi);
                    sts_word(lo_at + 4 * (k + i), lo);
                    if (C::kTurn < kStageGroups && n <= C::kTurn) {  // the groups of a short stage that no turn has
                        sts_word(hi_at + 4 * (C::kTurn + i), 0.f);
                        sts_word(lo_at + 4 * (C::kTurn + i), 0.f);
                    }
                    xs.next();
                }
                if (alive && window_ends(t, st)) {
                    fence_async_smem();
                    __syncwarp();
                    if (lane == 0) arrive_at(bar(C::kWindowFull, ws.i));
                    ws.next();
                }
            }
            u += t.s1 - t.s0;
        }
    }
    __syncthreads();
    if (tid == 0 && a.err && lds_word(dead) == 1u) atomicOr(a.err, 0x400u);
    tc_fence_before();
    __syncthreads();
    if (warp == 2) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

template <typename... Params, typename... Args>
cudaError_t launch_pdl(const Launch& l, void (*kern)(Params...), dim3 grid, int threads, uint32_t smem, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = l.stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = l.pdl ? 1 : 0;
    prefer_max_shared(kern);
    l.count();
    return cudaLaunchKernelEx(&cfg, kern, args...);
}

template <int MODE, int N>
cudaError_t launch_wide_t(const Launch& l, AffineArgs a, const LineMaps& maps, const Line& line, int grid) {
    auto kern = affine_wide_kernel<MODE, N>;
    cudaError_t e = allow_shared(kern, WideCfg<N>::kSmem);
    if (e != cudaSuccess) return e;
    a.dyn = dev_dyn(l);
    return launch_pdl(l, kern, dim3(grid), WideCfg<N>::kThreads, WideCfg<N>::kSmem, maps, a, line);
}

template <int MODE>
cudaError_t launch_wide(const Launch& l, const AffineArgs& a, const LineMaps& maps, const Line& line, int grid) {
    if (line.tile_cols <= 32) return launch_wide_t<MODE, 32>(l, a, maps, line, grid);
    if (line.tile_cols <= 64) return launch_wide_t<MODE, 64>(l, a, maps, line, grid);
    return launch_wide_t<MODE, 128>(l, a, maps, line, grid);
}

}  // namespace

cudaError_t launch_affine_wide(const Launch& l, int mode, const AffineArgs& a, int group, bool* handled) {
    // Rows of x whose group sums find room behind the shared tiles of the full scratch (40 MiB: 10,000 of 17,408 columns); more go in parts.
    const int sm = a.sm_count > 0 ? a.sm_count : 148, stages = (a.cols / kLineGroup + kStageGroups - 1) / kStageGroups;
    const size_t tiles = (size_t)sm * 2 * 128 * kLineRows * sizeof(float);
    if (a.batch > 128 && a.part_scratch_bytes > tiles) {
        const size_t rows = (a.part_scratch_bytes - tiles) / ((size_t)stages * 2 * kStageGroups * sizeof(float)) / 128 * 128;
        if (rows >= 128 && rows < (size_t)a.batch) {
            *handled = false;
            for (int r0 = 0; r0 < a.batch; r0 += (int)rows) {
                const cudaError_t e = launch_affine_wide(l, mode, affine_rows(a, r0, std::min((int)rows, a.batch - r0)), group, handled);
                if (e != cudaSuccess || !*handled) return e;
            }
            return cudaSuccess;
        }
    }
    LineMaps maps = {};
    Line line;
    GroupSums sums;
    int grid = 0;
    *handled = line_plan(mode, a, group, 128, kOwnCols, &maps, &line, &sums, &grid);
    if (!*handled) return cudaSuccess;
    if (sums.at) {
        const cudaError_t e = launch_pdl(l, group_sums_kernel, dim3(a.batch, std::min((line.stages + 7) / 8, 65535)), 256, 0, a.x, sums.at, a.batch, a.cols, line.stages);
        if (e != cudaSuccess) return e;
    }
    switch (mode) {
        case kAffinePlain: return launch_wide<kAffinePlain>(l, a, maps, line, grid);
        case kAffineAdd: return launch_wide<kAffineAdd>(l, a, maps, line, grid);
        case kAffineGateUp: return launch_wide<kAffineGateUp>(l, a, maps, line, grid);
        case kAffineDual: return launch_wide<kAffineDual>(l, a, maps, line, grid);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace smelt
