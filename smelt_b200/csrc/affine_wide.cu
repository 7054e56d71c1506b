// Quantised matrix product for many rows of x (prompt chunks, decode of many sequences):
// Y[M, R] = X[M, K] . W[R, K]^T with W affine u4, group 64, on the fifth-generation tensor cores.
//
// Replaces agent_affine_qmm_fixed_batched_full and its fused gate/up form (Resources/Shaders/agent_affine_qmm.h:107-316,
// :360-742; wrappers Resources/Shaders/lut_matvec.metal:6519-6545, :6615-6635).  The tensor core multiplies the
// dequantised weight w = scale * q + bias, evaluated in fp32 with one FMA, as TWO fp16 operands: hi = half(w) and
// lo = half(w - hi).  hi + lo carries 22 significant bits of w, so D += hi . x + lo . x in the fp32 accumulator is within
// 2^-22 of the factored form of the matvec family, and a tile's sums stay in tensor memory over all of K.
//
// Mapping.  One CTA an SM takes an equal stretch of the launch's line of work (affine_line.cuh); a tile is 128 weight
// rows, the MMA's M, by up to 256 rows of x, its N.  The roles, each on warps of its own, each a ring ahead of the next:
//   * weights: TMA, 128 rows x 256 columns of packed nibbles a stage, requested before the wait for the launch in front;
//   * activations: TMA, one 64-column group a stage, 128-byte swizzled: the MMA's B operand as it is;
//   * scales and biases, one warp;
//   * expansion: a thread owns a weight row and turns its 64 nibbles of a group into hi and lo, in pairs, straight into
//     tensor memory, from where the MMA takes its A operand.  (An A tile in shared memory is written once and read once per
//     256 rows of x, which with the B tile's two reads and its write is more than the SM's 128 bytes a clock.)
//   * issue: eight K = 16 MMAs a group, two groups a turn;
//   * epilogue: plain, + residual, SwiGLU of the gate | up halves, dual.
// What bounds it: with 256 rows of x a tile the tensor pipe (138 clocks an MMA measured alone, 2,260 of 2,208 for a turn of
// sixteen), which does the work twice; with 128 and fewer the expansion, about 370 instructions per row and group.  Measured
// against the form that expanded through shared memory and drained or staged by the same threads (us; gate/up 12288 x 4096
// x 2 | 4096 x 12288 + residual | 4096 x 4096): 32 rows 77.8 -> 52.2 | 47.6 -> 29.7 | 17.1 -> 14.7; 77 rows 185 -> 51.5 |
// 90.0 -> 35.5; 512 rows 347 -> 169 (609 TFLOP/s of weights times rows, twice that in the pipe) | 259 -> 100 | 79.7 -> 50.1.
// Every wait is bounded: on expiry the CTA sets bit 10 of the error word, its roles stop, copies and MMAs in flight are
// waited for (bounded too) and the tensor memory is freed.
#include "affine_line.cuh"

namespace smelt {

namespace {

constexpr int kThreads = 512, kEpilogueWarp = 4, kExpandWarp = 8, kExpandWarps = 8;
constexpr int kASlots = 2;  // hi | lo of two groups: 128 columns of tensor memory each

template <int N>
struct WideCfg {
    // Accumulators in tensor memory.  The tensor core truncates every sum it adds to, which over 512 additions (K = 4096, hi and
    // lo) is the largest error there is; up to 64 rows, which were summed group by group in registers before, hi and lo have
    // an accumulator each, and the large sums half the additions (relative error against float64, gate/up 12288 x 4096 at 32
    // rows: 2.0709e-4 in registers, 2.0751e-4 together, 2.0723e-4 apart; 2.07e-4 is the rounding of the result).
    static constexpr bool kApart = N == 64;
    static constexpr int kAccCols = kApart ? 2 * N : N, kAcc = 256 / kAccCols;
    static constexpr int kXBytes = N * kLineGroup * 2, kXStages = N == 256 ? 4 : 8, kRawStages = N == 64 ? 6 : 4;
    static constexpr uint32_t kSmem = kRawStages * kRawBytes + kXStages * kXBytes + 1024;
    static_assert(kSmem + 18 * 1024 <= 227u * 1024u, "shared memory");
};

// D[128 x N] (+)= A[128 x 16] . B[N x 16]^T, A from tensor memory (lane = row, two fp16 a column).
__device__ __forceinline__ void umma_f16_ta(uint32_t d, uint32_t a, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}"
        ::"r"(d), "r"(a), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(0u)
        : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t t, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(t), "r"(v[0]), "r"(v[1]), "r"(v[2]),
                 "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
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

// Sixteen sums of a row; those of the lo operand, if apart, LO columns further.
template <int LO>
__device__ __forceinline__ void fetch16(uint32_t src, float (&v)[16]) {
    uint32_t w[2][8], z[2][8];
    tmem_ld8(src, w[0]);
    tmem_ld8(src + 8, w[1]);
    if (LO) {
        tmem_ld8(src + LO, z[0]);
        tmem_ld8(src + LO + 8, z[1]);
    }
    tmem_wait_ld();
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = LO ? __uint_as_float(w[j / 8][j % 8]) + __uint_as_float(z[j / 8][j % 8]) : __uint_as_float(w[j / 8][j % 8]);
}

// silu(gate) * up in fp32; the quotient within two units in the last place, far below the fp16 result's
__device__ __forceinline__ __half swiglu_f32(float gate, float up) { return __float2half_rn(__fdividef(gate, 1.0f + expf(-gate)) * up); }

template <int MODE, int N>
__global__ void __launch_bounds__(kThreads, 1) affine_wide_kernel(const __grid_constant__ LineMaps maps, const AffineArgs a, const Line line) {
    using C = WideCfg<N>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* raw = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* x_tiles = raw + C::kRawStages * kRawBytes;
    __shared__ uint64_t raw_full[C::kRawStages], raw_empty[C::kRawStages], scale_full[C::kRawStages], x_full[C::kXStages], x_empty[C::kXStages], a_full[kASlots], a_empty[kASlots], acc_full[C::kAcc],
        acc_empty[C::kAcc];
    __shared__ uint32_t scales[C::kRawStages][kStageGroups][kLineRows];  // {scale, bias}
    __shared__ float exchange[MODE == kAffineGateUp ? 2 * kLineRows * 8 : 1];
    __shared__ uint32_t s_tmem, s_dead, s_ticket, s_go;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    pdl_trigger();
    if (tid == 0) {
        for (int i = 0; i < C::kRawStages; ++i) { mbar_init(&raw_full[i], 1); mbar_init(&raw_empty[i], kExpandWarps); mbar_init(&scale_full[i], 1); }
        for (int i = 0; i < C::kXStages; ++i) { mbar_init(&x_full[i], 1); mbar_init(&x_empty[i], 1); }
        for (int i = 0; i < kASlots; ++i) { mbar_init(&a_full[i], 4); mbar_init(&a_empty[i], 1); }
        for (int i = 0; i < C::kAcc; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 4); }
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

    if (warp == 0) {
        // ── packed weights ──
        if (lane == 0) {
            uint32_t it = 0;
            bool alive = true;
            for (int u = u0; u < u1 && alive;) {
                const Part t = part_at(line, u, u1, a.batch);
                for (int g = t.g0; g < t.g1; g += kStageGroups, ++it) {
                    const uint32_t s = it % C::kRawStages, use = it / C::kRawStages;
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
                for (int g = t.g0; g < t.g1; ++g, ++it) {
                    const uint32_t s = it % C::kXStages, use = it / C::kXStages;
                    if (use > 0 && !(alive = wait_alive(&x_empty[s], (use - 1) & 1, dead))) break;
                    mbar_arrive_expect_tx(&x_full[s], bytes);
                    tma_2d(x_tiles + s * C::kXBytes, &maps.x, g * kLineGroup, t.col0, &x_full[s]);
                }
                u += t.g1 - t.g0;
            }
            for (uint32_t i = it > C::kXStages ? it - C::kXStages : 0; i < it; ++i) mbar_poll_bounded(&x_full[i % C::kXStages], (i / C::kXStages) & 1);
        }
    } else if (warp == 2) {
        // ── issue ──
        const uint32_t idesc = (1u << 4) | ((uint32_t)(line.tile_cols >> 3) << 17) | ((uint32_t)(kLineRows >> 4) << 24);  // f32 += f16 x f16, K-major both
        uint32_t it = 0, pair = 0, done = 0;
        bool alive = true;
        for (int u = u0; u < u1 && alive; ++done) {
            const Part t = part_at(line, u, u1, a.batch);
            const uint32_t ds = done % C::kAcc, d = tmem + ds * C::kAccCols, d_lo = C::kApart ? d + N : d;
            if (done >= C::kAcc && !(alive = wait_warp(&acc_empty[ds], (done / C::kAcc - 1) & 1, dead))) break;
            tc_fence_after();
            for (int g = t.g0; g < t.g1; g += 2, ++pair) {  // two groups a turn: the waits of a turn take about as long as half a group's MMAs
                const uint32_t as = pair % kASlots, n = min(2, t.g1 - g), pa = (pair / kASlots) & 1;
                const uint32_t x0 = it % C::kXStages, x1 = (it + n - 1) % C::kXStages, p0 = (it / C::kXStages) & 1, p1 = ((it + n - 1) / C::kXStages) & 1;
                const bool b0 = peek(&x_full[x0], p0), b1 = peek(&x_full[x1], p1), b2 = peek(&a_full[as], pa);
                if (!__all_sync(0xffffffffu, b0)) alive = wait_warp(&x_full[x0], p0, dead);
                if (alive && !__all_sync(0xffffffffu, b1)) alive = wait_warp(&x_full[x1], p1, dead);
                if (alive && !__all_sync(0xffffffffu, b2)) alive = wait_warp(&a_full[as], pa, dead);
                if (!alive) break;
                tc_fence_after();
                if (elect_one()) {
                    for (uint32_t i = 0; i < n; ++i) {
                        const uint64_t b = smem_desc_sw128(smem_u32(x_tiles + (i ? x1 : x0) * C::kXBytes));
                        const uint32_t w = tmem_a + as * 128 + i * 64;
#pragma unroll
                        for (int k = 0; k < kLineGroup / 16; ++k) {  // 32 bytes further in the descriptor's address field
                            umma_f16_ta(d, w + k * 8, b + k * 2, idesc, (g != t.g0 || i != 0 || k != 0) ? 1u : 0u);
                            umma_f16_ta(d_lo, w + 32 + k * 8, b + k * 2, idesc, (!C::kApart || g != t.g0 || i != 0 || k != 0) ? 1u : 0u);
                        }
                        umma_commit(&x_empty[i ? x1 : x0]);
                    }
                    umma_commit(&a_empty[as]);
                    if (g + (int)n == t.g1) umma_commit(&acc_full[ds]);
                }
                __syncwarp();
                it += n;
            }
            u += t.g1 - t.g0;
        }
        if (pair > 0) mbar_poll_bounded(&a_empty[(pair - 1) % kASlots], ((pair - 1) / kASlots) & 1);  // the MMAs in flight read shared memory and write tensor memory
    } else if (warp == 3) {
        // ── scales and biases ──
        feed_scales<MODE, 4>(a, line, u0, u1, lane,
            [&](uint32_t it) { return it < C::kRawStages || wait_warp(&raw_empty[it % C::kRawStages], (it / C::kRawStages - 1) & 1, dead); },
            [&](uint32_t it, int i, int j, uint32_t sb) { scales[it % C::kRawStages][j][lane + 32 * i] = sb; },
            [&](uint32_t it) { if (lane == 0) mbar_arrive(&scale_full[it % C::kRawStages]); });
    } else if (warp < kEpilogueWarp + 4) {
        // ── epilogue ──
        const int quad = warp & 3, r = quad * 32 + lane;
        const uint32_t lane_base = tmem + ((uint32_t)(quad * 32) << 16);
        const bool leader = tid == kEpilogueWarp * 32;
        uint32_t done = 0, turn = 0;
        pdl_wait();
        for (int u = u0; u < u1; ++done) {
            const Part t = part_at(line, u, u1, a.batch);
            const uint32_t ds = done % C::kAcc;
            if (!wait_warp(&acc_full[ds], (done / C::kAcc) & 1, dead) && *dead == 0u) *dead = 1u;
            asm volatile("bar.sync 1, 128;" ::: "memory");  // the four warps go on together or not at all
            if (leader) s_go = *dead == 0u ? 1u : 0u;
            asm volatile("bar.sync 1, 128;" ::: "memory");
            if (s_go == 0u) break;
            tc_fence_after();
            const LineRow o = line_row<MODE>(a, line, t.row_tile, r);
            const uint32_t src = lane_base + ds * C::kAccCols;
            auto fetch = [&](int c0, float (&v)[16]) { fetch16<C::kApart ? N : 0>(src + c0, v); };
            const bool shared = t.g0 != 0 || t.g1 != line.groups;
            const size_t part = (size_t)line.tile_cols * kLineRows;
            Sharers sh = {0, 0, 0};
            bool finish = true;
            if (shared) {
                sh = sharers(line, t.tile, gridDim.x);
                float4* mine = reinterpret_cast<float4*>(a.part_scratch + (size_t)sh.slot(blockIdx.x) * part) + r;  // [four columns][row]
                for (int c0 = 0; c0 < t.live; c0 += 16) {
                    float v[16];
                    fetch(c0, v);
#pragma unroll
                    for (int j = 0; j < 16; j += 4) __stcg(mine + (c0 + j) / 4 * kLineRows, make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]));
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[ds]);
                __threadfence();
                asm volatile("bar.sync 1, 128;" ::: "memory");
                if (leader) s_ticket = (uint32_t)atomicAdd(a.part_counters + t.tile, 1);
                asm volatile("bar.sync 1, 128;" ::: "memory");
                finish = s_ticket == (uint32_t)(sh.last - sh.first);
                if (finish) {
                    __threadfence();
                    if (leader) a.part_counters[t.tile] = 0;  // the next launch finds every counter at zero
                }
            }
            if (finish) {
                const bool row_ok = o.row < o.rows;
                for (int c0 = 0; c0 < t.live; c0 += 16) {
                    float v[16];
                    if (shared) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) v[j] = 0.f;
                        for (int c = sh.first; c <= sh.last; c += 4) {  // four CTAs' sums on their way at a time: one after the other each cost 1 us per 16 columns
                            float4 f[4][4];
#pragma unroll
                            for (int z = 0; z < 4; ++z) {
                                const float4* p = reinterpret_cast<const float4*>(a.part_scratch + (size_t)sh.slot(min(c + z, sh.last)) * part) + c0 / 4 * kLineRows + r;
#pragma unroll
                                for (int j = 0; j < 4; ++j) f[z][j] = __ldcg(p + j * kLineRows);
                            }
#pragma unroll
                            for (int z = 0; z < 4; ++z)
                                if (c + z <= sh.last)
#pragma unroll
                                    for (int j = 0; j < 4; ++j) { v[4 * j] += f[z][j].x; v[4 * j + 1] += f[z][j].y; v[4 * j + 2] += f[z][j].z; v[4 * j + 3] += f[z][j].w; }
                        }
                    } else {
                        fetch(c0, v);
                    }
                    const int n = t.live - c0;
                    if (MODE == kAffineGateUp) {
                        // rows r and r ^ 64 are gate and up of one row of the result: the gate's thread takes the first eight columns, the up's the others
                        const bool up = r >= 64;
                        float* ex = exchange + (turn++ & 1) * kLineRows * 8;  // [value][row]
#pragma unroll
                        for (int j = 0; j < 8; ++j) ex[j * kLineRows + r] = up ? v[j] : v[8 + j];
                        asm volatile("bar.sync 1, 128;" ::: "memory");  // the other half is written before this one is again
                        __half* y = o.y + (size_t)(t.col0 + c0 + (up ? 8 : 0)) * o.rows + o.row;
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const float other = ex[j * kLineRows + (r ^ 64)];
                            const __half z = swiglu_f32(up ? other : v[j], up ? v[8 + j] : other);  // lut_matvec.metal:2228
                            if (row_ok && j + (up ? 8 : 0) < n) y[(size_t)j * o.rows] = z;
                        }
                    } else if (row_ok) {
                        const size_t at = (size_t)(t.col0 + c0) * o.rows + o.row;
                        __half res[16];
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            if (MODE == kAffineAdd) res[j] = j < n ? a.residual[at + (size_t)j * o.rows] : __half(0.f);
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            if (j < n) o.y[at + (size_t)j * o.rows] = MODE == kAffineAdd ? __hadd(__float2half_rn(v[j]), res[j]) : __float2half_rn(v[j]);  // lut_matvec.metal:1802-1803
                    }
                    __syncwarp();  // the next tensor-memory load needs the whole warp
                }
            }
            if (!shared) {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[ds]);
            }
            u += t.g1 - t.g0;
        }
    } else {
        // ── expansion: two sets of four warps take turns ──
        const int set = (warp - kExpandWarp) >> 2, quad = warp & 3, r = quad * 32 + lane;
        const uint32_t dst = tmem_a + ((uint32_t)(quad * 32) << 16), raw_a = smem_u32(raw);
        uint32_t pair = 0, stage = 0;
        bool alive = true;
        for (int u = u0; u < u1 && alive;) {
            const Part t = part_at(line, u, u1, a.batch);
            for (int g = t.g0; g < t.g1 && alive; g += kStageGroups, ++stage) {
                const uint32_t s = stage % C::kRawStages, ph = (stage / C::kRawStages) & 1;
                const bool b0 = peek(&raw_full[s], ph), b1 = peek(&scale_full[s], ph);
                if ((!__all_sync(0xffffffffu, b0) && !wait_warp(&raw_full[s], ph, dead)) || (!__all_sync(0xffffffffu, b1) && !wait_warp(&scale_full[s], ph, dead))) { alive = false; break; }
                const uint32_t src = raw_a + s * kRawBytes + r * 128;
                const int n = min(kStageGroups, t.g1 - g);
                for (int k = 0; 2 * k < n; ++k, ++pair) {
                    const uint32_t as = pair % kASlots, use = pair / kASlots;
                    if ((int)as != set) continue;
                    if (use > 0 && !wait_warp(&a_empty[as], (use - 1) & 1, dead)) { alive = false; break; }
                    tc_fence_after();
#pragma unroll 1
                    for (int i = 2 * k; i < min(n, 2 * k + 2); ++i) {
                        const float2 f = __half22float2(u32_as_h2(scales[s][i][r]));
                        const uint64_t s2 = pack2(f.x, f.x), b2 = pack2(f.y, f.y);
#pragma unroll
                        for (int p = 0; p < 2; ++p) {
                            const uint4 v = lds128(src + (((2 * i + p) ^ (r & 7)) << 4));
                            const uint32_t word[4] = {v.x, v.y, v.z, v.w};
                            uint32_t hi[16], lo[16];
#pragma unroll
                            for (int q = 0; q < 4; ++q) expand_hi_lo(word[q], s2, b2, hi + 4 * q, lo + 4 * q);
                            const uint32_t to = dst + as * 128 + (i & 1) * 64 + p * 16;
                            tmem_st16(to, hi);
                            tmem_st16(to + 32, lo);
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
