// Launcher interface of the affine u4 matvec family (affine_matvec.cu).
#pragma once
#include "common.cuh"

namespace smelt {

enum AffineMode : int {
    kAffinePlain = 0,   // y = half(acc)                               affine_matvec
    kAffineAdd = 1,     // y = half(acc) + residual (fp16 add)         fused_affine_matvec_add
    kAffineGateUp = 2,  // y = half(silu(gate) * up), fp32 gate/up     fused_affine_gate_up_swiglu
    kAffineDual = 3,    // y = half(acc0), y2 = half(acc1)             fused_dual_affine_matvec
};

// One row range of a multi-tensor launch (plain mode only): e.g. Q | K | V sharing x.
struct AffineSeg {
    const uint8_t* w;
    const __half* s;
    const __half* b;
    __half* y;     // [batch, rows] of this segment
    int rows;      // a multiple of 16 for every segment but the last
};

struct AffineArgs {
    const uint8_t* w[2];   // packed nibbles [rows, cols/2]; [1] = up / second matrix
    const __half* s[2];    // scales [rows, cols/group]
    const __half* b[2];    // biases [rows, cols/group]
    const __half* x;       // activations [batch, cols]
    __half* y;             // [batch, rows]
    __half* y2;            // dual mode: second output
    const __half* residual;  // add mode: [batch, rows]; may alias y
    int rows, cols, batch;
    // Streaming kernel only.  norm_w != null: x is RMS-normalised while it is staged, with
    // the rounding points of rms_norm_1pw (half(x*rs) times half(1+w)).  nseg > 1: plain mode
    // over several tensors; rows is then the total row count.
    const __half* norm_w;
    float norm_eps;
    int nseg;
    AffineSeg seg[3];
    int ks, nsplit;        // filled by the launcher
    int sm_count;          // SMs of the device (0 = assume 148)
    // Tensor-core product only: where CTAs that share a tile leave their fp32 sums, behind them the group sums of x
    // (tiles of more than 64 rows) and at the end the rows of a norm that is a launch of its own
    // (part_scratch_bytes bytes), and where they count their arrivals (one int per tile, 4096 of them,
    // all zero between launches).  Launches that use them must not overlap on the device.
    float* part_scratch;
    size_t part_scratch_bytes;
    int* part_counters;
    uint32_t* err;         // device error word (may be null)
    DevDyn dyn;            // filled by the launcher
};

// The launch for rows [r0, r0 + n) of x.
inline AffineArgs affine_rows(const AffineArgs& a, int r0, int n) {
    AffineArgs s = a;
    s.batch = n;
    s.x = a.x + (size_t)r0 * a.cols;
    if (a.y) s.y = a.y + (size_t)r0 * a.rows;
    if (a.y2) s.y2 = a.y2 + (size_t)r0 * a.rows;
    if (a.residual) s.residual = a.residual + (size_t)r0 * a.rows;
    for (int i = 0; i < a.nseg && i < 3; ++i) s.seg[i].y = a.seg[i].y + (size_t)r0 * a.seg[i].rows;
    return s;
}

cudaError_t launch_affine(const Launch& l, int mode, const AffineArgs& args, int group);
// A folded norm and its product (one tensor, gate and up, or Q, K and V with as many rows of K as of V) as the separate launches that they stand
// for: any alignment but that of the packed weights (16 bytes), any number of columns.
cudaError_t launch_affine_apart(const Launch& l, int mode, const AffineArgs& args, int group);
cudaError_t launch_affine_stream(const Launch& l, int mode, const AffineArgs& args, int group, bool* handled);
// Tensor-core product for many rows of x (affine_wide.cu; from how many: wide_first in affine_matvec.cu).
cudaError_t launch_affine_wide(const Launch& l, int mode, const AffineArgs& args, int group, bool* handled);
// Passes of the streaming kernel over the weights for up to sixteen rows of x, 0 where it does not take the launch.
int affine_stream_passes(int mode, const AffineArgs& args, int group);
cudaError_t launch_affine_imma(const Launch& l, int mode, const AffineArgs& args, int group, bool* handled);

}  // namespace smelt
