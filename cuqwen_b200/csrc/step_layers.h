// All layers of a decoded token as one kernel (step_layers.cuh): argument block and host interface.
#pragma once
#include <cuda.h>

#include "launch.h"

namespace cq {

// What the kernel and the host's map of its shared memory have in common.
constexpr int kStepWarps = 16;                // consumer warps
constexpr int kStepRed = 17;                  // floats of a warp's sixteen sums, with one between so that K-parts lie in different banks
constexpr int kStepBars = 32;                 // pairs of stage barriers: twice the slots of the ring, at least
constexpr int kStepRangeBytes = 64, kStepJobBytes = 16;
constexpr unsigned kStepWaitCycles = 2000000000u;      // about a second, and less than the 32-bit counter's period

enum StepMat : int { SM_Q = 0, SM_K, SM_V, SM_O, SM_GATE, SM_UP, SM_DOWN, SM_COUNT };
enum StepPhase : int { SP_QKV = 0, SP_O, SP_MLP, SP_DOWN, SP_COUNT };

// One of a layer's four matrix phases.  A block is `brows` consecutive rows of each of the phase's `mt` matrices (q/k/v: 16 rows i and the 16 rows i + hd/2 of a
// head), its 16-row tiles x `kp` K-parts are the consumer warps' work; it streams through the ring in `nst` stages of `units` column units
// (128 columns of a quantised matrix, 64 of an fp16 one).  Blocks go to CTAs round-robin, nb is the most a CTA has.
// U: units of a row; ustride: bytes between a stage's units; nt: tiles of a block; ngrp: scale groups of a row; ks: log2 of kp, rounded up.
struct alignas(16) StepGemv { int nst, units, U, stage_bytes, kp, nt, ustride, ngrp, K, brows, nblk, rt, box_bytes, mt, off_scale, scale_bytes, rows, nb, ks, pad; };

struct StepCore {                    // everything but the tensor maps; the kernel keeps it at the start of its shared memory
    const __half* scale[SM_COUNT];   // layer 0's; a layer's tensors lie layer_stride bytes behind those of the layer before
    const __half* bias[3];
    const __half* norm[2];
    size_t layer_stride;
    __half *x, *q, *k, *v, *att, *gate;      // x: in (token's embedding row) and out (what the final norm reads); the others receive the last layer's vectors
    __half *kc, *vc;                 // [layers][n_kv][max_seq][hd]
    const int* d_pos;
    const unsigned* epoch;           // number of this step; sequence numbers derive from it
    unsigned* err;
    // words {payload, sequence}: residual stream after attention / after the MLP (two halves a word), q k v (the halves d and d + hd/2 of a head), partials
    // [head][split][hd] and [head][split][max, sum] (fp32), attention output, SwiGLU output (two halves a word, or 66 words a group: digits, correction, scale)
    uint2 *w_x1, *w_x2, *w_qkv, *w_part, *w_ml, *w_att, *w_h;
    StepGemv g[SP_COUNT];
    int n_layers, dim, inter, n_heads, n_kv, grp, hd, max_seq, nsplit, staged_h;
    float eps, inv_dim, scale_log2, theta;
    unsigned wait_cycles, started, expired, seq0;   // bound of the waits, in SM cycles; in a CTA's copy: when it began, the code of the first wait that expired, the step's first sequence number less one
    int off_x, off_corr, off_red, off_rms, off_cur, off_job, off_zero, off_q, off_hbuf, off_res, off_rope, off_range, off_ring, slots, slot_bytes, off_bars, smem;
};
struct alignas(64) StepArgs {
    CUtensorMap tmap[SM_COUNT];      // byte maps {64, rows, row bytes / 64, layers}, box {64, brows, bytes of a stage's row piece / 64, 1}
    CUtensorMap kv[2];               // caches as rows of hd / 64 pieces of 128 bytes: {64 halves, all rows, pieces}, box {64, keys of a stage, pieces}, 128-byte swizzle
    StepCore c;
};

// What the plan needs to know of an engine.
struct StepShape { int quant, dim, inter, n_heads, n_kv, hd, n_layers, max_seq, nsplit, sms; };

// Work split and shared-memory map; false: this shape keeps the launch-by-launch step.  Words of the seven exchange buffers go to words[7] (in the order of
// StepCore).
bool step_layers_plan(const StepShape& s, StepCore& a, size_t (&words)[7]);
// Tensor maps of the seven matrices, layer 0's at w[].
int step_layers_maps(const StepShape& s, StepArgs& a, const void* const (&w)[SM_COUNT], const void* kc, const void* vc);
int launch_step_layers(int quant, const StepArgs& a, const LaunchCfg& cfg);

}  // namespace cq
