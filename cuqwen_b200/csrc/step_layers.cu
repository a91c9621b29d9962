// Host side of the one-kernel step: work split, shared-memory map, tensor maps.
#include <string.h>

#include "attn.cuh"
#include "gemv.cuh"
#include "step_layers.h"
#include "tensor_map.h"

namespace cq {

int launch_step_layers_i4(const StepArgs& a, const LaunchCfg& cfg);
int launch_step_layers_i8(const StepArgs& a, const LaunchCfg& cfg);
int launch_step_layers_f16(const StepArgs& a, const LaunchCfg& cfg);
int launch_step_layers(int quant, const StepArgs& a, const LaunchCfg& cfg) {
    return quant == Q_I4 ? launch_step_layers_i4(a, cfg) : quant == Q_I8 ? launch_step_layers_i8(a, cfg) : launch_step_layers_f16(a, cfg);
}

static constexpr int kWarps = kStepWarps, kSmem = 227 * 1024;

static int unit_bytes(int quant) { return quant == Q_I4 ? 64 : 128; }       // of one row: 128 columns quantised, 64 columns fp16
static int unit_cols(int quant) { return quant == Q_F16 ? 64 : 128; }

// Rows of a block.  Every phase ends when its slowest CTA does, so the rows of the CTA that has most are kept few: any even number of rows (tiles of sixteen are the
// products' matter, a box takes what it is given) whose scales begin on 16 bytes in every matrix of `ng` groups that is cut this way.
static int block_rows(int rows, int sms, bool scales, int ng0, int ng1) {
    int best = 8, best_cost = 1 << 30;
    for (int b = 8; b <= 128; b += 2) {
        if (scales && ((b * ng0) % 8 || (b * ng1) % 8)) continue;
        const int cost = ((rows + b - 1) / b + sms - 1) / sms * b;
        if (cost <= best_cost) { best_cost = cost; best = b; }
    }
    return best;
}

bool step_layers_plan(const StepShape& s, StepCore& a, size_t (&words)[7]) {
    const int qd = s.n_heads * s.hd, grp = s.n_heads / s.n_kv;
    if (s.sms < 1 || s.n_layers < 1 || s.n_layers > (int)kSeqPerStep - 2 || s.n_heads > s.sms || s.n_kv * s.nsplit > s.sms || s.nsplit > kMaxSplit || grp > kMaxGroup ||
        (s.hd != 64 && s.hd != 128) || (size_t)s.n_layers * s.n_kv * s.max_seq > 0x7fffffff || s.dim > 8192 || s.dim % kGroup || qd % kGroup || s.inter % kGroup || s.inter > 24576 || qd > 24576) return false;
    a.n_layers = s.n_layers; a.dim = s.dim; a.inter = s.inter; a.n_heads = s.n_heads; a.n_kv = s.n_kv; a.grp = grp; a.hd = s.hd; a.max_seq = s.max_seq; a.nsplit = s.nsplit; a.inv_dim = 1.0f / (float)s.dim;
    const bool q = s.quant != Q_F16;
    const int ngd = s.dim / kGroup, ngq = qd / kGroup, ngi = s.inter / kGroup, gb = unit_bytes(s.quant);
    const int rows_out = block_rows(s.dim, s.sms, q, ngq, ngi);
    int rows_mlp = block_rows(s.inter, s.sms, q, ngd, ngd);
    // whole 128-row groups let the SwiGLU output travel as digits, converted once instead of in every CTA of the down projection, where they cost next to nothing
    auto cost = [&](int b) { return ((s.inter + b - 1) / b + s.sms - 1) / s.sms * b; };
    a.staged_h = q && ngi >= 80 && cost(128) <= cost(rows_mlp) * 33 / 32;
    if (a.staged_h) rows_mlp = 128;
    // a slot: 16 KB (keys and values of 32 or 64 tokens), or what one unit of the widest phase needs
    a.slot_bytes = 2 * rows_mlp * gb > 16 * 1024 ? (2 * rows_mlp * gb + 1023) / 1024 * 1024 : 16 * 1024;
    // ... or one unit of each K-part, where that is little more (0.5B fp16: gate/up blocks of 34 rows, 17 KB)
    auto widen = [&](int rows, int mt, int K) {
        const int kp = kWarps / (mt * ((rows + 15) / 16)), U = K / unit_cols(s.quant), want = mt * rows * gb * (kp < U ? kp : U);
        if (want > a.slot_bytes && want <= 20 * 1024) a.slot_bytes = (want + 1023) / 1024 * 1024;
    };
    widen(16, 2, s.dim); widen(rows_out, 1, qd); widen(rows_mlp, 2, s.dim); widen(rows_out, 1, s.inter);
    auto phase = [&](int i, int K, int rows, int all, int nblk, int mt) {
        StepGemv& g = a.g[i];
        g.K = K; g.ngrp = K / kGroup; g.brows = rows; g.nblk = nblk; g.nb = (nblk + s.sms - 1) / s.sms; g.mt = mt; g.rt = (rows + 15) / 16; g.nt = mt * g.rt; g.kp = kWarps / g.nt; g.rows = all;
        for (g.ks = 0; 1 << g.ks < g.kp;) ++g.ks;
        const int U = K / unit_cols(s.quant);
        int u = a.slot_bytes / (mt * rows * gb);
        if (u * gb / 64 > 256) u = 256 * 64 / gb;                        // (a copy's box; before the next line, as stages of several K-parts hold whole rounds of them)
        if (u > g.kp) u = u / g.kp * g.kp;
        if (u > U) u = U;
        g.U = U; g.ustride = gb * rows; g.units = u; g.nst = (U + u - 1) / u;
        g.box_bytes = rows * u * gb; g.stage_bytes = mt * g.box_bytes;
        g.scale_bytes = q ? mt * rows * (K / kGroup) * 2 : 0;
    };
    phase(SP_QKV, s.dim, 16, 16, (s.n_heads + 2 * s.n_kv) * (s.hd / 32), 2);
    phase(SP_O, qd, rows_out, s.dim, (s.dim + rows_out - 1) / rows_out, 1);
    phase(SP_MLP, s.dim, rows_mlp, s.inter, (s.inter + rows_mlp - 1) / rows_mlp, 2);
    phase(SP_DOWN, s.inter, rows_out, s.dim, (s.dim + rows_out - 1) / rows_out, 1);
    // shared memory: the staged vector (digits or fp16) with the attention's merge buffers over it, small areas, scales, ring, barriers
    int K = s.dim > qd ? s.dim : qd;
    if (s.inter > K) K = s.inter;
    const int merge = 8 * (s.hd / 16 * 512 + 256), folds = kWarps * (s.hd + 2) * 4;
    int area = 2 * K, o = (int)sizeof(StepCore);
    for (int m : {merge, folds}) if (area < m) area = m;
    auto take = [&](int bytes, int align) { o = (o + align - 1) / align * align; const int at = o; o += bytes; return at; };
    a.off_x = take(area, 128);
    a.off_corr = take(K / kGroup * 8, 16); a.off_job = take(SP_COUNT * kWarps * kStepJobBytes, 16);
    a.off_zero = take(256, 16); a.off_red = take(2 * kWarps * kStepRed * 4, 16); a.off_rms = take(kWarps * 4, 16);
    a.off_q = take(kMaxGroup * (s.hd * 2 + 64), 16); a.off_cur = take(s.hd == 128 ? 32 * 128 + 256 : 256, 128); a.off_hbuf = take(256 + 264 + 8, 16);
    a.off_res = take(a.g[SP_O].nb * rows_out * 2, 16); a.off_rope = take(a.g[SP_QKV].nb * 16 * 8, 16); a.off_range = take(kStepRangeBytes, 16);
    for (int i = 0; i < SP_COUNT; ++i) a.g[i].off_scale = take(a.g[i].nb * a.g[i].scale_bytes, 128);
    a.off_ring = take(0, 1024);            // (the swizzle's pattern)
    const int bars = (2 * kStepBars + 2 * SP_COUNT) * 8;
    // a tile's last rows may lie beyond its block: their loads run up to 15 rows past the last stage, their scales up to 15 rows past the scales (into the ring)
    a.slots = (kSmem - o - 1024 - bars) / a.slot_bytes;
    if (a.slots > kStepBars / 2) a.slots = kStepBars / 2;
    if (a.slots < 4) return false;
    a.off_bars = a.off_ring + a.slots * a.slot_bytes + 1024; a.smem = a.off_bars + bars;
    for (const StepGemv& g : a.g) if (g.stage_bytes > a.slot_bytes || g.units < 1 || g.brows << g.ks > 32 * kWarps) return false;
    words[0] = words[1] = s.dim / 2; words[5] = qd / 2; words[2] = (size_t)(s.n_heads + 2 * s.n_kv) * (s.hd / 2);
    words[3] = (size_t)s.n_heads * s.nsplit * s.hd; words[4] = (size_t)s.n_heads * s.nsplit * 2;
    words[6] = a.staged_h ? (size_t)ngi * 66 : (size_t)s.inter / 2;
    return true;
}

int step_layers_maps(const StepShape& s, StepArgs& a, const void* const (&w)[SM_COUNT], const void* kc, const void* vc) {
    const int gb = unit_bytes(s.quant), cols = unit_cols(s.quant);
    for (int m = 0; m < SM_COUNT; ++m) {
        const StepGemv& g = a.c.g[m <= SM_V ? SP_QKV : m == SM_O ? SP_O : m <= SM_UP ? SP_MLP : SP_DOWN];
        const size_t rb = (size_t)g.K / cols * gb, rows = m == SM_Q ? (size_t)s.n_heads * s.hd : m <= SM_V ? (size_t)s.n_kv * s.hd : m == SM_O || m == SM_DOWN ? s.dim : s.inter;
        if (int r = encode_layer_map(&a.tmap[m], w[m], rb, rows, s.n_layers, a.c.layer_stride, g.units * gb, g.brows)) return r;
    }
    const size_t rows = (size_t)s.n_layers * s.n_kv * s.max_seq;
    if (int r = encode_cache_map(&a.kv[0], kc, rows, s.hd, s.hd == 128 ? 32 : 64)) return r;
    return encode_cache_map(&a.kv[1], vc, rows, s.hd, s.hd == 128 ? 32 : 64);
}

}  // namespace cq
