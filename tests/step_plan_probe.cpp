// Walks over the shapes that step_layers_plan takes and checks what the kernel relies on; prints how many there were.
#include <cstdio>

#include "../cuqwen_b200/csrc/step_layers.h"

using namespace cq;

int main() {
    long taken = 0, bad = 0;
    const int heads[][2] = {{1, 1}, {14, 2}, {12, 2}, {16, 2}, {28, 4}, {40, 8}, {8, 1}, {64, 8}, {96, 96}};
    for (int sms : {148, 132, 80})
        for (int quant = 0; quant < 3; ++quant)
            for (int hd : {64, 128})
                for (auto& h : heads)
                    for (int dim = 128; dim <= 8192; dim += dim < 1024 ? 128 : 896)
                        for (int inter = 128; inter <= 24576; inter += 128) {
                            if (h[0] * hd % 128) continue;
                            const StepShape s{quant, dim, inter, h[0], h[1], hd, 2, 4096, sms / h[1] ? sms / h[1] : 1, sms};
                            StepCore a = {};
                            size_t words[7];
                            if (!step_layers_plan(s, a, words)) continue;
                            ++taken;
                            bool ok = a.smem <= 227 * 1024 && a.off_ring % 1024 == 0 && a.slots >= 4 && 2 * a.slots <= kStepBars && 2 * hd * 2 * (hd == 128 ? 32 : 64) <= a.slot_bytes;
                            // past the ring: the rows of a tile that its block does not have; the staged vector and what the attention lays over it
                            ok = ok && a.off_bars - (a.off_ring + a.slots * a.slot_bytes) >= 15 * 64 && a.off_bars % 8 == 0;
                            const int area = a.off_corr - a.off_x;
                            ok = ok && area >= 8 * (hd / 16 * 512 + 256) && area >= kStepWarps * hd * 4 + kStepWarps * 8;
                            for (int i = 0; i < SP_COUNT; ++i) {
                                const StepGemv& g = a.g[i];
                                const int unit = quant == 2 ? 64 : 128, cols = quant ? 128 : 64, last = g.rows - (g.nblk - 1) * g.brows;
                                ok = ok && g.U == g.K / cols && g.units >= 1 && g.nst * g.units >= g.U && (g.nst - 1) * g.units < g.U;
                                ok = ok && (g.nst == 1 || g.units < g.kp || g.units % g.kp == 0);                  // one distance from a warp's group to its next
                                ok = ok && g.units * unit / 64 <= 256 && g.brows <= 128 && g.stage_bytes == g.mt * g.brows * g.units * unit && g.stage_bytes <= a.slot_bytes;
                                ok = ok && g.nt * g.kp <= kStepWarps && g.rt * 16 >= g.brows && g.brows << g.ks <= 32 * kStepWarps && 1 << g.ks >= g.kp && area >= 2 * g.K;
                                if (quant) ok = ok && g.brows * g.ngrp * 2 % 16 == 0 && g.off_scale % 16 == 0;       // untiled copies
                                if (quant && i != SP_QKV) ok = ok && last > 0 && last * g.ngrp * 2 % 16 == 0;
                            }
                            ok = ok && (!a.staged_h || (a.g[SP_MLP].brows == 128 && inter / 128 >= 80));
                            if (!ok && bad++ < 5) printf("bad: sms %d quant %d hd %d heads %d/%d dim %d inter %d\n", sms, quant, hd, h[0], h[1], dim, inter);
                        }
    printf("%ld shapes, %ld bad\n", taken, bad);
    return bad || taken < 10000;
}
