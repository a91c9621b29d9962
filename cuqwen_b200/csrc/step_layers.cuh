// All layers of a decoded token in ONE cooperative kernel, one CTA per SM: a producer thread and sixteen consumer warps.
//
// What bounds a decoded token is not the streaming of its weights but the chain between them: as separate launches every projection waits for the one
// before it (0.65 us), fetches the vector (1.3 us and more), normalises and converts it, all with the memory idle as soon as the ring it could fill ahead is full.
// Here the producer never waits for the step's data: it streams the weights, scales and cached keys and values of ALL layers, in the order
// in which the consumers use them, through one ring that fills the SM's shared memory, and runs ahead across the borders of phases and layers.
// The consumers hand their vectors from CTA to CTA through L2 as words {payload, sequence number} of eight bytes (the tensor-parallel exchange's form): a reader
// polls the very words it needs, so a hand-over is one store and one load (some 700 cycles), without a barrier, a flag or a fence.  A word's number is
// step * kSeqPerStep + layer + 1; a buffer is written once a layer, and every CTA that writes layer l + 1's words has read words that depend, through
// the phases between, on every reader of layer l's.  The CTAs wait for one another, hence the cooperative launch.
//
// Phases of a layer: q/k/v (RMSNorm, bias, rotation, cache store), attention partials per (KV head, key range), merge of a head's partials (one CTA a head), output projection +
// residual, gate/up + SwiGLU, down projection + residual.  A CTA keeps the residual of its own rows in shared memory (the two row-parallel projections are cut
// alike).  CTAs without work in a phase do not read its input.
//
// Measured, us a step, launch by launch -> here (one B200, in turn on the same box): 0.5B int4 at 255 keys 679 -> 428, 0.5B fp16 at 1777 with the penalty 660 -> 488, 7B int4 at 8192 1489 -> 1102, six 14B
// int8 layers at 31,999 688 -> 625.  What the phases take, in cycles of 1.9 GHz (0.5B int4 at 255 keys / 7B int4 at 8192, one thread's stamps, median of the CTAs): words from one phase's end until they
// are here 1600 to 1700 / 1800 to 2300; a vector to digits, or SwiGLU's digits to shared memory, 650 to 2400 / 1000 to 1900; products of q/k/v 1140 / 2700, of o 950 / 2660, of gate/up 2260 / 16,500
// (7B: 70 MB), of down 1820 / 10,950; a block's finish 930 to 1180 / 920 to 1460; attention: q 3500 / 2000, tiles 2700 / 3640, merge of the warps 2260 / 1990; merge of a head's partials 8700 (0.5B
// at 1777 keys) / 5800.  A 7B layer takes 66,000 cycles, its bytes alone would take 39,000.
// A warp's products of one group cost some 600 cycles next to the fifteen other warps' (operands from shared memory 390 and the integer MMAs 300), a chain, not a rate.  Slower were: the next
// group's weights loaded ahead (7B 1094 -> 1240 us), two groups side by side (1173), rolled loops in the attention (1100 to 1135), a head's merge shared out among the CTAs that it has (1128),
// polls through one lane a warp (1160) and weights asked into L2 ahead of the ring (1210).
//
// What this cost most to find: the consumers' code must fit the instruction caches (118 KB of phases inlined four times took 40 us a layer of the 0.5B model, 60 KB with one copy of
// the phases 19), no register may spill (the spill lines' L1 is what 227 KB of shared memory leave, 28 KB; the 14B int8 step 708 -> 637 us, six fp16 layers of 3B 371 -> 340), and keys and values
// must not collide in the banks (a tile 2300 -> 1500 cycles).
#pragma once
#include "attn_split.cuh"
#include "gemv.cuh"
#include "step_layers.h"

namespace cq {

constexpr int kStepConsumers = kStepWarps * 32, kStepThreads = kStepConsumers + 128;      // the producer has a warpgroup to itself, whose registers the consumers take over

template <int Q> struct StepUnit;             // bytes of a row's column unit
template <> struct StepUnit<Q_I4> { static constexpr int GB = 64, COLS = 128; };
template <> struct StepUnit<Q_I8> { static constexpr int GB = 128, COLS = 128; };
template <> struct StepUnit<Q_F16> { static constexpr int GB = 128, COLS = 64; };

__device__ __forceinline__ unsigned long long word_of(uint32_t v, uint32_t seq) { return ((unsigned long long)seq << 32) | v; }
__device__ __forceinline__ void st_word(uint2* p, uint32_t v, uint32_t seq) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(word_of(v, seq)) : "memory");
}
__device__ __forceinline__ void st_word2(uint2* p, uint32_t v0, uint32_t v1, uint32_t seq) {
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1,%2};" ::"l"(p), "l"(word_of(v0, seq)), "l"(word_of(v1, seq)) : "memory");
}
__device__ __forceinline__ void ld_word2(const uint2* p, unsigned long long& a, unsigned long long& b) {
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0,%1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, int w, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(bar) : "memory");
}

// Place in the ring: stage n of the step lies in slot n mod `slots` and is announced by barrier n mod 32 (more barriers than slots: see attend).
struct StepRing {
    uint32_t n, slot;                // next stage, its slot
    uint32_t red;                    // which of the two buffers of the warps' sums comes next
    __device__ __forceinline__ uint32_t bar() const { return (n & (kStepBars - 1)) * 8; }
    __device__ __forceinline__ uint32_t par() const { return (n / kStepBars) & 1u; }
    __device__ __forceinline__ void next(uint32_t slots) { ++n; if (++slot == slots) slot = 0; }
};
__device__ __forceinline__ uint32_t cycles32() { uint32_t t; asm volatile("mov.u32 %0, %clock;" : "=r"(t)); return t; }

// Shared memory of a CTA; the argument block lies at its start, where the consumers' phases read it: read from the parameters, the compiler carries the phases' constants
// through all layers, in registers that sixteen warps (112 a thread) do not have.
extern __shared__ __align__(1024) unsigned char step_smem[];

// Every wait, on the ring or on words, is over when the CTA has run for StepCore::wait_cycles (a step takes some thousandth of the default; a start of its own for every wait would cost a
// register).  The first one that ends so leaves its code in the CTA's argument block, and from then on every wait of the CTA ends at its first look: the CTA goes through the rest of the
// step at once, with whatever its memory holds (no value decides an address), and hands on the words that the other CTAs wait for.  The producer begins no copy after that; those
// under way: see land.
__device__ __forceinline__ uint32_t lds_volatile(uint32_t at) { uint32_t v; asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(v) : "r"(smem_u32(step_smem) + at)); return v; }
__device__ __forceinline__ uint32_t step_expired() { return lds_volatile(offsetof(StepCore, expired)); }
__device__ __forceinline__ bool step_expire(uint32_t code) {
    if (step_expired()) return true;
    if (cycles32() - lds_volatile(offsetof(StepCore, started)) <= lds_volatile(offsetof(StepCore, wait_cycles))) return false;
    asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(smem_u32(step_smem) + (uint32_t)offsetof(StepCore, expired)), "r"(code));
    return true;
}
__device__ __forceinline__ void step_report(unsigned* err) { if (const uint32_t code = step_expired()) atomicExch(err, code); }
// In few instructions: the layers' code has to stay in the instruction cache.
__device__ __forceinline__ void step_wait(uint32_t bar, uint32_t parity, uint32_t code) {
    if (mbar_try_wait(bar, parity)) return;
#pragma unroll 1
    while (!mbar_try_wait(bar, parity))
        if (step_expire(code)) return;
}
// Polls N pairs of words, `stride` words apart, and (EXTRA) the pair at q, until all carry `seq`.
template <int N, int EXTRA = 0>
__device__ __forceinline__ void poll_words(const uint2* p, int stride, const uint2* q, uint32_t seq, uint32_t (&v)[2 * (N + EXTRA)]) {
#pragma unroll 1
    for (;;) {
        uint32_t bad = 0;
        unsigned long long a[N + EXTRA], b[N + EXTRA];
#pragma unroll
        for (int i = 0; i < N; ++i) ld_word2(p + i * stride, a[i], b[i]);
        if (EXTRA) ld_word2(q, a[N + EXTRA - 1], b[N + EXTRA - 1]);
#pragma unroll
        for (int i = 0; i < N + EXTRA; ++i) { v[2 * i] = (uint32_t)a[i]; v[2 * i + 1] = (uint32_t)b[i]; bad |= ((uint32_t)(a[i] >> 32) ^ seq) | ((uint32_t)(b[i] >> 32) ^ seq); }
        if (bad == 0 || step_expire(11u)) return;
    }
}
template <int N>
__device__ __forceinline__ void poll_words(const uint2* p, int stride, uint32_t seq, uint32_t (&v)[2 * N]) { poll_words<N, 0>(p, stride, nullptr, seq, v); }

template <int Q, int HD>
struct StepLayers {
    static constexpr bool kInt = Q != Q_F16;
    static constexpr int GB = StepUnit<Q>::GB;
    static __device__ __forceinline__ const StepCore& core() { return *reinterpret_cast<const StepCore*>(step_smem); }
    static __device__ __forceinline__ uint32_t bar_full(const StepCore& a) { return smem_u32(step_smem) + a.off_bars; }
    static __device__ __forceinline__ uint32_t bar_empty(const StepCore& a) { return smem_u32(step_smem) + a.off_bars + kStepBars * 8; }
    static __device__ __forceinline__ uint32_t bar_sfull(const StepCore& a, int ph) { return smem_u32(step_smem) + a.off_bars + (2 * kStepBars + ph) * 8; }
    static __device__ __forceinline__ uint32_t bar_sempty(const StepCore& a, int ph) { return smem_u32(step_smem) + a.off_bars + (2 * kStepBars + SP_COUNT + ph) * 8; }
    // What every layer needs to know, computed once: the attention's key range, the head to merge, the blocks of each phase.
    struct Range { int kvh, split, t0, t1c, nstage, any, own, nne; int pos, fold_head; int nb[SP_COUNT]; };
    static_assert(sizeof(Range) <= kStepRangeBytes, "");
    static __device__ __forceinline__ const Range& range(const StepCore& a) { return *reinterpret_cast<const Range*>(step_smem + a.off_range); }
    // A warp's part of a phase's blocks: byte offset of its tile in a stage, of its tile's first scale row in a block's scales, its K-part (or none).
    struct alignas(kStepJobBytes) Job { int in_stage, scales, part; };
    static_assert(sizeof(Job) == kStepJobBytes, "");
    static __device__ __forceinline__ Job& job(const StepCore& a, int ph, int warp) { return reinterpret_cast<Job*>(step_smem + a.off_job)[ph * kStepWarps + warp]; }

    template <class T> static __device__ __forceinline__ const T* at_layer(const StepCore& a, const T* p, int l) { return reinterpret_cast<const T*>(reinterpret_cast<const char*>(p) + (size_t)l * a.layer_stride); }
    // block of the q/k/v phase -> matrix, first row inside it
    static __device__ __forceinline__ void qkv_tile(const StepCore& a, int blk, int& mat, int& row) {
        constexpr int spt = HD / 32;
        const int hh = blk / spt, sub = blk - hh * spt, nh = a.n_heads, nk = a.n_kv;
        mat = hh < nh ? 0 : hh < nh + nk ? 1 : 2;
        row = (mat == 0 ? hh : mat == 1 ? hh - nh : hh - nh - nk) * HD + sub * 16;
    }

    // ---- producer -----------------------------------------------------------
    static constexpr int kRowB = HD * 2, kKeys = HD == 128 ? 32 : 64, kHalf = kKeys * kRowB, kPer = kKeys / 32;      // keys of a stage, warps that share one
    static constexpr int kRowQ = kRowB + 64;      // a row of q in shared memory: two of them in different banks
    // Contexts of up to so many keys are one range a KV head, eight or nine warps' work, and its CTA writes the attention's output itself: the merge of partials, a hand-over and some 2000
    // cycles, falls away (us a step, 0.5B int4 at 120 keys 432 -> 413, at 250 434 -> 425; at 500 nothing: one SM streams all keys of a head).
    static constexpr int kDirect = 256;
    // A free slot for the next stage, whose barrier then expects `tx` bytes.  One thread issues all copies of an SM, some 40 instructions a stage
    // (slots of one size: with stages packed behind one another it took 90, and was what the large matrices waited for).
    // 0: a wait of this CTA has expired.  That is looked up behind the wait, which may have ended because warps let stages go that they had not waited for.
    static __device__ __forceinline__ uint32_t claim(const StepRing& R, uint32_t full, uint32_t slots, uint32_t tx) {
        const uint32_t before = R.n - slots;                // the stage that had the slot
        if (R.n >= slots) step_wait(full + (kStepBars + (before & (kStepBars - 1))) * 8, (before / kStepBars) & 1u, 4u);
        if (step_expired()) return 0u;
        const uint32_t bar = full + R.bar();
        mbar_expect_tx(bar, tx);
        return bar;
    }
    // Before the CTA ends, also early: the last copies announced by each barrier have arrived, as none may land in the shared memory of a CTA that comes after this one.  Bounded as a
    // step's waits are by default, whatever this step's are.
    static __device__ __forceinline__ void land(const StepCore& a, const StepRing& R, uint32_t scales) {
        const uint32_t full = bar_full(a), t0 = cycles32();
#pragma unroll 1
        for (uint32_t n = R.n > kStepBars ? R.n - kStepBars : 0u; n < R.n; ++n)
            while (!mbar_try_wait(full + (n & (kStepBars - 1)) * 8, (n / kStepBars) & 1u) && cycles32() - t0 <= kStepWaitCycles) {}
#pragma unroll 1
        for (int ph = 0; ph < SP_COUNT; ++ph)
            while (scales >> (8 + ph) & 1u && !mbar_try_wait(bar_sfull(a, ph), scales >> ph & 1u) && cycles32() - t0 <= kStepWaitCycles) {}
    }
    // false: see claim.  scales: which phases' scale barriers were armed (bits 8 ..) and the parity of their last use (bits 0 ..)
    static __device__ __forceinline__ bool produce_gemv(const StepArgs& args, StepRing& R, int ph, int l, int nb, uint32_t& scales) {
        const StepCore& a = args.c;
        const StepGemv& G = a.g[ph];
        const uint32_t sm0 = smem_u32(step_smem), ring = sm0 + a.off_ring, full = bar_full(a), slots = a.slots, slot_bytes = a.slot_bytes;
        const bool qkv = ph == SP_QKV;
        const int mt = qkv || ph == SP_MLP ? 2 : 1, m0 = ph == SP_O ? SM_O : ph == SP_MLP ? SM_GATE : SM_DOWN, ngrp = G.ngrp;
        if (kInt) {
            // the scales of all of the phase's blocks before the first stage: the consumers wait for them once, and the ring need not hold a whole block
            step_wait(bar_sempty(a, ph), (l & 1) ^ 1, 3u);
            uint32_t total = 0;
#pragma unroll 1
            for (int j = 0; j < nb; ++j) total += (uint32_t)(mt * ngrp * 2) * (qkv ? 16 : min(G.brows, G.rows - (int)(blockIdx.x + j * gridDim.x) * G.brows));
            if (step_expired()) return false;
            mbar_expect_tx(bar_sfull(a, ph), total);
            scales = (scales & ~(1u << ph)) | 256u << ph | (uint32_t)(l & 1) << ph;
        }
#pragma unroll 1
        for (int j = 0; j < 2 * nb; ++j) {                  // scales, then stages
            const bool stages = j >= nb;
            const int jj = stages ? j - nb : j, blk = (int)(blockIdx.x + jj * gridDim.x);
            if (!kInt && !stages) continue;
            int mat = m0, row = blk * G.brows, dm = 1, drow = 0;        // the second matrix of a pair, or the second half of a head
            if (qkv) { qkv_tile(a, blk, mat, row); dm = 0; drow = HD / 2; }
            if (!stages) {
                const uint32_t bytes = (uint32_t)((qkv ? 16 : min(G.brows, G.rows - row)) * ngrp * 2);
#pragma unroll 1
                for (int m = 0; m < mt; ++m)
                    bulk_g2s(sm0 + G.off_scale + jj * G.scale_bytes + m * G.brows * ngrp * 2, at_layer(a, a.scale[mat + m * dm], l) + (size_t)(row + m * drow) * ngrp, bytes, bar_sfull(a, ph));
                continue;
            }
            const CUtensorMap *map0 = &args.tmap[mat], *map1 = &args.tmap[mat + dm];
            const uint32_t box = G.box_bytes, tx = G.stage_bytes;
            const int dz = G.units * (GB / kChunkBytes), nst = G.nst;
            int z = 0;
#pragma unroll 1
            for (int p = 0; p < nst; ++p) {
                const uint32_t bar = claim(R, full, slots, tx), dst = ring + R.slot * slot_bytes;
                if (!bar) return false;
                tma_load_4d(dst, map0, 0, row, z, l, bar);
                if (mt == 2) tma_load_4d(dst + box, map1, 0, row + drow, z, l, bar);
                z += dz;
                R.next(slots);
            }
        }
        return true;
    }
    // cached keys and values of this CTA's key range: rows below `pos`, which earlier steps wrote
    static __device__ __forceinline__ Range make_range(const StepCore& a) {
        Range r;
        const int cta = blockIdx.x;
        r.pos = *a.d_pos;
        r.kvh = cta / a.nsplit; r.split = cta - r.kvh * a.nsplit;
        const int len = r.pos + 1, chunk = len <= kDirect ? kDirect : attn_chunk(len, a.nsplit);
        r.t0 = r.split * chunk;
        const int t1 = min(r.t0 + chunk, len);
        r.any = r.kvh < a.n_kv && r.t0 < len;
        r.own = r.any && t1 == len;                   // the step's own key and value, which come from the q/k/v phase
        r.t1c = min(t1, len - 1);
        r.nstage = r.any ? (r.t1c - r.t0 + kKeys - 1) / kKeys : 0;
        r.nne = (len + chunk - 1) / chunk;            // key ranges that are not empty
        const int per_head = gridDim.x / a.n_heads;
        r.fold_head = r.nne > 1 && cta % per_head == 0 && cta / per_head < a.n_heads ? cta / per_head : -1;
        for (int i = 0; i < SP_COUNT; ++i) r.nb[i] = cta < a.g[i].nblk ? (a.g[i].nblk - cta + (int)gridDim.x - 1) / (int)gridDim.x : 0;
        return r;
    }
    static __device__ __forceinline__ bool produce_kv(const StepArgs& args, StepRing& R, int l, const Range& r) {
        const StepCore& a = args.c;
        const uint32_t sm0 = smem_u32(step_smem), ring = sm0 + a.off_ring, full = bar_full(a), slots = a.slots, slot_bytes = a.slot_bytes;
        int row = (l * a.n_kv + r.kvh) * a.max_seq + r.t0;          // rows past the range's end come along and are not used
#pragma unroll 1
        for (int sn = 0; sn < r.nstage; ++sn) {
            const uint32_t bar = claim(R, full, slots, 2 * kHalf), dst = ring + R.slot * slot_bytes;
            if (!bar) return false;
            tma_load_3d(dst, &args.kv[0], 0, row, 0, bar);
            tma_load_3d(dst + kHalf, &args.kv[1], 0, row, 0, bar);
            row += kKeys;
            R.next(slots);
        }
        return true;
    }

    // ---- consumers ----------------------------------------------------------
    // One group of 128 values, four a lane (the digit blocks of gemv_stage.cuh, with a group a warp instead of half a warp: the maximum and the sum are one
    // instruction each, and a group is a quarter of the serial work).
    static __device__ __forceinline__ void digits_of_group(const float (&f)[4], int lane, unsigned char* xd, int2* cx) {
        float m = 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k) m = fmaxf(m, fabsf(f[k]));
        const uint32_t mb = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
        const int e = mb ? 13 - ((int)(mb >> 23) - 127) : 0;              // m in [2^p, 2^(p+1)): e = 13 - p
        const float up = __uint_as_float((uint32_t)(e + 127) << 23);
        int X[4];
        uint32_t d0[4], d1[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            X[k] = __float2int_rn(f[k] * up);
            const int lo = (int)(signed char)(X[k] & 0xff);
            d0[k] = (uint32_t)lo & 0xffu; d1[k] = (uint32_t)((X[k] - lo) >> 8) & 0xffu;
        }
        const int r = lane >> 1, odd = lane & 1;
        if (Q == Q_I4) {          // a chunk of eight is two lanes'; its bytes in the order 0 2 4 6, 1 3 5 7
            unsigned char* o = xd + ((r & 3) >> 1) * 128 + (r >> 2) * 32 + (r & 1) * 8 + odd * 2;
            *reinterpret_cast<unsigned short*>(o) = (unsigned short)(d0[0] | d0[2] << 8); *reinterpret_cast<unsigned short*>(o + 4) = (unsigned short)(d0[1] | d0[3] << 8);
            *reinterpret_cast<unsigned short*>(o + 16) = (unsigned short)(d1[0] | d1[2] << 8); *reinterpret_cast<unsigned short*>(o + 20) = (unsigned short)(d1[1] | d1[3] << 8);
        } else {
            unsigned char* o = xd + (r >> 3) * 128 + ((r >> 1) & 3) * 32 + (r & 1) * 8 + odd * 4;
            *reinterpret_cast<uint32_t*>(o) = d0[0] | d0[1] << 8 | d0[2] << 16 | d0[3] << 24;
            *reinterpret_cast<uint32_t*>(o + 16) = d1[0] | d1[1] << 8 | d1[2] << 16 | d1[3] << 24;
        }
        const int sum = Q == Q_I4 ? __reduce_add_sync(0xffffffffu, X[0] + X[1] + X[2] + X[3]) : 0;
        if (lane == 0) *cx = make_int2(8 * sum, (127 - e) << 23);
    }
    // The phase's input vector into shared memory, in the form the products want: from words of two halves (src), or plain (x of the first layer).
    // Quantised weights: a warp takes a group (two at a time, so that their loads overlap).  A norm's 1 / rms is not waited for: the digits are those of x * weight in fp32, and
    // the rows' sums are multiplied by it (norm_scale), which spares a barrier and a rounding to fp16.
    static __device__ __forceinline__ void stage_vec(const uint2* src, const __half* plain, const __half* norm_w, int K, uint32_t seq) {
        const StepCore& a = core();
        const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
        float* rms = reinterpret_cast<float*>(step_smem + a.off_rms);
        float ss = 0.f;
        if constexpr (kInt) {
            const int ngrp = K / kGroup;
            unsigned char* xd = step_smem + a.off_x;
            int2* cx = reinterpret_cast<int2*>(step_smem + a.off_corr);
#pragma unroll 1
            for (int grp = warp; grp < ngrp; grp += 2 * kStepWarps) {
                const bool two = grp + kStepWarps < ngrp;
                const int to2 = two ? kStepWarps * 32 : 0;               // without a second group the first one is read twice
                uint2 w0 = make_uint2(0x3c003c00u, 0x3c003c00u), w1 = w0;
                uint32_t v[4];
                if (norm_w) { const uint2* n = reinterpret_cast<const uint2*>(norm_w) + grp * 32 + lane; w0 = __ldg(n); w1 = __ldg(n + to2); }
                if (plain) { const uint2* x = reinterpret_cast<const uint2*>(plain) + grp * 32 + lane; const uint2 p = __ldcg(x), q = __ldcg(x + to2); v[0] = p.x; v[1] = p.y; v[2] = q.x; v[3] = q.y; }
                else poll_words<2>(src + grp * 64 + 2 * lane, 2 * to2, seq, v);
#pragma unroll 1
                for (int i = 0; i <= two; ++i) {
                    const uint32_t u0 = i ? v[2] : v[0], u1 = i ? v[3] : v[1], n0 = i ? w1.x : w0.x, n1 = i ? w1.y : w0.y;
                    const float2 f0 = __half22float2(*reinterpret_cast<const __half2*>(&u0)), f1 = __half22float2(*reinterpret_cast<const __half2*>(&u1));
                    const float2 g0 = __half22float2(*reinterpret_cast<const __half2*>(&n0)), g1 = __half22float2(*reinterpret_cast<const __half2*>(&n1));
                    ss += (f0.x * f0.x + f0.y * f0.y) + (f1.x * f1.x + f1.y * f1.y);
                    const float f[4] = {f0.x * g0.x, f0.y * g0.y, f1.x * g1.x, f1.y * g1.y};
                    digits_of_group(f, lane, xd + (grp + i * kStepWarps) * 256, cx + grp + i * kStepWarps);
                }
            }
            if (norm_w) { ss = warp_sum(ss); if (lane == 0) rms[warp] = ss; }
        } else {
            const int nchunk = K / 8;
            uint4* xs = reinterpret_cast<uint4*>(step_smem + a.off_x);
#pragma unroll 1
            for (int c8 = tid; c8 < nchunk; c8 += kStepConsumers) {
                uint4 v;
                if (plain) v = __ldcg(reinterpret_cast<const uint4*>(plain) + c8);
                else {
                    uint32_t w[4];
                    poll_words<2>(src + c8 * 4, 2, seq, w);
                    v = make_uint4(w[0], w[1], w[2], w[3]);
                }
                xs[c8] = v;
                if (norm_w) ss += chunk_sumsq(v);
            }
            if (norm_w) {          // fp16 operands: normalised before they are rounded
                ss = warp_sum(ss);
                if (lane == 0) rms[warp] = ss;
                consumer_sync(kStepConsumers);
                const float inv = norm_scale(a);
#pragma unroll 1
                for (int c8 = tid; c8 < nchunk; c8 += kStepConsumers) xs[c8] = apply_norm(xs[c8], __ldg(reinterpret_cast<const uint4*>(norm_w) + c8), inv);
            }
        }
        consumer_sync(kStepConsumers);
    }
    // 1 / rms from the warps' sums of squares.
    static __device__ __forceinline__ float norm_scale(const StepCore& a) {
        const float4* r = reinterpret_cast<const float4*>(step_smem + a.off_rms);
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < kStepWarps / 4; ++i) { const float4 v = r[i]; s += (v.x + v.y) + (v.z + v.w); }
        return rsqrtf(s * a.inv_dim + a.eps);
    }
    // The SwiGLU output in staged form: 64 words of digits a group, then correction and scale of each.
    static __device__ __forceinline__ void stage_groups(const uint2* src, int ngrp, uint32_t seq) {
        constexpr int NB = 5;
        const StepCore& a = core();
        const int n = ngrp * 32, tid = threadIdx.x;
        uint2* xd = reinterpret_cast<uint2*>(step_smem + a.off_x);
        uint32_t v[2 * NB];
        // NB x 512 pairs at a time, the last ones from where they end with the vector (some are then read twice); ngrp >= 80, so there are that many
#pragma unroll 1
        for (int u = tid;; u += NB * kStepConsumers) {
            const int over = u + (NB - 1) * kStepConsumers - (n - kStepConsumers + tid);
            if (over > 0) u -= over;
            poll_words<NB>(src + 2 * u, 2 * kStepConsumers, seq, v);
#pragma unroll
            for (int i = 0; i < NB; ++i) xd[u + i * kStepConsumers] = make_uint2(v[2 * i], v[2 * i + 1]);
            if (over >= 0) break;
        }
        if (tid < ngrp) {
            uint32_t c[2];
            poll_words<1>(src + 2 * (n + tid), 0, seq, c);
            reinterpret_cast<uint2*>(step_smem + a.off_corr)[tid] = make_uint2(c[0], c[1]);
        }
        consumer_sync(kStepConsumers);
    }

    // What a warp's products need to know of a phase, in registers before the phase's input arrives.
    struct Work {
        uint32_t in_stage, scales, scale_hi, x, zero, cx, full, slots, slot_bytes;
        int nst, units, U, kp, part, ustride, cstride;
    };
    // The sums of this warp's tile and K-part over a block's stages: rows g and g + 8 of the tile in tot[0], tot[1].
    // Quantised weights (gemv_math.cuh): a group's activations are two columns of the B operand, the planes of their digits; there are eight.  The warp's next four groups lie in
    // them side by side, and every one of the four's weights are multiplied with all: group i's sums are those that lane t = i receives, the others mean nothing.  So the
    // activations are read once for four groups (shared memory, which the weights pass through anyway, was the bound), and turning sums into fp32 and scaling them, which only a
    // quarter of the lanes had work for, also comes once for four.
    static __device__ __forceinline__ void block_sums(const Work& W, StepRing& R, uint32_t scales, float (&tot)[2]) {
        const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
        int left = W.U, u0 = 0;
        tot[0] = tot[1] = 0.f;
        float cf[1][2][4] = {};
        int mine[2][4] = {}, cnt = 0, first = W.part;
        uint4 xv[2] = {};
        const int d = min(W.kp, W.units);                           // from one of the warp's groups to the next
        auto flush = [&] {
            const int grp = first + t * d;
            const bool live = t < cnt;
            const uint2 c = lds64(live ? W.cx + grp * 8 : W.zero);
            const uint32_t sa = scales + (live ? grp * 2 : 0);
            const float xs = __uint_as_float(c.y), s0 = lds_h(sa), s1 = lds_h(sa + W.scale_hi);
            if (live) {
                tot[0] = fmaf((float)(group_sum<Q>(mine, 0) - (int)c.x), s0 * xs, tot[0]);
                tot[1] = fmaf((float)(group_sum<Q>(mine, 2) - (int)c.x), s1 * xs, tot[1]);
            }
            first += 4 * d; cnt = 0;
        };
#pragma unroll 1
        for (int p = 0; p < W.nst; ++p) {
            uint32_t w0 = W.in_stage + R.slot * W.slot_bytes + W.part * W.ustride;
            const uint32_t bar = W.full + R.bar();
            step_wait(bar, R.par(), 1u);
            const int n = u0 + min(W.units, left);
#pragma unroll 1
            for (int grp = u0 + W.part; grp < n; grp += W.kp) {
                if constexpr (kInt) {
                    uint4 w[1][2][QT<Q>::NI];
                    int ci[1][2][4];
                    load_group_w<Q, 1>(w0, W.cstride, 0, w);
                    if (cnt == 0) {
                        const uint32_t xa = W.x + min(grp + (g >> 1) * d, W.U - 1) * 256;
                        xv[0] = lds128(xa); xv[1] = lds128(xa + 128);
                    }
                    mma_group_int<Q, 1>(w, xv, ci);
                    if (t == cnt) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) { mine[0][i] = ci[0][0][i]; mine[1][i] = ci[0][1][i]; }
                    }
                    if (++cnt == 4) flush();
                } else {
                    uint4 wa[2], wb[2], x[2];
#pragma unroll
                    for (int c = 0; c < 2; ++c) { wa[c] = lds128(w0 + c * W.cstride); wb[c] = lds128(w0 + c * W.cstride + 8 * kChunkBytes); x[c] = lds128(W.x + grp * 128 + c * 64); }
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        mma16816(cf[0][0], wa[c].x, wb[c].x, wa[c].y, wb[c].y, x[c].x, x[c].y);
                        mma16816(cf[0][1], wa[c].z, wb[c].z, wa[c].w, wb[c].w, x[c].z, x[c].w);
                    }
                }
                w0 += W.kp * W.ustride;
            }
            left -= W.units; u0 += W.units;
            __syncwarp();
            if (lane == 0) mbar_arrive(bar + kStepBars * 8);
            R.next(W.slots);
        }
        if (kInt) {
            if (cnt) flush();
#pragma unroll
            for (int o = 1; o < 4; o <<= 1) { tot[0] += __shfl_xor_sync(0xffffffffu, tot[0], o); tot[1] += __shfl_xor_sync(0xffffffffu, tot[1], o); }
        } else { tot[0] = cf[0][0][0] + cf[0][1][0]; tot[1] = cf[0][0][2] + cf[0][1][2]; }
    }

    static __device__ __forceinline__ void gemv(int ph, int nb, int l, uint32_t seq, StepRing& R) {
        const StepCore& a = core();
        unsigned char* sm = step_smem;
        const uint32_t sm0 = smem_u32(step_smem);
        const StepGemv& G = a.g[ph];
        const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
        const Job J = job(a, ph, warp);
        const bool last = l == a.n_layers - 1;
        Work W;
        W.ustride = G.ustride; W.cstride = W.ustride / (GB / kChunkBytes); W.nst = G.nst; W.units = G.units; W.U = G.U; W.kp = G.kp; W.part = J.part;
        W.slots = a.slots; W.slot_bytes = a.slot_bytes; W.full = bar_full(a);
        W.in_stage = sm0 + a.off_ring + J.in_stage + g * kChunkBytes + t * 16;
        W.scales = sm0 + G.off_scale + J.scales + g * G.ngrp * 2; W.scale_hi = 16 * G.ngrp;
        W.x = sm0 + a.off_x + (kInt ? t * 32 + (g & 1) * 16 : t * 16); W.zero = sm0 + a.off_zero; W.cx = sm0 + a.off_corr;
        const uint32_t empty_scales = bar_sempty(a, ph);
        float* const red0 = reinterpret_cast<float*>(sm + a.off_red);
        // the rows' K-parts meet in neighbouring lanes: 1 << ks threads a row
        const int ks = G.ks, row = tid >> ks, part = tid & ((1 << ks) - 1);
        const int red_at = (part * G.nt + (row >> 4)) * kStepRed + (row & 15), red_up = G.mt == 2 ? G.rt * kStepRed : 0;
#pragma unroll 1
        for (int j = 0; j < nb; ++j) {
            const int blk = (int)(blockIdx.x + j * gridDim.x);
            int mat = 0, row0 = blk * G.brows, rows = 16;
            // what the threads that finish the rows need, fetched ahead as well
            __half b0 = __half(0), b1 = __half(0), res = __half(0);
            __half *out0 = nullptr, *cache = nullptr;
            uint2* word = nullptr;
            float2 cs = make_float2(1.f, 0.f);
            if (ph == SP_QKV) {
                qkv_tile(a, blk, mat, row0);
                if (row < 16) {
                    const __half* bp = at_layer(a, a.bias[mat], l) + row0 + row;
                    b0 = __ldg(bp); b1 = __ldg(bp + HD / 2);
                    const int rr = row0 + row, head = rr / HD, d = rr - head * HD, hh = head + (mat == 0 ? 0 : mat == 1 ? a.n_heads : a.n_heads + a.n_kv);
                    word = a.w_qkv + hh * (HD / 2) + d;
                    if (mat < 2) cs = reinterpret_cast<const float2*>(sm + a.off_rope)[j * 16 + row];
                    if (mat > 0) cache = (mat == 1 ? a.kc : a.vc) + (((size_t)l * a.n_kv + head) * a.max_seq + range(a).pos) * HD + d;
                    if (last) out0 = (mat == 0 ? a.q : mat == 1 ? a.k : a.v) + rr;
                }
            } else {
                rows = min(G.brows, G.rows - row0);
                if (row < rows) {
                    word = (ph == SP_O ? a.w_x1 : ph == SP_MLP ? a.w_h : a.w_x2) + (row0 + row) / 2;
                    if (ph != SP_MLP) res = reinterpret_cast<const __half*>(sm + a.off_res)[j * G.brows + row];
                    if (last && ph != SP_O) out0 = (ph == SP_MLP ? a.gate : a.x) + row0 + row;
                }
            }
            if (j == 0) {
                if (kInt) step_wait(bar_sfull(a, ph), l & 1, 2u);
                if (kInt && ph == SP_DOWN && a.staged_h) stage_groups(a.w_h, G.ngrp, seq);
                else {
                    const uint2* src = ph == SP_QKV ? a.w_x2 : ph == SP_O ? a.w_att : ph == SP_MLP ? a.w_x1 : a.w_h;
                    const __half* norm = ph == SP_QKV ? at_layer(a, a.norm[0], l) : ph == SP_MLP ? at_layer(a, a.norm[1], l) : nullptr;
                    stage_vec(src, ph == SP_QKV && l == 0 ? a.x : nullptr, norm, G.K, ph == SP_QKV ? seq - 1 : seq);
                }
            }
            float tot[2];
            block_sums(W, R, W.scales + j * G.scale_bytes, tot);
            float* red = red0 + R.red * (kStepWarps * kStepRed);
            R.red ^= 1u;
            if (t == 0) { red[warp * kStepRed + g] = tot[0]; red[warp * kStepRed + g + 8] = tot[1]; }
            consumer_sync(kStepConsumers);
            if (kInt && j == nb - 1 && tid == kStepConsumers - 1) mbar_arrive(empty_scales);       // all warps have read the scales
            if (warp * 32 >= rows << ks) continue;                  // (whole warps stay: rows meet in shuffles)
            const bool in = part < W.kp && row < rows, live = part == 0 && row < rows;
            float v0 = in ? red[red_at] : 0.f, v1 = in ? red[red_at + red_up] : 0.f;
            const float inv = kInt && (ph == SP_QKV || ph == SP_MLP) ? norm_scale(a) : 1.f;
            if (ks) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float y0 = __shfl_xor_sync(0xffffffffu, v0, 1 << i), y1 = __shfl_xor_sync(0xffffffffu, v1, 1 << i);
                    if (i < ks) { v0 += y0; v1 += y1; }
                }
            }
            v0 *= inv; v1 *= inv;
            __half h = __half(0);
            if (ph == SP_QKV) {
                // bias, one rounding, rotation from the rounded values (as EPI_QKV of gemv.cuh); v: angle 0
                if (live) {
                    const float f0 = __half2float(__float2half(v0 + __half2float(b0))), f1 = __half2float(__float2half(v1 + __half2float(b1)));
                    const __half o0 = __float2half(f0 * cs.x - f1 * cs.y), o1 = __float2half(f1 * cs.x + f0 * cs.y);
                    st_word(word, (uint32_t)__half_as_ushort(o0) | (uint32_t)__half_as_ushort(o1) << 16, seq);
                    if (cache) { cache[0] = o0; cache[HD / 2] = o1; }
                    if (out0) { out0[0] = o0; out0[HD / 2] = o1; }
                }
                continue;
            }
            if (ph == SP_MLP) {
                const float sig = __fdividef(1.0f, 1.0f + __expf(-v0));
                h = __float2half(v0 * sig * v1);
            } else {
                h = __float2half(__half2float(res) + v0);
                if (live) reinterpret_cast<__half*>(sm + a.off_res)[j * G.brows + row] = h;
            }
            if (live && out0) *out0 = h;
            if (kInt && ph == SP_MLP && a.staged_h) {               // a block is a whole group (128 rows)
                __half* hb = reinterpret_cast<__half*>(sm + a.off_hbuf);
                hb[tid] = h;
                asm volatile("bar.sync 2, 128;" ::: "memory");
                if (warp == 0) {
                    unsigned char* xd = sm + a.off_hbuf + 256;
                    const uint2 v = reinterpret_cast<const uint2*>(hb)[lane];
                    const float2 f0 = __half22float2(*reinterpret_cast<const __half2*>(&v.x)), f1 = __half22float2(*reinterpret_cast<const __half2*>(&v.y));
                    const float f[4] = {f0.x, f0.y, f1.x, f1.y};
                    digits_of_group(f, lane, xd, reinterpret_cast<int2*>(xd + 256));
                    __syncwarp();
                    const uint2 d = reinterpret_cast<const uint2*>(xd)[lane];
                    st_word2(a.w_h + (size_t)blk * 64 + 2 * lane, d.x, d.y, seq);
                    if (lane == 0) { const uint2 e = reinterpret_cast<const uint2*>(xd)[32]; st_word2(a.w_h + (size_t)(a.inter / kGroup) * 64 + 2 * blk, e.x, e.y, seq); }
                }
            } else {
                const uint32_t u = __half_as_ushort(h), nx = __shfl_down_sync(0xffffffffu, u, 1 << ks);
                if (live && !(row & 1)) st_word(word, u | nx << 16, seq);
            }
        }
    }

    // 32 keys of a stage (attn_tile32's arithmetic, one softmax update for all).  The rows lie as the copy's 128-byte swizzle leaves them: 64 columns of row r make 128 bytes, its 16-byte
    // chunk j at place j ^ (r & 7).  Lane g of a fragment takes key (and chunk of V) perm(g) instead of g, so that the eight lanes of a quarter-warp, two g by four t, read eight
    // different places; of rows as they are cached, 256 bytes apart, 2 lanes of K and 4 of V met in a bank.  n: keys that exist.
    static __device__ __forceinline__ int perm(int g) { return g >> 1 | (g & 1) << 2; }
    static __device__ __forceinline__ void tile(AttnState<HD>& st, uint32_t sQ, uint32_t sK, uint32_t sV, int n, float scale, int g, int t) {
        constexpr int NCH = HD / 32, NC = HD / 64, NMT = HD / 16, COLS = kKeys * 128;
        const uint32_t k0 = sK + perm(g) * 128 + ((t ^ perm(g)) << 4), k1 = sK + perm(g) * 128 + ((4 + t ^ perm(g)) << 4);
        const uint32_t v0 = sV + t * 128 + ((t ^ perm(g)) << 4), v1 = sV + (t + 4) * 128 + ((t + 4 ^ perm(g)) << 4);
        float sc[4][4];                      // block b = keys 8b .. 8b + 7: the lane holds head g, keys 8b + t and 8b + t + 4 in [0], [1]
#pragma unroll
        for (int b = 0; b < 4; ++b) sc[b][0] = sc[b][1] = sc[b][2] = sc[b][3] = 0.f;
#pragma unroll
        for (int i = 0; i < NCH; ++i) {
            const uint4 qf = lds128(sQ + i * 64);
            uint4 kf[4];
#pragma unroll
            for (int b = 0; b < 4; ++b) kf[b] = lds128((i & 1 ? k1 : k0) + (i >> 1) * COLS + b * 1024);
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                mma16816(sc[b], qf.x, 0u, qf.y, 0u, kf[b].x, kf[b].y);
                mma16816(sc[b], qf.z, 0u, qf.w, 0u, kf[b].z, kf[b].w);
            }
        }
        float mx = -INFINITY;
#pragma unroll
        for (int b = 0; b < 4; ++b)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                sc[b][j] = 8 * b + t + 4 * j < n ? sc[b][j] * scale : -INFINITY;
                mx = fmaxf(mx, sc[b][j]);
            }
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        const float m_new = fmaxf(st.m_run, mx), alpha = ex2(st.m_run - m_new);       // finite: key 0 exists
        float psum = 0.f;
        uint32_t pb[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const float p0 = ex2(sc[b][0] - m_new), p1 = ex2(sc[b][1] - m_new);
            psum += p0 + p1;
            pb[b] = pack_h2(p0, p1);
        }
        st.l_run = st.l_run * alpha + psum;
        st.m_run = m_new;
        if (__any_sync(0xffffffffu, alpha != 1.0f)) {
            const float al = __shfl_sync(0xffffffffu, alpha, 8 * t), ah = __shfl_sync(0xffffffffu, alpha, 8 * t + 4);
#pragma unroll
            for (int m = 0; m < NMT; ++m) { st.o[m][0] *= al; st.o[m][1] *= ah; st.o[m][2] *= al; st.o[m][3] *= ah; }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {        // keys 16h .. 16h + 15: one k-step of P.V, in the order of the scores
            // 64 columns at a time: all of a row's fragments at once are 16 registers more, and what other phases keep in registers then spills (fp16 with heads of 128, us a step with 40 and with 0
            // bytes spilled: eight layers of 1.5B at 3000 keys 356 -> 324, six of 3B 371 -> 340, four of 7B 540 -> 519, where the separate launches take 346, 355 and 518).
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                uint4 vv[4];
#pragma unroll
                for (int r = 0; r < 4; ++r) vv[r] = lds128((r & 1 ? v1 : v0) + c * COLS + h * 2048 + (r >> 1) * 1024);
                if (n < 16 * h + 16) {       // a row that does not exist may hold anything: its weight is 0, and 0 times that must be 0
#pragma unroll
                    for (int r = 0; r < 4; ++r)
                        if (16 * h + 8 * (r >> 1) + t + 4 * (r & 1) >= n) vv[r] = make_uint4(0u, 0u, 0u, 0u);
                }
#pragma unroll
                for (int ep = 0; ep < 4; ++ep) {
                    const uint32_t wA = u4c(vv[0], ep), wB = u4c(vv[1], ep), wC = u4c(vv[2], ep), wD = u4c(vv[3], ep);
                    mma16816(st.o[c * 4 + ep], prmt(wA, wB, 0x5410), prmt(wA, wB, 0x7632), prmt(wC, wD, 0x5410), prmt(wC, wD, 0x7632), pb[2 * h], pb[2 * h + 1]);
                }
            }
        }
    }

    // Attention over this CTA's key range for the query heads of its KV head.
    static __device__ __forceinline__ void attend(uint32_t seq, bool last, StepRing& R) {
        constexpr int NMT = HD / 16;
        const StepCore& a = core();
        unsigned char* sm = step_smem;
        const uint32_t sm0 = smem_u32(step_smem);
        const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
        const Range& r = range(a);
        const int grp = a.grp;
        unsigned char* qs = sm + a.off_q;                            // rows of q; the step's own key and value as row 0 of a stage of their own (V 128 bytes behind K)
        {
            const int nq = grp * HD / 4, j = tid - kStepConsumers / 2;           // pairs of words: of q by the first half of the threads, of k and v by the next ones
            const bool isq = tid < nq, isk = j < HD / 4;
            if (isq || (r.own && j >= 0 && j < HD / 2)) {
                const int u = isq ? tid : isk ? j : j - HD / 4;                     // pair inside the heads' / the head's words
                const int h0 = isq ? r.kvh * grp : (isk ? a.n_heads : a.n_heads + a.n_kv) + r.kvh;
                uint32_t v[2];
                poll_words<1>(a.w_qkv + h0 * (HD / 2) + 2 * u, 0, seq, v);
                const int hl = 2 * u / (HD / 2), d = 2 * u - hl * (HD / 2);
                unsigned char* o = isq ? qs + hl * kRowQ + d * 2 : sm + a.off_cur + (isk ? 0 : 128) + d * 2;
                *reinterpret_cast<uint32_t*>(o) = prmt(v[0], v[1], 0x5410);
                *reinterpret_cast<uint32_t*>(o + (isq || HD == 64 ? HD : kKeys * 128)) = prmt(v[0], v[1], 0x7632);
            }
        }
        consumer_sync(kStepConsumers);
        const uint32_t sQ = g < grp ? sm0 + a.off_q + g * kRowQ + t * 16 : sm0 + a.off_zero;        // (heads that do not exist: zeros)
        AttnState<HD> st;
        st.reset();
        // A warp waits for its own stages only and lets the others go at once.  That is safe with 32 barriers and at most 16 slots: it is at most 15 stages past one that it saw full, before
        // which all but the last `slots` stages had been let go by all warps, so no warp is still to arrive at the barrier's use before.
        const int nstage = r.nstage, keys = r.t1c - r.t0, ns = nstage + r.own;                             // the step's own key and value are one more stage, of one key, outside the ring
        const uint32_t ring = a.off_ring, slots = a.slots, slot_bytes = a.slot_bytes, full = bar_full(a);
        
#pragma unroll 1
        for (int sn = 0; sn < ns; ++sn) {                            // a warp takes 32 keys of its stages
            const bool in_ring = sn < nstage;
            if ((sn & (kStepWarps / kPer - 1)) == warp / kPer) {
                const int skip = 32 * (warp & (kPer - 1)), n = (in_ring ? keys - sn * kKeys : 1) - skip;
                const uint32_t sK = sm0 + (in_ring ? ring + R.slot * slot_bytes : a.off_cur) + skip * 128;
                if (in_ring) step_wait(full + R.bar(), R.par(), 6u);
                if (n > 0) tile(st, sQ, sK, sK + (in_ring ? kHalf : 128), n, a.scale_log2, g, t);
            }
            if (in_ring) {
                __syncwarp();
                if (lane == 0) mbar_arrive(full + kStepBars * 8 + R.bar());
                R.next(slots);
            }
        }
        // Merge the warps' states in the area of the staged vectors, which no product reads now: the upper eight into the lower ones, those in one go.
        int nw = min(kPer * ns, kStepWarps);
        if (nw > 8) {
            constexpr int per = NMT * 512 + 256;
            unsigned char* b = sm + a.off_x + (warp & 7) * per;
            if (warp >= 8 && warp < nw) {
#pragma unroll
                for (int mt = 0; mt < NMT; ++mt) reinterpret_cast<float4*>(b)[mt * 32 + lane] = make_float4(st.o[mt][0], st.o[mt][1], st.o[mt][2], st.o[mt][3]);
                reinterpret_cast<float2*>(b + NMT * 512)[lane] = make_float2(st.m_run, st.l_run);
            }
            consumer_sync(kStepConsumers);
            if (warp + 8 < nw) {
                const float2 ml = reinterpret_cast<const float2*>(b + NMT * 512)[lane];
                const float mn = fmaxf(st.m_run, ml.x);
                const float fa = st.m_run == -INFINITY ? 0.f : ex2(st.m_run - mn), fb = ml.x == -INFINITY ? 0.f : ex2(ml.x - mn);
                st.l_run = st.l_run * fa + ml.y * fb; st.m_run = mn;
                const float fa0 = __shfl_sync(0xffffffffu, fa, 8 * t), fa1 = __shfl_sync(0xffffffffu, fa, 8 * t + 4);
                const float fb0 = __shfl_sync(0xffffffffu, fb, 8 * t), fb1 = __shfl_sync(0xffffffffu, fb, 8 * t + 4);
#pragma unroll
                for (int mt = 0; mt < NMT; ++mt) {
                    const float4 o = reinterpret_cast<const float4*>(b)[mt * 32 + lane];
                    st.o[mt][0] = st.o[mt][0] * fa0 + o.x * fb0; st.o[mt][1] = st.o[mt][1] * fa1 + o.y * fb1;
                    st.o[mt][2] = st.o[mt][2] * fa0 + o.z * fb0; st.o[mt][3] = st.o[mt][3] * fa1 + o.w * fb1;
                }
            }
            consumer_sync(kStepConsumers);
            nw = 8;
        }
        // fragments as they are: [warp][row tile][lane], columns = heads 2t and 2t + 1; a thread merges one lane's place of all warps
        unsigned char* frag = sm + a.off_x;
        float2* ml_all = reinterpret_cast<float2*>(frag + 8 * NMT * 512);          // [warp][head]
        if (warp < nw) {
            st.l_run += __shfl_xor_sync(0xffffffffu, st.l_run, 1);
            st.l_run += __shfl_xor_sync(0xffffffffu, st.l_run, 2);
            if (t == 0) ml_all[warp * kMaxGroup + g] = make_float2(st.m_run, st.l_run);
#pragma unroll
            for (int mt = 0; mt < NMT; ++mt) reinterpret_cast<float4*>(frag)[(warp * NMT + mt) * 32 + lane] = make_float4(st.o[mt][0], st.o[mt][1], st.o[mt][2], st.o[mt][3]);
        }
        const int slot0 = (r.kvh * grp + 2 * t) * a.nsplit + r.split, nsplit = a.nsplit;
        consumer_sync(kStepConsumers);
        if (warp < NMT) {
            float4 ml[8];
            float M0 = -INFINITY, M1 = -INFINITY, L0 = 0.f, L1 = 0.f;
#pragma unroll
            for (int w = 0; w < 8; ++w) {
                ml[w] = make_float4(-INFINITY, 0.f, -INFINITY, 0.f);
                if (w < nw) ml[w] = *reinterpret_cast<const float4*>(ml_all + w * kMaxGroup + 2 * t);
                M0 = fmaxf(M0, ml[w].x); M1 = fmaxf(M1, ml[w].z);
            }
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int w = 0; w < 8; ++w)
                if (w < nw) {
                    const float4 o = reinterpret_cast<const float4*>(frag)[(w * NMT + warp) * 32 + lane];
                    const float f0 = ml[w].x == -INFINITY ? 0.f : ex2(ml[w].x - M0), f1 = ml[w].z == -INFINITY ? 0.f : ex2(ml[w].z - M1);
                    acc.x += o.x * f0; acc.y += o.y * f1; acc.z += o.z * f0; acc.w += o.w * f1;
                    L0 += ml[w].y * f0; L1 += ml[w].w * f1;
                }
            const int d = ((warp >> 2) * 8 + perm(g)) * 8 + 2 * (warp & 3);
            if (r.nne == 1) {                                            // the only range: nothing is left to merge
                const float i0 = __frcp_rn(L0), i1 = __frcp_rn(L1);
                const __half2 h0 = __floats2half2_rn(acc.x * i0, acc.z * i0), h1 = __floats2half2_rn(acc.y * i1, acc.w * i1);
                const int at = (r.kvh * grp + 2 * t) * HD + d;
                if (2 * t < grp) { st_word(a.w_att + at / 2, *reinterpret_cast<const uint32_t*>(&h0), seq); if (last) *reinterpret_cast<__half2*>(a.att + at) = h0; }
                if (2 * t + 1 < grp) { st_word(a.w_att + (at + HD) / 2, *reinterpret_cast<const uint32_t*>(&h1), seq); if (last) *reinterpret_cast<__half2*>(a.att + at + HD) = h1; }
                return;
            }
            if (2 * t < grp) {
                st_word2(a.w_part + (size_t)slot0 * HD + d, __float_as_uint(acc.x), __float_as_uint(acc.z), seq);
                if (warp == 0 && g == 0) st_word2(a.w_ml + slot0 * 2, __float_as_uint(M0), __float_as_uint(L0), seq);
            }
            if (2 * t + 1 < grp) {
                st_word2(a.w_part + (size_t)(slot0 + nsplit) * HD + d, __float_as_uint(acc.y), __float_as_uint(acc.w), seq);
                if (warp == 0 && g == 0) st_word2(a.w_ml + (slot0 + nsplit) * 2, __float_as_uint(M1), __float_as_uint(L1), seq);
            }
        }
    }

    // Merge of a head's partials: warp w takes splits w, w + 16, ..., a lane HD / 32 columns.
    static __device__ __forceinline__ void fold(int l, uint32_t seq, int head) {
        constexpr int ND = HD / 32, NP = ND / 2;
        const StepCore& a = core();
        const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
        const int nne = range(a).nne;
        float M = -INFINITY, L = 0.f, acc[ND] = {};
#pragma unroll 1
        for (int s = warp; s < nne; s += kStepWarps) {
            const int slot = head * a.nsplit + s;
            uint32_t v[2 * NP + 2];                                  // the values, then maximum and sum, in one round trip
            poll_words<NP, 1>(a.w_part + (size_t)slot * HD + lane * ND, 2, a.w_ml + slot * 2, seq, v);
            const float m = __uint_as_float(v[2 * NP]), Mn = fmaxf(M, m);
            const float fo = M == -INFINITY ? 0.f : ex2(M - Mn), fn = m == -INFINITY ? 0.f : ex2(m - Mn);
#pragma unroll
            for (int k = 0; k < ND; ++k) acc[k] = acc[k] * fo + __uint_as_float(v[k]) * fn;
            L = L * fo + __uint_as_float(v[2 * NP + 1]) * fn; M = Mn;
        }
        consumer_sync(kStepConsumers);                               // every thread has left the merge of this CTA's own partial
        float* o_w = reinterpret_cast<float*>(step_smem + a.off_x);
        float* ml_w = o_w + kStepWarps * HD;
#pragma unroll
        for (int k = 0; k < ND; ++k) o_w[warp * HD + lane * ND + k] = acc[k];
        if (lane == 0) { ml_w[2 * warp] = M; ml_w[2 * warp + 1] = L; }
        consumer_sync(kStepConsumers);
        if (tid < HD) {                                              // (a warp without a split left a maximum of minus infinity and zeros)
            float2 ml[kStepWarps];
            float Mx = -INFINITY, o = 0.f, Ls = 0.f;
#pragma unroll
            for (int w = 0; w < kStepWarps; ++w) { ml[w] = reinterpret_cast<const float2*>(ml_w)[w]; Mx = fmaxf(Mx, ml[w].x); }
#pragma unroll
            for (int w = 0; w < kStepWarps; ++w) {
                const float f = ml[w].x == -INFINITY ? 0.f : ex2(ml[w].x - Mx);
                o += o_w[w * HD + tid] * f;
                Ls += ml[w].y * f;
            }
            const __half h = __float2half(o * __frcp_rn(Ls));
            const uint32_t u = __half_as_ushort(h), nx = __shfl_down_sync(0xffffffffu, u, 1);
            if (!(tid & 1)) st_word(a.w_att + (head * HD + tid) / 2, u | nx << 16, seq);
            if (l == a.n_layers - 1) a.att[head * HD + tid] = h;
        }
    }
};

template <int Q, int HD>
__global__ void __launch_bounds__(kStepThreads, 1) step_layers_kernel(const __grid_constant__ StepArgs args) {
    using S = StepLayers<Q, HD>;
    const StepCore& a = args.c;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    pdl_launch_dependents();
    if (tid < (int)(sizeof(StepCore) / 4))
        reinterpret_cast<uint32_t*>(step_smem)[tid] = tid == (int)(offsetof(StepCore, started) / 4) ? cycles32() : tid == (int)(offsetof(StepCore, seq0) / 4) ? *a.epoch * kSeqPerStep : reinterpret_cast<const uint32_t*>(&a)[tid];
    if (tid == 0) {
#pragma unroll 1
        for (int i = 0; i < kStepBars; ++i) { mbar_init(S::bar_full(a) + i * 8, 1); mbar_init(S::bar_empty(a) + i * 8, kStepWarps); }
#pragma unroll 1
        for (int i = 0; i < SP_COUNT; ++i) { mbar_init(S::bar_sfull(a, i), 1); mbar_init(S::bar_sempty(a, i), 1); }
        mbar_fence_init();
        *reinterpret_cast<typename S::Range*>(step_smem + a.off_range) = S::make_range(a);
    }
    if (tid < 64) reinterpret_cast<uint32_t*>(step_smem + a.off_zero)[tid] = 0u;
    if (tid < SP_COUNT * kStepWarps) {
        const int ph = tid / kStepWarps, w = tid % kStepWarps;
        const StepGemv& G = a.g[ph];
        const int tile = w % G.nt, part = w / G.nt, m = tile / G.rt, r = tile - m * G.rt;
        S::job(a, ph, w) = typename S::Job{m * G.box_bytes + r * 16 * kChunkBytes, (m * G.brows + r * 16) * G.ngrp * 2, part < G.kp ? part : 1 << 30};
    }
    __syncthreads();
    // 640 threads are launched with 96 registers each, 61,440; 512 x 112 + 128 x 32 are as many
    if (warp >= kStepWarps) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
        if (warp == kStepWarps && lane == 0) {
            StepRing P{0u, 0u, 0u};
            const typename S::Range& rg = S::range(a);
            uint32_t scales = 0u;
#pragma unroll 1
            for (int i = 0; i < a.n_layers * SP_COUNT; ++i) {
                const int l = i / SP_COUNT, ph = i % SP_COUNT;
                if (ph == SP_O && !S::produce_kv(args, P, l, rg)) break;
                if (rg.nb[ph] && !S::produce_gemv(args, P, ph, l, rg.nb[ph], scales)) break;
            }
            S::land(a, P, scales);
            step_report(a.err);
        }
        return;
    }
    asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
    // this CTA's rows of the residual stream, and the rotation of its rows of q and k, which are the same in every layer
    {
        const StepGemv& G = a.g[SP_O];
        __half* res = reinterpret_cast<__half*>(step_smem + a.off_res);
#pragma unroll 1
        for (int j = 0; j < S::range(a).nb[SP_O]; ++j) {
            const int row = (int)(blockIdx.x + j * gridDim.x) * G.brows + tid;
            if (tid < G.brows && row < a.dim) res[j * G.brows + tid] = __ldcg(a.x + row);
        }
        float2* rope = reinterpret_cast<float2*>(step_smem + a.off_rope);
#pragma unroll 1
        for (int j = 0; j < S::range(a).nb[SP_QKV]; ++j) {
            int mat, row;
            S::qkv_tile(a, (int)(blockIdx.x + j * gridDim.x), mat, row);
            if (tid < 16) { float c, s; rope_cs((row + tid) % HD, HD, S::range(a).pos, a.theta, 1, &c, &s); rope[j * 16 + tid] = make_float2(c, s); }
        }
        // Both arrays are written by the first warps and read by the threads that finish a row, of up to four warps, before any other barrier: the rotation when layer 0's
        // q/k/v phase begins, the residual in a CTA whose first work is the output projection.
        consumer_sync(kStepConsumers);
    }
    StepRing R{0u, 0u, 0u};
    // One copy of the code for the four matrix phases: it has to fit the instruction cache.
#pragma unroll 1
    for (int i = 0; i < a.n_layers * SP_COUNT; ++i) {
        const int l = i / SP_COUNT, ph = i % SP_COUNT;
        const uint32_t seq = S::core().seq0 + (uint32_t)l + 1u;
        if (ph == SP_QKV && warp == kStepWarps - 1 && (int)blockIdx.x == l % (int)gridDim.x && l + 1 < a.n_layers) {      // the small tensors of the layer ahead come to L2 before their first use
#pragma unroll 1
            for (int k = 0; k < 5; ++k) {
                const __half* p = S::at_layer(a, k < 2 ? a.norm[k] : a.bias[k - 2], l + 1);
                const int n = k < 2 ? a.dim : k == 2 ? a.n_heads * HD : a.n_kv * HD;
#pragma unroll 1
                for (int o = lane * 64; o < n; o += 32 * 64) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + o));
            }
        }
        const typename S::Range& rg = S::range(a);
        if (ph == SP_O) {
            if (rg.any) S::attend(seq, l == a.n_layers - 1, R);
            if (rg.fold_head >= 0) S::fold(l, seq, rg.fold_head);
            // Both end with a few warps reading the area that the output projection's input is staged in, whose first words may be other heads'.
            if (rg.any || rg.fold_head >= 0) consumer_sync(kStepConsumers);
        }
        if (rg.nb[ph]) S::gemv(ph, rg.nb[ph], l, seq, R);
    }
    step_report(a.err);
}

template <int Q>
int launch_step_layers_q(const StepArgs& a, const LaunchCfg& cfg) {
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(cfg.sm_count); lc.blockDim = dim3(kStepThreads); lc.dynamicSmemBytes = a.c.smem; lc.stream = cfg.stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;        // its CTAs wait for one another
    at[0].val.cooperative = 1;
    lc.attrs = at; lc.numAttrs = 1;
    auto* kernel = a.c.hd == 128 ? step_layers_kernel<Q, 128> : step_layers_kernel<Q, 64>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, a.c.smem);
    if (e != cudaSuccess) return (int)e;
    return (int)cudaLaunchKernelEx(&lc, kernel, a);
}

}  // namespace cq
