// The batched-token GEMM kernel and its launcher (see prefill_gemm.cuh for the design).
#include "prefill_gemm.cuh"
#include "stack_dev.cuh"
#include "tcgen05.cuh"

#include <algorithm>
#include <cmath>

namespace cq {

// Shared-memory matrix descriptor of a K-major tile in the 128-byte-swizzled canonical layout: rows of 128 bytes,
// eight-row groups 1024 bytes apart.  Fields: start address >> 4 [0,14), leading byte offset >> 4 [16,30) (unused by
// swizzled K-major tiles), stride byte offset >> 4 [32,46), descriptor version 1 [46,48), layout type 2 = 128-byte
// swizzle [61,64).
__device__ __forceinline__ uint64_t umma_desc(uint32_t smem_addr) {
    return (uint64_t)((smem_addr >> 4) & 0x3fffu) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}

// W weights (32 or 16: one half or one quarter of a row's K block) -> W / 8 sixteen-byte chunks of fp16(q * scale),
// stored at the row's swizzled places.  raw: shared address of the part's bytes; brow: the row in the B tile; chunk0:
// the part's first chunk.
template <int Q, int W>
__device__ __forceinline__ void convert_part(uint32_t raw, uint32_t brow, int sw, int chunk0, __half2 sc2) {
    if (Q == Q_I4) {
        // two's-complement nibbles, element 2p in the low nibble of byte p: (n ^ 8) | 0x6400 is fp16(1024 + q + 8)
        const __half2 off = __floats2half2_rn(1032.f, 1032.f);
        uint32_t w4[4];
        if (W == 32) { const uint4 rw = lds128(raw); w4[0] = rw.x; w4[1] = rw.y; w4[2] = rw.z; w4[3] = rw.w; }
        else { asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(w4[0]), "=r"(w4[1]) : "r"(raw)); w4[2] = w4[3] = 0u; }
#pragma unroll
        for (int i = 0; i < W / 8; ++i) {
            const uint32_t w = w4[i];
            uint32_t t[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t u = ((w >> (4 * j)) & 0x000f000fu) ^ 0x64086408u;          // (element j, element j + 4)
                const __half2 hv = __hmul2(__hsub2(*reinterpret_cast<const __half2*>(&u), off), sc2);
                t[j] = *reinterpret_cast<const uint32_t*>(&hv);
            }
            uint4 o;
            o.x = __byte_perm(t[0], t[1], 0x5410); o.y = __byte_perm(t[2], t[3], 0x5410);
            o.z = __byte_perm(t[0], t[1], 0x7632); o.w = __byte_perm(t[2], t[3], 0x7632);
            sts128(brow + (((chunk0 + i) ^ sw) << 4), o);
        }
    } else {
        // signed bytes: (b ^ 0x80) under a 0x64 exponent byte is fp16(1024 + b + 128)
        const __half2 off = __floats2half2_rn(1152.f, 1152.f);
#pragma unroll
        for (int h = 0; h < W / 16; ++h) {
            const uint4 rw = lds128(raw + h * 16);
            const uint32_t w4[4] = {rw.x, rw.y, rw.z, rw.w};
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                uint32_t t[4];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const uint32_t x = w4[2 * i + j] ^ 0x80808080u;
                    const uint32_t lo = __byte_perm(x, 0x64646464u, 0x4140), hi = __byte_perm(x, 0x64646464u, 0x4342);
                    const __half2 a = __hmul2(__hsub2(*reinterpret_cast<const __half2*>(&lo), off), sc2);
                    const __half2 b = __hmul2(__hsub2(*reinterpret_cast<const __half2*>(&hi), off), sc2);
                    t[2 * j] = *reinterpret_cast<const uint32_t*>(&a); t[2 * j + 1] = *reinterpret_cast<const uint32_t*>(&b);
                }
                sts128(brow + (((chunk0 + h * 2 + i) ^ sw) << 4), make_uint4(t[0], t[1], t[2], t[3]));
            }
        }
    }
}

// A warp's 32 x 32 block of partial sums into another CTA's shared memory: four columns of all lanes are 512 contiguous bytes.
__device__ __forceinline__ void push_block(uint32_t remote, int lane, const float (&v)[32]) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
        asm volatile("st.shared::cluster.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(remote + (uint32_t)((i * 32 + lane) * 16)), "f"(v[4 * i]), "f"(v[4 * i + 1]), "f"(v[4 * i + 2]), "f"(v[4 * i + 3]) : "memory");
}
__device__ __forceinline__ void add_block(uint32_t local, int lane, float (&v)[32]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint4 o = lds128(local + (uint32_t)((i * 32 + lane) * 16));
        v[4 * i] += __uint_as_float(o.x); v[4 * i + 1] += __uint_as_float(o.y); v[4 * i + 2] += __uint_as_float(o.z); v[4 * i + 3] += __uint_as_float(o.w);
    }
}

// Eight gate and eight up columns in turn -> clamped gated unit, one row's 32 columns.
__device__ __forceinline__ void pf_store_glu(const PfGemmArgs& a, const float (&v)[32], int token, int r, int R) {
    __nv_bfloat16* dst = a.out_b + (size_t)token * a.ldo + r / 2;
#pragma unroll
    for (int i = 0; i < 32; i += 16)
        if (r + i < R) {
            uint32_t o[4];
#pragma unroll
            for (int k = 0; k < 4; ++k)
                o[k] = pack_bf(clamped_glu_f(v[i + 2 * k], v[i + 8 + 2 * k], a.c0, a.c1), clamped_glu_f(v[i + 2 * k + 1], v[i + 9 + 2 * k], a.c0, a.c1));
            *reinterpret_cast<uint4*>(dst + i / 2) = make_uint4(o[0], o[1], o[2], o[3]);
        }
}

// What the epilogue of four columns reads from memory: the residual, the stream it adds to, a table row.
template <int MODE>
__device__ __forceinline__ uint4 pf_other(const PfGemmArgs& a, int token, int col, int r) {
    uint4 o = make_uint4(0u, 0u, 0u, 0u);
    auto two = [&](const void* p) { const uint2 t = *reinterpret_cast<const uint2*>(p); o.x = t.x; o.y = t.y; };
    if (MODE == PF_ADD_F32) o = *reinterpret_cast<const uint4*>(a.out_f + (size_t)token * a.ldo + col);
    else if (MODE == PF_DECAY_F32) o = *reinterpret_cast<const uint4*>(a.bias_f + col);
    else if (MODE == PF_BF16_GELU_SIDE) {
        const __nv_bfloat16* e = a.side + (size_t)a.tokens[token] * a.side_pitch + r;
        uint32_t w[4];                // a table row starts at any element
#pragma unroll
        for (int j = 0; j < 4; ++j) w[j] = r + j < a.side_dim ? (uint32_t)__bfloat16_as_ushort(e[j]) : 0u;
        o.x = w[0] | (w[1] << 16); o.y = w[2] | (w[3] << 16);
    } else if (MODE == PF_RESID) two(a.out_h + (size_t)token * a.ldo + col);
    else if (MODE == PF_OUT_F16) { if (a.bias) two(a.bias + col); }
    return o;
}
// Four sums of one token -> the output's columns col .. col + 3 (row r .. of their matrix).
template <int MODE>
__device__ __forceinline__ void pf_finish(const PfGemmArgs& a, float4 v, uint4 o, int token, int col, int r) {
    const size_t at = (size_t)token * a.ldo + col;
    const float4 f = make_float4(__uint_as_float(o.x), __uint_as_float(o.y), __uint_as_float(o.z), __uint_as_float(o.w));
    float4* const out = reinterpret_cast<float4*>(a.out_f + at);
    if (MODE == PF_OUT_F32) *out = v;
    else if (MODE == PF_ADD_F32) *out = make_float4(fmaf(a.c0, v.x, f.x), fmaf(a.c0, v.y, f.y), fmaf(a.c0, v.z, f.z), fmaf(a.c0, v.w, f.w));
    else if (MODE == PF_CAP_F32) *out = make_float4(a.c0 * tanhf(v.x / a.c0), a.c0 * tanhf(v.y / a.c0), a.c0 * tanhf(v.z / a.c0), a.c0 * tanhf(v.w / a.c0));
    else if (MODE == PF_DECAY_F32) *out = make_float4(expf(-expf(v.x + f.x)), expf(-expf(v.y + f.y)), expf(-expf(v.z + f.z)), expf(-expf(v.w + f.w)));
    else if (MODE == PF_RESID || MODE == PF_OUT_F16) {
        const float2 lo = __half22float2(*reinterpret_cast<const __half2*>(&o.x)), hi = __half22float2(*reinterpret_cast<const __half2*>(&o.y));
        *reinterpret_cast<uint2*>(a.out_h + at) = make_uint2(pack_h2(lo.x + v.x, lo.y + v.y), pack_h2(hi.x + v.z, hi.y + v.w));
    } else {
        float w[4] = {v.x, v.y, v.z, v.w};
        if (MODE == PF_BF16_RELU2) {
#pragma unroll
            for (int k = 0; k < 4; ++k) { w[k] = fmaxf(w[k], 0.f); w[k] *= w[k]; }
        } else if (MODE == PF_BF16_GELU_SIDE) {
            const uint32_t e[2] = {o.x, o.y};
#pragma unroll
            for (int k = 0; k < 4; ++k)
                w[k] = r + k < a.side_dim ? gelu_tanh_f(w[k]) * __uint_as_float(k & 1 ? e[k >> 1] & 0xffff0000u : e[k >> 1] << 16) : 0.f;
        }
        *reinterpret_cast<uint2*>(a.out_b + at) = make_uint2(pack_bf(w[0], w[1]), pack_bf(w[2], w[3]));
    }
}
// A warp's unit of an epilogue: 32 tokens from t0 on x 32 rows of the matrix from r on.  sums(v, false) gives a lane, which is a token, its 32
// sums, sums(v, true) those of the up rows beside them (SwiGLU).  One instance per mode, chosen once: with all modes in one
// loop, its unrolled copies of tanhf, expf and the rest lay between the instructions that ran, and a CTA, which runs them a few
// times only, waited for instructions (gate/up 4864 x 896, fp16, 640 tokens: 19.0 us, with this 16.7; bfloat16 13,440 x 1536, 1999 tokens: 85.8, with this 73.7).
template <int MODE, class Sums>
__device__ __forceinline__ void pf_unit(const PfGemmArgs& a, uint32_t stage, int lane, int t0, int r, int R, int coff, Sums sums) {
    if (MODE == PF_SWIGLU || MODE == PF_BF16_GLU) {
        // a lane's columns are 64 bytes side by side: they go out as they are
        float v[32];
        sums(v, false);
        if (MODE == PF_BF16_GLU) { if (t0 + lane < a.T) pf_store_glu(a, v, t0 + lane, r, R); return; }
        float u[32];
        sums(u, true);
        const int t = t0 + lane;
        __half* dst = a.out_h + (size_t)t * a.ldo + r;
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = v[i] * __fdividef(1.0f, 1.0f + __expf(-v[i])) * u[i];
#pragma unroll
        for (int i = 0; i < 32; i += 8)
            if (t < a.T && r + i < R)
                *reinterpret_cast<uint4*>(dst + i) = make_uint4(pack_h2(v[i], v[i + 1]), pack_h2(v[i + 2], v[i + 3]), pack_h2(v[i + 4], v[i + 5]), pack_h2(v[i + 6], v[i + 7]));
        return;
    }
    // Sums leave tensor memory with a token per lane; they go through 4 KB of shared memory (rows of 128 bytes, 16-byte
    // chunks swizzled by row) so that a warp's loads and stores cover whole lines: eight lanes a token, four columns each.
    constexpr bool kEarly = MODE == PF_RESID || MODE == PF_OUT_F16 || MODE == PF_ADD_F32;      // read for the whole unit before the sums are there
    constexpr int kUnroll = MODE == PF_CAP_F32 || MODE == PF_DECAY_F32 || MODE == PF_BF16_GELU_SIDE ? 1 : 8;
    const int lr = lane >> 3, lc = lane & 7, rc = r + lc * 4, col = coff + rc;
    uint4 other[8];
    if (kEarly)
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int token = t0 + i * 4 + lr;
            other[i] = token < a.T && rc < R ? pf_other<MODE>(a, token, col, rc) : make_uint4(0u, 0u, 0u, 0u);
        }
    float v[32];
    sums(v, false);
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 8; ++i)
        sts128(stage + (uint32_t)(lane * 128 + ((i ^ (lane & 7)) << 4)), make_uint4(__float_as_uint(v[4 * i]), __float_as_uint(v[4 * i + 1]), __float_as_uint(v[4 * i + 2]), __float_as_uint(v[4 * i + 3])));
    __syncwarp();
#pragma unroll kUnroll
    for (int i = 0; i < 8; ++i) {
        const int row = i * 4 + lr, token = t0 + row;
        const uint4 w = lds128(stage + (uint32_t)(row * 128 + ((lc ^ (row & 7)) << 4)));
        if (token < a.T && rc < R)
            pf_finish<MODE>(a, make_float4(__uint_as_float(w.x), __uint_as_float(w.y), __uint_as_float(w.z), __uint_as_float(w.w)), kEarly ? other[i] : pf_other<MODE>(a, token, col, rc), token, col, rc);
    }
}

template <int M> struct PfModeTag { static constexpr int value = M; };

template <int Q, int NT, int MH, int CG>
__global__ void __launch_bounds__(kPfThreads, NT == 64 ? 2 : 1) prefill_gemm_kernel(const __grid_constant__ PfGemmArgs a) {
    extern __shared__ unsigned char pf_smem_raw[];
    const uint32_t base = (smem_u32(pf_smem_raw) + 1023u) & ~1023u;
    constexpr int BR = NT / CG;                                // weight rows whose B tile this CTA holds
    constexpr int NA = pf_na(Q, BR, MH), NB = pf_nb(Q, BR, MH), kRawBytes = pf_raw_bytes(Q, BR), kPfBBytes = BR * 128;
    constexpr bool kRaw = Q == Q_I4 || Q == Q_I8;              // weights that are widened on the way
    constexpr uint32_t kPfIdesc = Q == Q_BF16 ? umma_idesc_bf16(kPfM * CG, NT, 0) : umma_idesc_f16(kPfM * CG, NT, 0);
    constexpr int kCols = NT > 128 ? 256 : NT;                 // tensor-memory columns between the accumulators of two token halves
    constexpr int kASlot = MH * kPfABytes;                     // X tiles of one slot
    const uint32_t ring_a = base, ring_b = ring_a + NA * kASlot, ring_raw = ring_b + NB * kPfBBytes;
    const uint32_t bars = ring_raw + NA * kRawBytes;
    const uint32_t bar_full = bars, bar_afree = bar_full + 8 * NA, bar_conv = bar_afree + 8 * NA, bar_bfree = bar_conv + 8 * NB, bar_done = bar_bfree + 8 * NB;
    const uint32_t tmem_slot = bar_done + 8;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tm = blockIdx.x / CG, rank = CG == 2 ? blockIdx.x & 1 : 0, tn = blockIdx.y;
    const int S = CG == 2 ? 1 : gridDim.z, z = CG == 2 ? 0 : blockIdx.z;      // S CTAs (a cluster) share a tile's K blocks
    auto token0 = [&](int h) { return ((tm * MH + h) * CG + rank) * kPfM; };  // first token of this CTA's half h
    const bool swiglu = a.mode == PF_SWIGLU;
    const int rows_mat = swiglu ? NT / 2 : NT;                // rows of each matrix in this tile
    const int nmat = swiglu && CG == 1 ? 2 : 1;               // matrices in this CTA's B tile (of a pair's, the even CTA has the gate rows, the odd one the up rows)
    int seg = 0, coff = 0, tseg = tn;                         // plain modes: which matrix this row tile belongs to, its first output column
    if (!swiglu)
        while (seg + 1 < a.nseg && tseg >= (a.seg_rows[seg] + NT - 1) / NT) { tseg -= (a.seg_rows[seg] + NT - 1) / NT; coff += a.seg_rows[seg]; ++seg; }
    const int row0 = tseg * rows_mat;                         // first row inside the matrix
    const int R = a.seg_rows[seg], xrow = Q == Q_BF16 ? a.seg_xrow[seg] : 0;
    const int nk1 = (a.K + kPfKB - 1) / kPfKB, nkb = Q == Q_BF16 ? nk1 + (a.K2 + kPfKB - 1) / kPfKB : nk1;      // columns past the end arrive as zeros
    // this CTA's K blocks [kb0, kb0 + nit): whole groups of 128 columns, so that a split starts with a scale of its own
    const int kstep = kRaw ? 2 : 1, nku = nkb / kstep;
    const int kb0 = (int)((long)nku * z / S) * kstep, nit = (int)((long)nku * (z + 1) / S) * kstep - kb0;
    constexpr int kRawKb = Q == Q_I4 ? 32 : 64;               // raw bytes of one row in one K block
    bool failed = false;

    if (threadIdx.x == 32) { prefetch_map(&a.tx); if (Q == Q_BF16 && a.K2 > 0) { prefetch_map(&a.tx2); prefetch_map(&a.tw2); } }
    if (threadIdx.x == 0) {
        prefetch_map(&a.tw[CG == 2 && swiglu ? rank : seg]);
        for (int s = 0; s < NA; ++s) { mbar_init(bar_full + 8 * s, 1); mbar_init(bar_afree + 8 * s, 1); }
        for (int s = 0; s < NB; ++s) { mbar_init(bar_conv + 8 * s, CG == 1 ? kPfConvWarps : kRaw ? 2 * kPfConvWarps : 1); mbar_init(bar_bfree + 8 * s, 1); }
        mbar_init(bar_done, 1);
        mbar_fence_init();
    }
    if (warp == 1) {
        if (CG == 2) { tmem_alloc2(tmem_slot, (uint32_t)(MH * kCols)); tmem_relinquish2(); }
        else { tmem_alloc(tmem_slot, (uint32_t)(MH * kCols)); tmem_relinquish(); }
    }
    tc_fence_before();
    __syncthreads();
    if (CG == 2) cluster_sync();      // the other CTA's barriers stand before anything arrives there
    tc_fence_after();
    const uint32_t tmem = lds32(tmem_slot);
    pdl_launch_dependents();      // after the allocation: a CTA of the next launch that takes tensor memory early can not keep one of this launch waiting

    if (warp == 0) {
        if (lane == 0) {
            const uint32_t wbytes = !kRaw ? (uint32_t)kPfBBytes : (uint32_t)(BR * kRawKb);
            const int wrow = CG == 2 && !swiglu ? row0 + rank * BR : row0, wmat = CG == 2 && swiglu ? rank : seg;
            auto load_w = [&](int it) {
                const int kb = kb0 + it, sa = it % NA, sb = it % NB;      // fp16, bf16: NB == NA, freed together
                mbar_expect_tx(bar_full + 8 * sa, (uint32_t)kASlot + wbytes);
                if (Q == Q_BF16 && kb >= nk1) { tma_load_2d(ring_b + sb * kPfBBytes, &a.tw2, (kb - nk1) * kPfKB, wrow, bar_full + 8 * sa); return; }      // the second product
                for (int m = 0; m < nmat; ++m) {
                    if (!kRaw) tma_load_2d(ring_b + sb * kPfBBytes + m * rows_mat * 128, &a.tw[wmat + m], kb * kPfKB, wrow, bar_full + 8 * sa);
                    else tma_load_2d(ring_raw + sa * kRawBytes + m * rows_mat * kRawKb, &a.tw[wmat + m], kb * kRawKb, wrow, bar_full + 8 * sa);
                }
            };
            auto load_x = [&](int it) {
                const int kb = kb0 + it, sa = it % NA;
                const bool second = Q == Q_BF16 && kb >= nk1;
                for (int h = 0; h < MH; ++h)        // a half that lies past the last token arrives as zeros
                    if (second) tma_load_2d(ring_a + sa * kASlot + h * kPfABytes, &a.tx2, (kb - nk1) * kPfKB, token0(h), bar_full + 8 * sa);
                    else tma_load_2d(ring_a + sa * kASlot + h * kPfABytes, &a.tx, kb * kPfKB, xrow + token0(h), bar_full + 8 * sa);
            };
            // the weights of the first slots do not depend on the launch before this one
            const int pre = nit < NA ? nit : NA;
            for (int it = 0; it < pre; ++it) load_w(it);
            pdl_wait();
            for (int it = 0; it < pre; ++it) load_x(it);
            for (int it = pre; it < nit; ++it) {
                if (!mbar_wait(bar_afree + 8 * (it % NA), ((uint32_t)(it / NA) & 1u) ^ 1u)) { failed = true; break; }
                load_w(it);
                load_x(it);
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 1) {
            // the odd CTA of a pair: its tiles stand - the converter warps say so themselves, TMA's arrivals are passed on
            const uint32_t conv0 = map_to_rank(bar_conv, 0);
            for (int it = 0; it < (kRaw ? 0 : nit); ++it) {
                if (!mbar_wait(bar_full + 8 * (it % NA), (uint32_t)(it / NA) & 1u)) { failed = true; break; }
                mbar_arrive_cluster(conv0 + 8 * (it % NB));
            }
        } else if (lane == 0) {
            for (int it = 0; it < nit && !failed; ++it) {
                const int sa = it % NA, sb = it % NB; const uint32_t pa = (uint32_t)(it / NA) & 1u, pb = (uint32_t)(it / NB) & 1u;
                if (!mbar_wait(bar_full + 8 * sa, pa)) { failed = true; break; }
                if ((kRaw || CG == 2) && !mbar_wait(bar_conv + 8 * sb, pb)) { failed = true; break; }      // of a pair: both CTAs' tiles
                tc_fence_after();
                const uint32_t at = ring_a + sa * kASlot, bt = ring_b + sb * kPfBBytes;
#pragma unroll
                for (int h = 0; h < MH; ++h)
#pragma unroll
                    for (int k4 = 0; k4 < kPfKB / 16; ++k4)
                        (CG == 2 ? umma2_f16 : umma_f16)(tmem + (uint32_t)(h * kCols), umma_desc(at + h * kPfABytes + k4 * 32), umma_desc(bt + k4 * 32), kPfIdesc, (uint32_t)((it | k4) != 0));
                (CG == 2 ? umma2_commit : umma_commit)(bar_afree + 8 * sa);           // both slots may be refilled once these MMAs have read them
                if (kRaw) (CG == 2 ? umma2_commit : umma_commit)(bar_bfree + 8 * sb);
            }
            (CG == 2 ? umma2_commit : umma_commit)(bar_done);
        }
    } else {
        // a thread widens a whole row of the K block (as many rows as converter threads), or, with two or four times
        // as many threads as rows, a half or a quarter of one
        constexpr int BP = BR > 128 ? 256 : BR > 64 ? 128 : 64;
        constexpr int kPerRow = kPfConvWarps * 32 / BP;       // threads per B row: 1, 2 or 4
        const int c = (threadIdx.x - 64) & (BP - 1);          // B row of this thread (96- and 112-row tiles leave some without one)
        const int kpart = (threadIdx.x - 64) / BP;
        const int cc = CG == 2 ? rank * BR + c : c;           // row of the whole tile
        const int mat = swiglu ? cc / rows_mat : 0, rin = swiglu ? cc % rows_mat : cc;
        const int grow = row0 + rin;
        const bool mine = BP == BR || c < BR, valid = mine && grow < R;
        const uint32_t conv_to = CG == 2 ? map_to_rank(bar_conv, 0) : 0u;
        if (kRaw) {
            const int g0 = kb0 >> 1, ngrp = nit >> 1;          // scale groups of this CTA
            const __half* srow = a.s[seg + (mine ? mat : 0)] + (size_t)(valid ? grow : 0) * (a.K / kGroup) + g0;
            // the scales of the next two groups are already on their way while a group is widened (a load from L2 takes
            // longer than the MMAs of a K block)
            const __half zero = __float2half(0.f);
            __half sc = valid && ngrp > 0 ? srow[0] : zero, sc1 = valid && ngrp > 1 ? srow[1] : zero, sc2 = valid && ngrp > 2 ? srow[2] : zero;
            for (int it = 0; it < nit && !failed; ++it) {
                const int sa = it % NA, sb = it % NB; const uint32_t pa = (uint32_t)(it / NA) & 1u, pb = (uint32_t)(it / NB) & 1u;
                const __half sc_use = sc;
                if (it & 1) { sc = sc1; sc1 = sc2; const int g3 = (it >> 1) + 3; sc2 = valid && g3 < ngrp ? srow[g3] : zero; }
                if (!mbar_wait(bar_full + 8 * sa, pa)) { failed = true; break; }
                if (!mbar_wait(bar_bfree + 8 * sb, pb ^ 1u)) { failed = true; break; }     // the MMAs of two K blocks ago have read this B slot
                if (mine) {
                    constexpr int QQ = kRaw ? Q : Q_I8;
                    const uint32_t rawrow = ring_raw + sa * kRawBytes + c * kRawKb, brow = ring_b + sb * kPfBBytes + c * 128;
                    if (kPerRow == 4) convert_part<QQ, 16>(rawrow + kpart * (kRawKb / 4), brow, c & 7, kpart * 2, __half2half2(sc_use));
                    else {
#pragma unroll
                        for (int kh = kpart; kh < 2; kh += kPerRow)
                            convert_part<QQ, 32>(rawrow + kh * (kRawKb / 2), brow, c & 7, kh * 4, __half2half2(sc_use));
                    }
                }
                fence_async_smem();                            // the tensor core reads through the async proxy
                __syncwarp();
                if (lane == 0) { if (CG == 2) mbar_arrive_cluster(conv_to + 8 * sb); else mbar_arrive(bar_conv + 8 * sb); }
            }
        }
        if (!failed && !mbar_wait(bar_done, 0u)) failed = true;
        tc_fence_after();
        pdl_wait();               // the epilogue adds to, and overwrites, what earlier launches leave
    }

    // Epilogue: TMEM lane = token, column = weight row of the tile.  A unit is 32 tokens x 32 columns (and the up rows' columns
    // beside the gate rows'); unit n = lane quarter * C + chunk belongs to CTA n mod S of the cluster, two warps a quarter.
    const int C = MH * (swiglu ? NT / 64 : NT / 32), per = C / MH, unit_bytes = swiglu ? 8192 : 4096, per_cta = 4 * C / S;
    const int q = warp & 3, hh = warp >= 2 ? (warp - 2) >> 2 : 0;      // TMEM lane quarter (fixed by the warp's number)
    auto taddr = [&](int c) { const int h = c / per; return tmem + (uint32_t)(h * kCols + (c - h * per) * 32) + ((uint32_t)(q * 32) << 16); };
    if (S > 1) {
        // the other CTAs' units go into their rings, which no copy or MMA uses any more once every CTA has passed the first barrier
        __syncwarp();
        cluster_sync();
        if (warp >= 2)
#pragma unroll 1
            for (int c = hh; c < C; c += 2) {
                const int n = q * C + c, owner = n % S;
                if (owner == z) continue;
                const uint32_t to = map_to_rank(base + (uint32_t)(((z < owner ? z : z - 1) * per_cta + n / S) * unit_bytes), (uint32_t)owner);
                float v[32];
                tmem_ld32(taddr(c), v);
                push_block(to, lane, v);
                if (swiglu) { tmem_ld32(taddr(c) + NT / 2, v); push_block(to + 4096, lane, v); }
            }
        __syncwarp();
        cluster_sync();
    }
    auto units = [&](auto mode) {
        constexpr int MODE = decltype(mode)::value;
#pragma unroll 1
        for (int c = 0; c < C; ++c) {
            const int n = q * C + c, slot = n / S;
            if (failed || n % S != z || (slot & 1) != hh) continue;
            const int h = c / per, t0 = token0(h) + q * 32, r = row0 + (c - h * per) * 32;      // the unit's first token and first matrix row
            if (r >= R || t0 >= a.T) continue;
            const uint32_t stage = base + (uint32_t)(S > 1 ? slot * unit_bytes : (warp - 2) * 4096);      // of a split: the block this warp has just read
            pf_unit<MODE>(a, stage, lane, t0, r, R, coff, [&](float (&v)[32], bool up) {
                tmem_ld32(taddr(c) + (up ? NT / 2 : 0), v);
                for (int o = 0; o + 1 < S; ++o) add_block(base + (uint32_t)((o * per_cta + slot) * unit_bytes + (up ? 4096 : 0)), lane, v);
            });
            __syncwarp();
        }
    };
    if (warp >= 2) {
        if (a.mode == PF_OUT_F32) units(PfModeTag<PF_OUT_F32>{});
        else if constexpr (Q == Q_BF16) {
            switch (a.mode) {
                case PF_BF16: units(PfModeTag<PF_BF16>{}); break;
                case PF_BF16_RELU2: units(PfModeTag<PF_BF16_RELU2>{}); break;
                case PF_ADD_F32: units(PfModeTag<PF_ADD_F32>{}); break;
                case PF_BF16_GELU_SIDE: units(PfModeTag<PF_BF16_GELU_SIDE>{}); break;
                case PF_CAP_F32: units(PfModeTag<PF_CAP_F32>{}); break;
                case PF_BF16_GLU: units(PfModeTag<PF_BF16_GLU>{}); break;
                default: units(PfModeTag<PF_DECAY_F32>{}); break;
            }
        } else if (a.mode == PF_RESID) units(PfModeTag<PF_RESID>{});
        else if (a.mode == PF_SWIGLU) units(PfModeTag<PF_SWIGLU>{});
        else units(PfModeTag<PF_OUT_F16>{});
    }
    if (failed && a.err) atomicExch(a.err, 11u);
    tc_fence_before();
    __syncthreads();
    if (CG == 2) cluster_sync();
    if (warp == 1) { if (CG == 2) tmem_dealloc2(tmem, (uint32_t)(MH * kCols)); else tmem_dealloc(tmem, (uint32_t)(MH * kCols)); }
}

// ---- host side ------------------------------------------------------------------------------------------------------
typedef CUresult (*PfEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                               const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static PfEncodeFn pf_encode() {
    static PfEncodeFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) p = nullptr;
        return (PfEncodeFn)p;
    }();
    return fn;
}
// Row-major 2-D map: `cols` elements a row (row pitch = cols elements, or `pitch`), box box_cols x box_rows.
static int pf_map(CUtensorMap* m, const void* p, CUtensorMapDataType dt, int elem, size_t rows, size_t cols, int box_cols, int box_rows, bool swizzle, size_t pitch = 0) {
    PfEncodeFn fn = pf_encode();
    if (!fn) return (int)cudaErrorNotSupported;
    const cuuint64_t dims[2] = {cols, rows}, strides[1] = {(pitch ? pitch : cols) * (size_t)elem};
    const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows}, estr[2] = {1, 1};
    const CUresult r = fn(m, dt, 2, const_cast<void*>(p), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : (int)cudaErrorInvalidValue;
}

template <int Q, int NT, int MH, int CG>
static int pf_go_tile(const PfGemmArgs& a, dim3 grid, cudaStream_t stream) {
    static bool once = false;
    if (!once) {
        const cudaError_t e = cudaFuncSetAttribute(prefill_gemm_kernel<Q, NT, MH, CG>, cudaFuncAttributeMaxDynamicSharedMemorySize, pf_smem_bytes(Q, NT / CG, MH));
        if (e != cudaSuccess) return (int)e;
        once = true;
    }
    cudaLaunchConfig_t lc = {};
    lc.gridDim = grid; lc.blockDim = dim3(kPfThreads); lc.dynamicSmemBytes = pf_smem_bytes(Q, NT / CG, MH); lc.stream = stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[0].val.programmaticStreamSerializationAllowed = a.pdl;
    at[1].id = cudaLaunchAttributeClusterDimension; at[1].val.clusterDim.x = CG; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = grid.z;
    lc.attrs = at; lc.numAttrs = CG * grid.z > 1 ? 2 : 1;
    return (int)cudaLaunchKernelEx(&lc, prefill_gemm_kernel<Q, NT, MH, CG>, a);
}

struct PfPlan { int nt, mh, split, cg; int tokens() const { return kPfM * mh * cg; } };

template <int Q>
static int pf_go(const PfGemmArgs& a, const PfPlan& p, int mtiles, int tiles, cudaStream_t stream) {
    const dim3 grid(mtiles * p.cg, tiles, p.split);
    if (p.cg == 2) {
        if (p.mh == 1) return p.nt == 256 ? pf_go_tile<Q, 256, 1, 2>(a, grid, stream) : p.nt == 192 ? pf_go_tile<Q, 192, 1, 2>(a, grid, stream) : pf_go_tile<Q, 128, 1, 2>(a, grid, stream);
        return p.nt == 256 ? pf_go_tile<Q, 256, 2, 2>(a, grid, stream) : p.nt == 224 ? pf_go_tile<Q, 224, 2, 2>(a, grid, stream) : pf_go_tile<Q, 192, 2, 2>(a, grid, stream);
    }
    if (p.mh == 1) return p.nt == 256 ? pf_go_tile<Q, 256, 1, 1>(a, grid, stream) : p.nt == 128 ? pf_go_tile<Q, 128, 1, 1>(a, grid, stream) : pf_go_tile<Q, 64, 1, 1>(a, grid, stream);
    return p.nt == 256 ? pf_go_tile<Q, 256, 2, 1>(a, grid, stream) : pf_go_tile<Q, 128, 2, 1>(a, grid, stream);
}

static int pf_row_tiles(const int* rows, int nmat, bool swiglu, int nt) {
    int t = 0;
    for (int m = 0; m < (swiglu ? 1 : nmat); ++m) t += (rows[m] + (swiglu ? nt / 2 : nt) - 1) / (swiglu ? nt / 2 : nt);
    return t;
}

// SMs that clusters of n CTAs (one CTA to an SM) can fill at once: a cluster lies within one GPU processing cluster, so sizes of
// four and eight leave some over (measured on 148 SMs: 33 clusters of four run side by side and 36 do not, 14 of eight and 16 not).
static int pf_room(int n, int sms) { return std::max(1, n <= 2 ? sms : n == 4 ? sms * 132 / 148 : sms * 112 / 148); }

// Tile and split of a product, by an estimate: waves of CTAs, each a fixed part and a part per K block (the largest of its MMAs, its bytes through
// shared memory and its widening), and for a split the exchange of partial sums.  The constants began as SM cycles and are fitted to
// measurements of every legal shape and split: the products of five models and two layer-list designs at 8 to 8191 tokens in fp16, int8,
// int4 and bfloat16, 1250 products.  The fit makes a wave dear (the fixed part is some 30,000 whatever the K), and a partly filled last one nearly as dear
// as a full one.  Over those products the choice is 0.9 % slower than the fastest shape on average, more than 10 % slower for 29
// of them and at the most 25 %; over 210 products of random sizes 1.4 %, 10 and 26 %.  (With the constants as they had been derived: 3.2 %, 157 and
// 49 %; 2.3 %, 21 and 33 %.)  What the lines are about:
//   few tiles  a split of K over a cluster: 61 tokens x [896 x 4864] int8 38 us in 14 tiles, 12 in 14 clusters of eight; 500 tokens x
//              [3584 x 18944] int4 151 us with 64-row tiles, 81 with 256 x 256 tiles in clusters of four
//   many       pairs, and the width that fills the last wave: 2048 tokens x [3584 x 3584] int4 53 us with single CTAs, 46 with pairs of 224
//              rows; 4096 tokens x [1536 x 13440] bfloat16 167 us with single CTAs, 126 with pairs of 192 rows
static PfPlan pf_plan(int quant, int T, const int* rows, int nmat, bool swiglu, int nkb, int sms) {
    static const int shapes[][3] = {{64, 1, 1}, {128, 1, 1}, {256, 1, 1}, {128, 2, 1}, {256, 2, 1}, {128, 1, 2}, {192, 1, 2}, {256, 1, 2}, {192, 2, 2}, {224, 2, 2}, {256, 2, 2}};      // rows, token halves, CTAs
    PfPlan best{256, 1, 1, 1};
    double best_t = 1e30;
    for (const auto& f : shapes) {
        const int nt = f[0], mh = f[1], cg = f[2], br = nt / cg;
        if ((mh * cg > 1 && T <= kPfM) || (mh * cg > 2 && T <= 2 * kPfM) || (swiglu && nt % 64)) continue;
        const int tok = kPfM * mh * cg, ctas = (T + tok - 1) / tok * pf_row_tiles(rows, nmat, swiglu, nt) * cg;
        const double raw = pf_raw_bytes(quant, br), xb = mh * kPfABytes, bb = br * 128;
        const double smem = (xb + 2 * raw + bb + mh * (kPfABytes + bb)) / 136, widen = quant == Q_I4 ? 3.65 * br : quant == Q_I8 ? 4.0 * br : 0.0;
        const double kcyc = std::max(std::max(2.25 * mh * nt, smem), std::max(widen, 460.0)) + (cg == 2 ? 70.0 : 0.0);
        const int kstep = pf_widens(quant) ? 2 : 1, nku = nkb / kstep, units = 4 * mh * nt / (swiglu ? 64 : 32);
        for (int s = 1; s <= (cg == 2 ? 1 : 8) && s <= nku; s *= 2) {
            if (units % s || (mh == 2 && nt == 256 && s > 4)) break;
            const double fill = (double)ctas * s / pf_room(s, sms), full = std::ceil(fill), waves = full > 1 ? full - 0.13 * (full - fill) : full;
            const double t = waves * (30000.0 + 7.0 * mh * nt + (double)((nku + s - 1) / s) * kstep * kcyc) + (s > 1 ? 1400.0 + 14.0 * mh * nt * (s - 1) / s : 0.0);
            if (t < best_t) { best_t = t; best = PfPlan{nt, mh, s, cg}; }
        }
    }
    return best;
}
static int pf_sms() {
    int sms = 0, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms > 0 ? sms : 1;
}

static int pf_launch(int quant, PfGemmArgs& a, const void* x, const void* const* w, const int* rows, int nmat, const PfPlan& p, cudaStream_t stream) {
    const bool swiglu = a.mode == PF_SWIGLU;
    const int mtiles = (a.T + p.tokens() - 1) / p.tokens(), tiles = pf_row_tiles(rows, nmat, swiglu, p.nt), rows_mat = swiglu ? p.nt / 2 : p.nt / p.cg;      // rows_mat: rows of a copy
    if (int r = pf_map(&a.tx, x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (size_t)a.T, (size_t)a.K, kPfKB, kPfM, true)) return r;
    a.R = 0;
    for (int m = 0; m < nmat; ++m) {
        int r;
        if (quant == Q_F16) r = pf_map(&a.tw[m], w[m], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (size_t)rows[m], (size_t)a.K, kPfKB, rows_mat, true);
        else {
            const size_t rb = quant == Q_I4 ? (size_t)a.K / 2 : (size_t)a.K;
            r = pf_map(&a.tw[m], w[m], CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, (size_t)rows[m], rb, quant == Q_I4 ? 32 : 64, rows_mat, false);
        }
        if (r) return r;
        a.seg_rows[m] = rows[m];
        if (!swiglu || m == 0) a.R += rows[m];
    }
    a.nseg = swiglu ? 1 : nmat;
    return quant == Q_I4 ? pf_go<Q_I4>(a, p, mtiles, tiles, stream) : quant == Q_I8 ? pf_go<Q_I8>(a, p, mtiles, tiles, stream) : pf_go<Q_F16>(a, p, mtiles, tiles, stream);
}

int launch_prefill_gemm(int quant, PfGemmArgs& a, const void* x, const void* const* w, const int* rows, int nmat, cudaStream_t stream) {
    if (a.T <= 0 || a.K <= 0 || a.K % kGroup || a.ldo % 8 || quant < 0 || quant > 2 || nmat < 1 || nmat > 3) return (int)cudaErrorInvalidValue;
    const bool swiglu = a.mode == PF_SWIGLU;
    if (swiglu && (nmat != 2 || rows[0] != rows[1])) return (int)cudaErrorInvalidValue;
    for (int m = 0; m < nmat; ++m) if (!w[m] || rows[m] <= 0 || rows[m] % 8) return (int)cudaErrorInvalidValue;
    return pf_launch(quant, a, x, w, rows, nmat, pf_plan(quant, a.T, rows, nmat, swiglu, a.K / kPfKB, pf_sms()), stream);
}

static int pf_launch_bf16(PfGemmArgs& a, const void* x, int ldx, const PfBf16Mat* m, int nmat, const void* x2, int ldx2, const PfBf16Mat* m2, const PfPlan& p, cudaStream_t stream) {
    const CUtensorMapDataType bf = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    int xrows = a.T;
    for (int i = 0; i < nmat; ++i) if (m[i].xrow + a.T > xrows) xrows = m[i].xrow + a.T;
    if (int r = pf_map(&a.tx, x, bf, 2, (size_t)xrows, (size_t)a.K, kPfKB, kPfM, true, (size_t)ldx)) return r;
    int tiles = 0;
    a.R = 0;
    for (int i = 0; i < nmat; ++i) {
        a.seg_xrow[i] = m[i].xrow;
        if (int r = pf_map(&a.tw[i], m[i].w, bf, 2, (size_t)m[i].rows, (size_t)a.K, kPfKB, p.nt / p.cg, true, (size_t)m[i].pitch)) return r;
        a.seg_rows[i] = m[i].rows;
        tiles += (m[i].rows + p.nt - 1) / p.nt; a.R += m[i].rows;
    }
    a.nseg = nmat;
    if (x2) {
        if (int r = pf_map(&a.tx2, x2, bf, 2, (size_t)a.T, (size_t)a.K2, kPfKB, kPfM, true, (size_t)ldx2)) return r;
        if (int r = pf_map(&a.tw2, m2->w, bf, 2, (size_t)m2->rows, (size_t)a.K2, kPfKB, p.nt / p.cg, true, (size_t)m2->pitch)) return r;
    }
    return pf_go<Q_BF16>(a, p, (a.T + p.tokens() - 1) / p.tokens(), tiles, stream);
}

int launch_prefill_gemm_bf16(PfGemmArgs& a, const void* x, int ldx, const PfBf16Mat* m, int nmat, const void* x2, int ldx2, const PfBf16Mat* m2, cudaStream_t stream) {
    if (a.T <= 0 || a.K <= 0 || a.K % 8 || a.ldo % 8 || ldx % 8 || nmat < 1 || nmat > kPfMaxMat || (a.mode != PF_OUT_F32 && a.mode < PF_BF16) || (a.mode == PF_BF16_GLU && (nmat != 1 || m->rows % 16)) || (x2 && (nmat != 1 || !m2 || m2->rows != m->rows || a.K2 % 8 || ldx2 % 8)))
        return (int)cudaErrorInvalidValue;
    if (!x2) a.K2 = 0;
    int rows[kPfMaxMat];
    for (int i = 0; i < nmat; ++i) {
        if (m[i].xrow < 0 || !m[i].w || m[i].rows <= 0 || m[i].rows % 8 || m[i].pitch % 8 || m[i].pitch < a.K) return (int)cudaErrorInvalidValue;
        rows[i] = m[i].rows;
    }
    const int nkb = (a.K + kPfKB - 1) / kPfKB + (a.K2 + kPfKB - 1) / kPfKB;
    return pf_launch_bf16(a, x, ldx, m, nmat, x2, ldx2, m2, pf_plan(Q_BF16, a.T, rows, nmat, false, nkb, pf_sms()), stream);
}

}  // namespace cq
