// Causal attention for a tile of prompt tokens on the tcgen05 tensor cores (head_dim 64 or 128): the batched counterpart of
// the reference's decode attention (src/kernels.cu:105-288), which the reference applies once per prompt token
// (src/main.cu:86-92).  prefill_attn.cu holds an mma.sync kernel, used for few queries near the beginning.
//
// One CTA = two tiles of 128 queries, or one where there are SMs enough; one CTA to an SM.  The tiles of a KV group (128 queries of one of
// its heads each) are numbered from the last queries down, the heads of the same queries side by side, and go to CTAs in that order: two tiles of a CTA
// then mostly see the same keys, at most one CTA of a group goes without a second one, and the longest start first.  Per tile of 128 keys:
//   warp 8      TMA: K and V tiles of the head's KV group (64-column boxes, hardware-swizzled), two slots each
//   warp 9      one lane issues, for the two query tiles in turn, O += P V of a key tile (A = P from tensor memory, B = V as the MN-major
//               operand straight from its cache layout) and S = Q K^T of the next (both operands K-major)
//   warps 0-3   softmax of the first query tile, warps 4-7 of the second: one thread per query row (TMEM lane = row) reads its 128 scores,
//               masks, writes P = 2^(s - m) as fp16 over them, row sum in fp32; when a row's maximum outgrows m by 2^8, m moves
//               and O is rescaled in TMEM by 2^(m_old - m_new) (rare after the first tiles)
// While one tile's softmax runs, the tensor core works for the other.  A row belongs to one thread and P stays in tensor memory, so a tile costs
// no barrier among the softmax warps and no pass through shared memory; what bounds it is the chain of a tile - scores, exponentials (1024
// cycles of an SM partition's unit), P V, next scores - of which the two query tiles hide half.  Against two threads to a row, P in shared
// memory, 64-key tiles and two CTAs to an SM: 40 heads x 8190 queries 782 us for 999 (0.88 PFLOP/s), 16 heads x 3000 queries at 1000 115 for 140.
// Two tiles of one head to every CTA left SMs idle where there are few, and half of the last CTAs idle: 40 heads x 777 queries at 3000 135 us, now 76;
// 28 heads x 192 from 0 on 11.3, now 8.7; 14 heads of 64 x 512 at 1000 31.3, now 27.7 (64-key tiles, two CTAs to an SM: 92, 7.7 and 27.0).
// The tensor core finishes its MMAs in the order of issue: when S of a key tile is there, so is P V of the one before, and O may be rescaled.
// Every mbarrier wait is bounded; a wait that runs out sets *err and the CTA drains.
#include "prefill.cuh"
#include "stack_dev.cuh"
#include "tcgen05.cuh"

#include <algorithm>

namespace cq {

constexpr int kTaBM = 128, kTaBN = 128, kTaQ = 2;      // queries of a tile, keys of a tile, query tiles of a CTA
constexpr int kTaThreads = 320;
// Per head_dim HD (128 or 64): a tile of Q, K or V = HD / 64 blocks of [128 rows][128 bytes].  Q x 2, K x 2, V x 2, barriers; the dynamic
// shared memory is declared 1024-byte aligned.
constexpr int kTaBlk = 128 * 128;
__host__ __device__ constexpr int ta_tile(int hd) { return hd / 64 * kTaBlk; }
__host__ __device__ constexpr int ta_smem(int hd) { return 6 * ta_tile(hd) + 256; }
// TMEM columns: S (128; P in the first 64 of them) and O (HD, 128 at the most) of one query tile or two.  A launch without pairs takes
// half of the memory, so that the next launch's first CTAs find some.
__host__ __device__ constexpr uint32_t ta_cols(bool pairs) { return pairs ? 512u : 256u; }

struct PfAttnTcArgs {
    CUtensorMap tq;          // q as [T][ldq] fp16, box 64 x 128, swizzled
    CUtensorMap tk, tv;      // caches as [n_kv][rows][hd] fp16, box 64 x 128 x 1, swizzled
    __half* out;
    int T, pos0, n_kv, grp, ldq;
    int singles;             // query tiles of a KV group, from the longest down, that have a CTA to themselves
    float scale_log2;
    unsigned* err;
};

__device__ __forceinline__ float ta_ex2(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }

template <int HD>
__global__ void __launch_bounds__(kTaThreads, 1) prefill_attn_tc_kernel(const __grid_constant__ PfAttnTcArgs a) {
    constexpr int kTile = ta_tile(HD), NBLK = HD / 64;
    extern __shared__ __align__(1024) unsigned char ta_smem_raw[];
    const uint32_t base = smem_u32(ta_smem_raw);
    const uint32_t sQ = base, sK = sQ + 2 * kTile, sV = sK + 2 * kTile, bars = sV + 2 * kTile;
    const uint32_t b_q = bars, b_kfull = bars + 8, b_kfree = bars + 24, b_vfull = bars + 40, b_vfree = bars + 56, b_s = bars + 72, b_p = bars + 88, b_o = bars + 120, tmem_slot = bars + 136;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kvh = blockIdx.x % a.n_kv, cta = blockIdx.x / a.n_kv, nqt = (a.T + kTaBM - 1) / kTaBM, units = nqt * a.grp;
    const int u0 = cta < a.singles ? cta : 2 * cta - a.singles;
    const int nq = cta >= a.singles && u0 + 1 < units ? 2 : 1;            // query tiles of this CTA; the last one sees the most keys
    const int qlast = (nqt - 1 - u0 / a.grp) * kTaBM, hlast = kvh * a.grp + u0 % a.grp;
    const int qfirst = nq > 1 ? (nqt - 1 - (u0 + 1) / a.grp) * kTaBM : qlast, hfirst = nq > 1 ? kvh * a.grp + (u0 + 1) % a.grp : hlast;
    auto q0 = [&](int i) { return i == nq - 1 ? qlast : qfirst; };        // tile i: first query, head
    auto head = [&](int i) { return i == nq - 1 ? hlast : hfirst; };
    auto key_end = [&](int i) { return a.pos0 + min(q0(i) + kTaBM, a.T); };             // keys that it sees at all
    auto tiles = [&](int i) { return (key_end(i) + kTaBN - 1) / kTaBN; };
    const int nj = tiles(nq - 1);
    const uint32_t cols = ta_cols(a.singles < units);
    bool failed = false;

    if (threadIdx.x == 256) { prefetch_map(&a.tq); prefetch_map(&a.tk); prefetch_map(&a.tv); }
    if (threadIdx.x == 0) {
        mbar_init(b_q, 1);
        for (int s = 0; s < 2; ++s) {
            mbar_init(b_kfull + 8 * s, 1); mbar_init(b_kfree + 8 * s, 1); mbar_init(b_vfull + 8 * s, 1); mbar_init(b_vfree + 8 * s, 1);
            mbar_init(b_s + 8 * s, 1); mbar_init(b_p + 16 * s, 4); mbar_init(b_p + 16 * s + 8, 4); mbar_init(b_o + 8 * s, 1);
        }
        mbar_fence_init();
    }
    if (warp == 9) { tmem_alloc(tmem_slot, cols); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = lds32(tmem_slot);
    pdl_launch_dependents();      // after the allocation: what the next launch takes early can not keep a CTA of this one waiting
    const uint32_t tS = tmem, tO = tmem + cols / 2;

    if (warp == 8) {
        if (lane == 0) {
            pdl_wait();           // everything below follows from these loads
            mbar_expect_tx(b_q, (uint32_t)(nq * kTile));
            for (int i = 0; i < nq; ++i)
                for (int b = 0; b < NBLK; ++b) tma_load_2d(sQ + i * kTile + b * kTaBlk, &a.tq, head(i) * HD + 64 * b, q0(i), b_q);
            for (int j = 0; j < nj; ++j) {
                const int s = j & 1; const uint32_t free_par = (((uint32_t)j >> 1) & 1u) ^ 1u;
                if (!mbar_wait(b_kfree + 8 * s, free_par)) { failed = true; break; }
                mbar_expect_tx(b_kfull + 8 * s, (uint32_t)kTile);
                for (int b = 0; b < NBLK; ++b) tma_load_3d(sK + s * kTile + b * kTaBlk, &a.tk, 64 * b, j * kTaBN, kvh, b_kfull + 8 * s);
                if (!mbar_wait(b_vfree + 8 * s, free_par)) { failed = true; break; }
                mbar_expect_tx(b_vfull + 8 * s, (uint32_t)kTile);
                for (int b = 0; b < NBLK; ++b) tma_load_3d(sV + s * kTile + b * kTaBlk, &a.tv, 64 * b, j * kTaBN, kvh, b_vfull + 8 * s);
            }
        }
    } else if (warp == 9) {
        if (lane == 0) {
            constexpr uint32_t idS = umma_idesc_f16(kTaBM, kTaBN, 0), idPV = umma_idesc_f16(kTaBM, HD, 1);
            // S of query tile i and key tile j; the last query tile's reads the K slot last
            auto issue_s = [&](int i, int j) {
                const int s = j & 1;
#pragma unroll
                for (int ks = 0; ks < HD / 16; ++ks) {
                    const uint32_t off = (uint32_t)((ks >> 2) * kTaBlk + (ks & 3) * 32);
                    umma_f16(tS + (uint32_t)(i * kTaBN), umma_desc_sw128(sQ + i * kTile + off, 16, 1024), umma_desc_sw128(sK + s * kTile + off, 16, 1024), idS, (uint32_t)(ks != 0));
                }
                umma_commit(b_s + 8 * i);
                if (i == nq - 1) umma_commit(b_kfree + 8 * s);
            };
            if (!mbar_wait(b_q, 0u) || !mbar_wait(b_kfull, 0u)) failed = true;
            tc_fence_after();
            if (!failed) for (int i = 0; i < nq; ++i) issue_s(i, 0);
            for (int j = 0; j < nj && !failed; ++j) {
                const int s = j & 1;
                if (!mbar_wait(b_vfull + 8 * s, ((uint32_t)j >> 1) & 1u)) { failed = true; break; }
                if (j + 1 < nj && !mbar_wait(b_kfull + 8 * (s ^ 1), ((uint32_t)(j + 1) >> 1) & 1u)) { failed = true; break; }
                for (int i = 0; i < nq && !failed; ++i) {
                    const int mine = tiles(i);
                    if (j >= mine) continue;
                    const int steps = min(kTaBN / 32, (key_end(i) - j * kTaBN + 31) / 32) * 2;
                    for (int half = 0; half < 2; ++half) {        // P arrives in halves of 64 keys
                        if (!mbar_wait(b_p + 16 * i + 8 * half, (uint32_t)j & 1u)) { failed = true; break; }
                        tc_fence_after();
#pragma unroll
                        for (int k4 = 0; k4 < 4; ++k4) {          // sixteen keys a step: V rows 16 ks .., P columns 16 ks .. (two to a 32-bit column)
                            const int ks = half * 4 + k4;
                            if (ks < steps) umma_f16_ta(tO + (uint32_t)(i * HD), tS + (uint32_t)(i * kTaBN + ks * 8), umma_desc_sw128(sV + s * kTile + ks * 2048, kTaBlk, 1024), idPV, (uint32_t)((j | ks) != 0));
                        }
                    }
                    if (failed) break;
                    if (i == nq - 1) umma_commit(b_vfree + 8 * s);
                    if (j + 1 < mine) issue_s(i, j + 1);
                    else umma_commit(b_o + 8 * i);
                }
            }
        }
    } else if ((warp >> 2) < nq) {
        const int i = warp >> 2, r = (warp & 3) * 32 + lane;              // query tile, row of it = TMEM lane
        const int qi = q0(i), qpos = a.pos0 + qi + r, mine = tiles(i);
        const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16, s_at = tS + (uint32_t)(i * kTaBN) + lane_off, o_at = tO + (uint32_t)(i * HD) + lane_off;
        // m is the exponent the row's probabilities are scaled by, not always its running maximum: it moves only when
        // a tile's maximum exceeds it by more than 2^8 (probabilities then stay below 256, well inside fp16, and the
        // row sum is fp32), so that most tiles need no rescale of O in TMEM.
        float m = -INFINITY, l = 0.f;
        const f32x2 scale2 = pack2(a.scale_log2, a.scale_log2);
        for (int j = 0; j < mine; ++j) {
            if (!failed && !mbar_wait(b_s + 8 * i, (uint32_t)j & 1u)) failed = true;
            tc_fence_after();
            const int key0 = j * kTaBN, nc = min(4, (key_end(i) - key0 + 31) / 32);       // 32-key pieces that some query sees (uniform over the tile); P V leaves the others out
            uint32_t x[4][32];
#pragma unroll
            for (int c = 0; c < 4; ++c) if (c < nc) tmem_ld32_issue(s_at + (uint32_t)(c * 32), x[c]);
            tmem_wait_ld();
            float mx4[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                mx4[c] = -INFINITY;
                if (c >= nc) continue;
                const int key = key0 + c * 32;
                if (key + 31 > a.pos0 + qi) {                 // some key of this piece may lie past some query (uniform over the tile)
#pragma unroll
                    for (int k = 0; k < 32; ++k) if (key + k > qpos) x[c][k] = 0xff800000u;      // -infinity
                }
#pragma unroll
                for (int k = 0; k < 32; ++k) mx4[c] = fmaxf(mx4[c], __uint_as_float(x[c][k]));
            }
            const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * a.scale_log2;
            const bool move = mx > m + 8.0f;                              // also true on the first tile (m = -inf; key 0 is visible to every query)
            if (__any_sync(0xffffffffu, move)) {                          // warp-uniform: the TMEM accesses below are warp-wide
                float alpha = 1.f;
                if (move) { alpha = m == -INFINITY ? 0.f : ta_ex2(m - mx); m = mx; l *= alpha; }
                if (j > 0) {
#pragma unroll 1
                    for (int c = 0; c < HD / 32; ++c) {
                        float v[32];
                        tmem_ld32(o_at + (uint32_t)(c * 32), v);
#pragma unroll
                        for (int k = 0; k < 32; ++k) v[k] *= alpha;
                        tmem_st32(o_at + (uint32_t)(c * 32), v);
                    }
                }
            }
            const f32x2 m2 = pack2(-m, -m);
            f32x2 sum[2] = {0ull, 0ull};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                if (c < nc) {
                    uint32_t pk[16];
#pragma unroll
                    for (int k = 0; k < 32; k += 2) {
                        float e0, e1;
                        unpack2(fma2(pack2(__uint_as_float(x[c][k]), __uint_as_float(x[c][k + 1])), scale2, m2), e0, e1);
                        e0 = ta_ex2(e0); e1 = ta_ex2(e1);
                        sum[(k >> 1) & 1] = add2(sum[(k >> 1) & 1], pack2(e0, e1));
                        pk[k >> 1] = pack_h2(e0, e1);
                    }
                    tmem_st16(s_at + (uint32_t)(c * 16), pk);
                }
                if (c & 1) {
                    tmem_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(b_p + 16 * i + 8 * (c >> 1));
                }
            }
            l += sum2(add2(sum[0], sum[1]));
        }
        if (!failed && !mbar_wait(b_o + 8 * i, 0u)) failed = true;
        tc_fence_after();
        const float inv = 1.0f / l;
        const int t = qi + r;
#pragma unroll 1
        for (int c = 0; c < HD / 32; ++c) {
            float v[32];
            tmem_ld32(o_at + (uint32_t)(c * 32), v);
            if (t < a.T && !failed) {
                __half* dst = a.out + (size_t)t * a.ldq + head(i) * HD + c * 32;
#pragma unroll
                for (int k = 0; k < 32; k += 8)
                    *reinterpret_cast<uint4*>(dst + k) = make_uint4(pack_h2(v[k] * inv, v[k + 1] * inv), pack_h2(v[k + 2] * inv, v[k + 3] * inv),
                                                                    pack_h2(v[k + 4] * inv, v[k + 5] * inv), pack_h2(v[k + 6] * inv, v[k + 7] * inv));
            }
            __syncwarp();
        }
    }
    if (failed && a.err) atomicExch(a.err, 12u);
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 9) tmem_dealloc(tmem, cols);
}

typedef CUresult (*TaEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                               const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static TaEncodeFn ta_encode() {
    static TaEncodeFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) p = nullptr;
        return (TaEncodeFn)p;
    }();
    return fn;
}

template <int HD>
static int ta_go(const PfAttnTcArgs& k, dim3 grid, const LaunchCfg& cfg) {
    static bool once = false;
    if (!once) {
        const cudaError_t e = cudaFuncSetAttribute(prefill_attn_tc_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, ta_smem(HD));
        if (e != cudaSuccess) return (int)e;
        once = true;
    }
    return st_launch(prefill_attn_tc_kernel<HD>, grid, dim3(kTaThreads), (size_t)ta_smem(HD), cfg, k);
}

int launch_prefill_attn_tc(int head_dim, const PfAttnArgs& a, int n_kv, unsigned* err, const LaunchCfg& cfg) {
    const int kTaHD = head_dim;
    if (head_dim != 64 && head_dim != 128) return (int)cudaErrorInvalidValue;
    if (a.T <= 0 || a.pos0 < 0 || a.pos0 + a.T > a.max_seq || a.grp <= 0 || a.ldq % 8 || n_kv <= 0 || a.n_heads != n_kv * a.grp) return (int)cudaErrorInvalidValue;
    TaEncodeFn fn = ta_encode();
    if (!fn) return (int)cudaErrorNotSupported;
    PfAttnTcArgs k; memset(&k, 0, sizeof k);
    const cuuint32_t estr[3] = {1, 1, 1};
    {
        const cuuint64_t dims[2] = {(cuuint64_t)a.ldq, (cuuint64_t)a.T}, strides[1] = {(cuuint64_t)a.ldq * 2};
        const cuuint32_t box[2] = {64, kTaBM};
        if (fn(&k.tq, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<__half*>(a.q), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) return (int)cudaErrorInvalidValue;
    }
    const __half* caches[2] = {a.kc, a.vc};
    CUtensorMap* maps[2] = {&k.tk, &k.tv};
    for (int i = 0; i < 2; ++i) {
        const cuuint64_t dims[3] = {(cuuint64_t)kTaHD, (cuuint64_t)(a.pos0 + a.T), (cuuint64_t)n_kv};      // rows past the last query's arrive as zeros, whatever the cache holds there
        const cuuint64_t strides[2] = {(cuuint64_t)kTaHD * 2, (cuuint64_t)a.max_seq * kTaHD * 2};
        const cuuint32_t box[3] = {64, kTaBN, 1};
        if (fn(maps[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<__half*>(caches[i]), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) return (int)cudaErrorInvalidValue;
    }
    k.out = a.out; k.T = a.T; k.pos0 = a.pos0; k.n_kv = n_kv; k.grp = a.grp; k.ldq = a.ldq; k.scale_log2 = a.scale_log2; k.err = err;
    const int units = (a.T + kTaBM - 1) / kTaBM * a.grp;
    // Alone a tile is done sooner (14 heads of 64, 129 queries at 8000: 126 us for 136 in pairs): as many as leave no CTA without an SM, and none
    // with more than two tiles to an SM.
    const int slots = cfg.sm_count / n_kv;
    k.singles = std::min(units, std::max(0, 2 * slots - units));
    const dim3 grid((k.singles + (units - k.singles + 1) / 2) * n_kv);
    return head_dim == 128 ? ta_go<128>(k, grid, cfg) : ta_go<64>(k, grid, cfg);
}

}  // namespace cq
