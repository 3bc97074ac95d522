// Tensor-core stages of the SSD chunked forward for sm_100a: tcgen05.mma with TMEM accumulators,
// operands brought into 128-byte-swizzled shared memory by TMA (cp.async.bulk.tensor, no multicast).
//
// The shape served here: 16-bit inputs (bf16 / fp16), headdim 64, dstate 128, chunks of 256 steps.  Kernels:
//
//   chunk_state / state_stream   S^T[n,p] = sum_k B[k,n] (w_k x[k,p]), w_k = exp(min(dA_last - dA_k, 0)) dt_k, per chunk, and
//               the recurrence over chunks (fused in state_stream); leave the state entering each chunk in 16 bits
//   output      per chunk and group, over its heads: C.B^T, the decay-masked product with x, C.H, the D skip and the gate
//   varlen      end states of packed sequences (bf16)
//
// Every mbarrier wait is bounded: on expiry the kernel records a code in the status word, skips the dependent work and
// still releases its TMEM before it exits.
#include <algorithm>
#include <atomic>
#include <type_traits>

#include "ssd_common.cuh"
#include "tc_sm100.cuh"
#include "tensor_map.cuh"

namespace mb200 {

// ---- host: tensor maps of the 16-bit operands (SWIZZLE_128B tiles) -----------------------------------
// fmt: 1 = bfloat16, 0 = float16 (the encoding of the MMA instruction descriptor)
static bool encode_16bit(CUtensorMap *map, int fmt, const void *base, int rank, const uint64_t *dims, const uint64_t *strides_bytes,
                         const uint32_t *box)
{
    return encode_tiled(map, fmt == 1 ? MB200_BF16 : MB200_F16, base, rank, dims, strides_bytes, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

namespace {

using namespace tc;

constexpr int kQ = kTcChunk, kP = 64, kN = 128;  // steps per chunk, columns of a head, states

// status codes written to the scratch status word
enum { kStBarB = 11, kStBarX, kStBarScaled, kStBarDone, kStSmemAlign };

template <typename T> struct Pack2;
template <> struct Pack2<__nv_bfloat16> {
    static __device__ __forceinline__ uint32_t mul(uint32_t a, uint32_t b)   // two 16-bit products, one instruction
    {
        __nv_bfloat162 r = __hmul2(*reinterpret_cast<__nv_bfloat162 *>(&a), *reinterpret_cast<__nv_bfloat162 *>(&b));
        return *reinterpret_cast<uint32_t *>(&r);
    }
    static __device__ __forceinline__ float2 unpack(uint32_t v) { return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162 *>(&v)); }
    static __device__ __forceinline__ uint32_t pack(float a, float b)
    {
        __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
        return *reinterpret_cast<uint32_t *>(&h);
    }
};
template <> struct Pack2<__half> {
    static __device__ __forceinline__ uint32_t mul(uint32_t a, uint32_t b)
    {
        __half2 r = __hmul2(*reinterpret_cast<__half2 *>(&a), *reinterpret_cast<__half2 *>(&b));
        return *reinterpret_cast<uint32_t *>(&r);
    }
    static __device__ __forceinline__ float2 unpack(uint32_t v) { return __half22float2(*reinterpret_cast<__half2 *>(&v)); }
    static __device__ __forceinline__ uint32_t pack(float a, float b)
    {
        __half2 h = __floats2half2_rn(a, b);
        return *reinterpret_cast<uint32_t *>(&h);
    }
};
template <typename T> struct Fmt;
template <> struct Fmt<__nv_bfloat16> { static constexpr int v = 1; };
template <> struct Fmt<__half> { static constexpr int v = 0; };

__device__ __forceinline__ uint8_t *align1024(uint8_t *p)
{
    return reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(p) + 1023) & ~uintptr_t(1023));
}
// Barrier over the 512 element-wise threads of the state-stream kernel (named barrier 1) that also ANDs a
// predicate across them, so a bounded wait that ran out in one warp stops every warp at the same point.
__device__ __forceinline__ bool stream_barrier_and(bool p)
{
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred q, o;\n\t"
        "setp.ne.u32 q, %1, 0;\n\t"
        "bar.red.and.pred o, 1, 512, q;\n\t"
        "selp.u32 %0, 1, 0, o;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)p)
        : "memory");
    return r != 0;
}
__device__ __forceinline__ uint4 lds128(uint32_t addr)
{
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ float lds32(uint32_t addr)
{
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ void lds128f(uint32_t addr, float (&v)[4])
{
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(addr));
}
__device__ __forceinline__ void lds_pair2(uint32_t addr, uint64_t &a, uint64_t &b)      // four floats as two packed pairs
{
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(addr));
}
__device__ __forceinline__ void sts128(uint32_t addr, uint4 v)
{
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// ====================================================================================== chunk state
// grid (nheads, nchunks, batch), 288 threads.  smem: B 2 x 32 KB (n halves, [256 k x 64 n]), x 32 KB.
// TMEM: 64 columns.  S^T[n,p] = sum_k B[k,n] (w_k x[k,p]): the per-step weight w_k is applied to the x rows
// (half as many elements as B, and x is per head anyway), one row per thread, in place, fp32 product with
// one rounding; B is used as TMA delivered it.
constexpr int kStateThreads = 288;
template <typename T>
__global__ void __launch_bounds__(kStateThreads) ssd_tc_chunk_state_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_B,
                                                                          const float *dtb, const float *dAb, float *states, int nchunks,
                                                                          int nheads, int heads_per_group, const int32_t *seq_idx, int seqlen,
                                                                          int *status)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t *sm = align1024(smem_raw);
    uint8_t *Bs = sm;               // two boxes [256 x 64]
    uint8_t *xs = sm + 65536;       // [256 x 64]
    uint64_t *bars = reinterpret_cast<uint64_t *>(sm + 98304);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 4);
    const int h = blockIdx.x, c = blockIdx.y, b = blockIdx.z;
    const int g = h / heads_per_group;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // the row weight is requested before the set-up barrier so its latency hides behind it and the TMA loads
    float pre_dA = 0.f, pre_dt = 0.f, pre_last = 0.f;
    if (threadIdx.x < 256) {
        const float *dtc = dtb + (((int64_t)b * nheads + h) * nchunks + c) * kQ;
        const float *dAc = dAb + (((int64_t)b * nheads + h) * nchunks + c) * kQ;
        pre_last = dAc[kQ - 1];
        pre_dA = dAc[threadIdx.x];
        pre_dt = dtc[threadIdx.x];
        if (seq_idx) {      // packed sequences: only steps of the chunk's last sequence reach its end state
            const int32_t *sid = seq_idx + (int64_t)b * seqlen;
            const int t = c * kQ + threadIdx.x, t_last = min(c * kQ + kQ, seqlen) - 1;
            if (t < seqlen && sid[t] != sid[t_last]) pre_dt = 0.f;
        }
    }
    if (threadIdx.x == 256) {
        mbar_init(&bars[0], 1);      // B landed
        mbar_init(&bars[1], 1);      // x landed
        mbar_init(&bars[2], 8);      // x rows weighted: one arrival per element-wise warp
        mbar_init(&bars[3], 1);      // MMAs done
        mbar_fence_init();
    }
    if (warp == 8) tmem_alloc(tmem_slot, 64);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    if (warp == 8) {
        if (lane == 0) {
            mbar_expect_tx(&bars[1], 32768);
            tma_load_4d(xs, &tm_x, &bars[1], 0, h, c * kQ, b);
            mbar_expect_tx(&bars[0], 65536);
            for (int kb = 0; kb < 2; ++kb) tma_load_4d(Bs + kb * 32768, &tm_B, &bars[0], kb * 64, g, c * kQ, b);
        }
        __syncwarp();
        const bool ok = __all_sync(0xffffffffu, mbar_wait(&bars[2], 0, status, kStBarScaled) && mbar_wait(&bars[0], 0, status, kStBarB));
        tc_fence_after_sync();
        const uint32_t idesc = instr_desc_f16(128, 64, Fmt<T>::v, 1, 1), tm = warp_uniform(tmem);
        const uint64_t dB = smem_desc_sw128(smem_u32(Bs), 32768, 1024), dx = smem_desc_sw128(smem_u32(xs), 16, 1024);
        if (elect_one()) {
            if (ok) mma_steps_ss(kQ / 16, tm, dB, 128, dx, 128, idesc, false);
            mma_commit(&bars[3]);
        }
        __syncwarp();
    } else {
        const int k = threadIdx.x;
        const float w = __expf(fminf(pre_last - pre_dA, 0.f)) * pre_dt;
        const bool ok = mbar_wait(&bars[1], 0, status, kStBarX);
        if (ok) {
            const uint32_t base = smem_u32(xs) + k * 128;
#pragma unroll
            for (int ch = 0; ch < 8; ++ch) {
                const uint32_t addr = base + ((ch ^ (k & 7)) << 4);
                uint4 v = lds128(addr);
                uint32_t *e = reinterpret_cast<uint32_t *>(&v);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float2 f = Pack2<T>::unpack(e[q]);
                    e[q] = Pack2<T>::pack(f.x * w, f.y * w);
                }
                sts128(addr, v);
            }
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars[2]);
        const bool done = mbar_wait(&bars[3], 0, status, kStBarDone);
        tc_fence_after_sync();
        if (__all_sync(0xffffffffu, ok && done)) {   // tcgen05.ld is warp-collective
            float *S = states + (((int64_t)b * nchunks + c) * nheads + h) * (int64_t)(kP * kN);
            const int n = (warp & 3) * 32 + lane;     // TMEM lane = state index
            const int p0 = (warp >> 2) * 32;          // which half of the head's columns this warp stores
            float v[32];
            tmem_ld32(tmem + ((uint32_t)((warp & 3) * 32) << 16) + p0, v);
#pragma unroll
            for (int j = 0; j < 32; ++j) S[(p0 + j) * kN + n] = v[j];
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 8) tmem_dealloc(tmem, 64);
}

// ====================================================================================== state stream
// Chunk states and the inter-chunk recurrence in ONE pass: grid (nheads, batch), a CTA walks the chunks of its
// (batch, head) in order, so the fp32 chunk states never leave the SM.  Per chunk c it forms
// S_c^T[n,p] = sum_k B[k,n] (w_k x[k,p]) on the tensor core exactly as the chunk-state kernel does, keeps the
// running state H in registers (thread = one state index n and 16 columns p), stores the state ENTERING chunk
// c as a 16-bit [n][p] tile (the B operand of the output kernel's C.H product, fetched there by TMA) and
// folds H <- exp(dA_last_c) H + S_c.  After the last chunk H is the final state.
// 576 threads: warps 0-15 weight the x rows and own the running state (16 warps because this work is a chain
// of shared-memory and TMEM round trips that only more warps in flight can hide), warp 16 issues TMA loads,
// warp 17 the MMAs.  Shared memory: stages of half a chunk (B 2 x 16 KB + x 16 KB per head for 128 steps) and one
// 16 KB state tile per head; TMEM: two accumulators of 64 columns per head, so the MMAs of chunk c overlap the fold
// of chunk c-1.  A CTA serves one head or two heads of one group (template parameter HEADS): with two, the B tile
// is fetched and read by the tensor core once for both (N = 128).
constexpr int kStreamMinUnits = 74;                    // (batch, head) units from which one CTA per unit pays: half the SMs
constexpr int kStreamWarps = 16;                       // element-wise warps
constexpr int kStreamThreads = (kStreamWarps + 2) * 32;
// HEADS heads of one group per CTA share the B tile: one stage is half a chunk of B (2 x 16 KB) and of every head's
// x (16 KB each).  One head: 4 stages of 48 KB; two heads: 3 stages of 64 KB; plus one 16 KB state tile per head.
template <int HEADS> struct StreamCfg {
    static constexpr uint32_t kStage = 2 * 16384 + HEADS * 16384;
    static constexpr int kStages = HEADS == 1 ? 4 : 3;
    static constexpr uint32_t kSmem = kStages * kStage + HEADS * 16384 + 256 + 1024;
};
enum { kStStreamFull = 41, kStStreamWeighted, kStStreamEmpty, kStStreamAcc, kStStreamAccEmpty };

template <typename T, int HEADS>
__global__ void __launch_bounds__(kStreamThreads, 1)
ssd_tc_state_stream_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_B,
                           const __grid_constant__ CUtensorMap tm_Hs, const float *dtb, const float *dAb, const float *initial,
                           float *final_states, float *range_decay, float *prefix_decay, float *state_copy, float *decay_copy,
                           int store_entering, int nchunks, int nheads, int heads_per_group, int unit0, const int32_t *seq_idx, int seqlen,
                           int *status)
{
    using Cfg = StreamCfg<HEADS>;
    constexpr int NST = Cfg::kStages;
    constexpr uint32_t kStage = Cfg::kStage;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *sm = align1024(smem_raw);
    uint8_t *tile = sm + NST * kStage;
    uint64_t *bars = reinterpret_cast<uint64_t *>(tile + HEADS * 16384);
    uint64_t *full = bars, *weighted = bars + 4, *empty = bars + 8, *acc_full = bars + 12, *acc_empty = bars + 14;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 16);
    // work unit = HEADS consecutive heads of one batch row (all of one group); units are numbered batch-major
    const int unit = unit0 + blockIdx.x, upb = nheads / HEADS;
    const int h0 = (unit % upb) * HEADS, b = unit / upb;
    const int g = h0 / heads_per_group;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nstages = 2 * nchunks;
    if (threadIdx.x == kStreamWarps * 32) {
        for (int i = 0; i < NST; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&weighted[i], kStreamWarps);      // one arrival per element-wise warp
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], kStreamWarps);
        }
        mbar_fence_init();
    }
    if (warp == kStreamWarps) tmem_alloc(tmem_slot, 128 * HEADS);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    pdl_trigger();
    // x and B are the caller's and may be loaded; dt and dA come from the launch before this one
    if (warp != kStreamWarps) pdl_wait();

    if (warp == kStreamWarps) {
        // ------------------------------------------------------------------ TMA loads, up to NST stages ahead
        if (lane == 0) {
            int issued = 0;
            for (int i = 0; i < nstages; ++i) {
                const int st = i % NST;
                if (i >= NST && !mbar_wait(&empty[st], ((i / NST) - 1) & 1, status, kStStreamEmpty)) break;
                uint8_t *dst = sm + st * kStage;
                const int t0 = i * 128;
                mbar_expect_tx(&full[st], kStage);
                for (int hd = 0; hd < HEADS; ++hd)
                    tma_load_4d(dst + 2 * 16384 + hd * 16384, &tm_x, &full[st], 0, h0 + hd, t0, b);
                for (int kb = 0; kb < 2; ++kb) tma_load_4d(dst + kb * 16384, &tm_B, &full[st], kb * 64, g, t0, b);
                ++issued;
            }
            // nothing may still be landing in this CTA's shared memory when it exits
            for (int i = issued > NST ? issued - NST : 0; i < issued; ++i) mbar_wait(&full[i % NST], (i / NST) & 1, status, kStStreamFull);
        }
    } else if (warp == kStreamWarps + 1) {
        // ------------------------------------------------------------------ MMAs: S^T[n, (head, p)] += B[k, n] xw[k, (head, p)]
        const uint32_t idesc = instr_desc_f16(128, 64 * HEADS, Fmt<T>::v, 1, 1), tm = warp_uniform(tmem);
        const uint64_t desc_B = smem_desc_sw128(smem_u32(sm), 16384, 1024), desc_x = smem_desc_sw128(smem_u32(sm) + 2 * 16384, 16384, 1024);
        bool ok = true;
        int st = 0, phase = 0;           // stage, and how often the ring has gone round
#pragma unroll 1
        for (int c = 0; c < nchunks && ok; ++c) {
            const uint32_t acc = tm + (uint32_t)(c & 1) * 64 * HEADS;
            if (c >= 2) ok = __all_sync(0xffffffffu, mbar_wait(&acc_empty[c & 1], ((c >> 1) - 1) & 1, status, kStStreamAccEmpty));
#pragma unroll 1
            for (int half = 0; half < 2; ++half) {
                ok = ok && __all_sync(0xffffffffu, mbar_wait(&weighted[st], phase & 1, status, kStStreamWeighted));
                if (!ok) break;
                tc_fence_after_sync();
                if (elect_one()) {
                    const uint64_t off = st * (kStage / 16);
                    mma_steps_ss(8, acc, desc_B + off, 128, desc_x + off, 128, idesc, half > 0);
                    mma_commit(&empty[st]);
                    if (half) mma_commit(&acc_full[c & 1]);
                }
                __syncwarp();
                if (++st == NST) { st = 0; ++phase; }
            }
        }
    } else {
        // ------------------------------------------------------------------ element-wise warps
        const int tid = threadIdx.x;
        // weighting: the 512 threads split into HEADS groups; a group's threads share out the 128 rows x 8 chunks
        // of its head's x tile
        constexpr int TPH = kStreamWarps * 32 / HEADS, TPR = TPH / 128, NCH = 8 / TPR;
        const int whead = tid / TPH, wt = tid % TPH;
        const int r = wt / TPR, cq = (wt % TPR) * NCH;       // my x row inside a stage and my first 16-byte chunk of it
        const int n = (warp & 3) * 32 + lane;                // TMEM lane = state index
        const int p0 = (warp >> 2) * 16;                     // my quarter of every head's columns
        // (batch row, head) of mine, and their first elements for my n and p0 in a (batch, head, headdim, dstate) tensor
        int64_t bh[HEADS], elem0[HEADS];
#pragma unroll
        for (int hd = 0; hd < HEADS; ++hd) {
            bh[hd] = (int64_t)b * nheads + h0 + hd;
            elem0[hd] = (bh[hd] * kP + p0) * kN + n;
        }
        float H[HEADS][16];
#pragma unroll
        for (int hd = 0; hd < HEADS; ++hd)
#pragma unroll
            for (int j = 0; j < 16; ++j) H[hd][j] = initial ? initial[elem0[hd] + j * kN] : 0.f;
        // per chunk: dA and dt of my two x rows (my weighting head), and every head's dA at the end of the chunk.
        // Packed sequences: a row of another sequence than the chunk's last weighs nothing (dt = 0), and a chunk
        // whose last step belongs to another sequence than the previous chunk's carries nothing over (decay 0).
        const int32_t *sid = seq_idx ? seq_idx + (int64_t)b * seqlen : nullptr;
        const int64_t mine = bh[HEADS == 2 && whead ? HEADS - 1 : 0] * nchunks * kQ + r;
        const float *dA_mine = dAb + mine, *dt_mine = dtb + mine;
        auto scalars = [&](int c, float (&v)[5 + HEADS]) {
            const float *dAc = dA_mine + (int64_t)c * kQ, *dtc = dt_mine + (int64_t)c * kQ;
            v[0] = dAc[0]; v[1] = dtc[0]; v[2] = dAc[128]; v[3] = dtc[128];
#pragma unroll
            for (int hd = 0; hd < HEADS; ++hd) v[4 + hd] = dAb[bh[hd] * nchunks * kQ + (int64_t)c * kQ + kQ - 1];
            v[4 + HEADS] = 1.f;         // 0 when nothing carries over into the state after this chunk
            if (sid) {
                const int t_last = min(c * kQ + kQ, seqlen) - 1;
                const int s_last = sid[t_last], s_prev = c > 0 ? sid[c * kQ - 1] : 0;
                const int t0r = c * kQ + r, t1r = t0r + 128;
                if (t0r < seqlen && sid[t0r] != s_last) v[1] = 0.f;
                if (t1r < seqlen && sid[t1r] != s_last) v[3] = 0.f;
                if (s_last != s_prev) v[4 + HEADS] = 0.f;
            }
        };
        float nxt[5 + HEADS];
        scalars(0, nxt);
        float dec_prev[HEADS], dA_total[HEADS];
#pragma unroll
        for (int hd = 0; hd < HEADS; ++hd) dec_prev[hd] = 0.f, dA_total[hd] = 0.f;
        bool ok = true;
        auto fold = [&](int c) {      // H <- dec H + S_c once the MMAs of chunk c have completed
            ok = __all_sync(0xffffffffu, ok && mbar_wait(&acc_full[c & 1], (c >> 1) & 1, status, kStStreamAcc));   // tcgen05.ld is warp-collective
            if (!ok) return;
            tc_fence_after_sync();
            float v[HEADS][16];
#pragma unroll
            for (int hd = 0; hd < HEADS; ++hd)
                tmem_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(c & 1) * 64 * HEADS + hd * 64 + p0, v[hd]);
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[c & 1]);
#pragma unroll
            for (int hd = 0; hd < HEADS; ++hd)
#pragma unroll
                for (int j = 0; j < 16; ++j) H[hd][j] = fmaf(dec_prev[hd], H[hd][j], v[hd][j]);
        };
        for (int c = 0; c < nchunks && ok; ++c) {
            float cur[5 + HEADS];
#pragma unroll
            for (int q = 0; q < 5 + HEADS; ++q) cur[q] = nxt[q];
            if (c + 1 < nchunks) scalars(c + 1, nxt);
            float my_last = cur[4];
#pragma unroll
            for (int hd = 1; hd < HEADS; ++hd) my_last = whead == hd ? cur[4 + hd] : my_last;
            // weight my x rows of both halves: w_k = exp(dA_last - dA_k) dt_k
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int i = 2 * c + half, st = i % NST;
                const float w = __expf(fminf(my_last - cur[2 * half], 0.f)) * cur[2 * half + 1];
                ok = ok && mbar_wait(&full[st], (i / NST) & 1, status, kStStreamFull);
                if (ok) {
                    const uint32_t base = smem_u32(sm + st * kStage + 2 * 16384 + whead * 16384) + r * 128;
#pragma unroll
                    for (int ch = 0; ch < NCH; ++ch) {
                        const uint32_t addr = base + (((cq + ch) ^ (r & 7)) << 4);
                        uint4 v = lds128(addr);
                        uint32_t *e = reinterpret_cast<uint32_t *>(&v);
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const float2 f = Pack2<T>::unpack(e[q]);
                            e[q] = Pack2<T>::pack(f.x * w, f.y * w);
                        }
                        sts128(addr, v);
                    }
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0 && ok) mbar_arrive(&weighted[st]);
            }
            if (c > 0) fold(c - 1);
#pragma unroll
            for (int hd = 0; hd < HEADS; ++hd) {
                dec_prev[hd] = __expf(cur[4 + hd]) * cur[4 + HEADS];
                if (tid == 0 && prefix_decay) prefix_decay[bh[hd] * nchunks + c] = __expf(dA_total[hd]);   // decay from the range start to chunk c
                dA_total[hd] += cur[4 + hd];
            }
            // the states entering chunk c leave as 16-bit [n][p] tiles (not when only the range summary is wanted)
            if (tid == 0 && store_entering) tma_store_wait_read();   // the previous stores have finished reading the tiles
            ok = stream_barrier_and(ok);                     // from here on every element-wise warp agrees on ok
            if (!ok) break;
            if (store_entering) {
#pragma unroll
                for (int hd = 0; hd < HEADS; ++hd) {
                    const uint32_t row = smem_u32(tile + hd * 16384) + n * 128;
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        uint4 o;
                        o.x = Pack2<T>::pack(H[hd][8 * q + 0], H[hd][8 * q + 1]);
                        o.y = Pack2<T>::pack(H[hd][8 * q + 2], H[hd][8 * q + 3]);
                        o.z = Pack2<T>::pack(H[hd][8 * q + 4], H[hd][8 * q + 5]);
                        o.w = Pack2<T>::pack(H[hd][8 * q + 6], H[hd][8 * q + 7]);
                        sts128(row + ((((p0 >> 3) + q) ^ (n & 7)) << 4), o);
                    }
                }
                fence_proxy_async();
                asm volatile("bar.sync 1, 512;" ::: "memory");
                if (tid == 0) {
                    for (int hd = 0; hd < HEADS; ++hd)
                        tma_store_3d(&tm_Hs, tile + hd * 16384, 0, 0, (int)((((int64_t)b * nchunks + c) * nheads) + h0 + hd));
                    tma_store_commit();
                }
            }
        }
        if (ok) fold(nchunks - 1);
#pragma unroll
        for (int hd = 0; hd < HEADS; ++hd) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                if (!ok) continue;
                if (final_states) final_states[elem0[hd] + j * kN] = H[hd][j];
                if (state_copy) state_copy[elem0[hd] + j * kN] = H[hd][j];
            }
        }
        if (tid == 0) {
            tma_store_wait_read();
            for (int hd = 0; hd < HEADS; ++hd) {
                if (ok && range_decay) range_decay[bh[hd]] = __expf(dA_total[hd]);
                if (ok && decay_copy) decay_copy[bh[hd]] = __expf(dA_total[hd]);
            }
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == kStreamWarps) tmem_dealloc(tmem, 128 * HEADS);
}

// ====================================================================================== chunk output
// out[m] = exp(dA_m) C_m . H_c + sum_{k <= m} (C_m . B_k) exp(dA_m - dA_k) dt_k x_k + D x_m, gated by silu(z_m).
//
// Per (chunk of 256 steps, head) x, z and the entering state H come in (32 + 32 + 16 KB) and out leaves (32 KB), 1.15 GB for batch 8, 4096
// steps, 80 heads: 0.18 ms of DRAM.  A kernel with one CTA per (chunk, head, 128 rows) fetched C and C.B^T again for every head: 136 KB
// into shared memory per 128 rows, and each of its short CTAs paid the whole latency chain (0.365 ms for that shape).  Here one persistent
// CTA per SM walks over the HEADS of a (chunk, group) "unit": C stays in shared memory, C.B^T is formed once per unit on the tensor core
// and stays in REGISTERS (causal and sequence masks already applied), so that a head costs its own x, z, H and out and nothing else.  The
// (unit, head) pairs are split evenly over the CTAs in unit order, so a CTA meets few units and no wave is left nearly empty.
//
// 768 threads, in roles that hand a head on to one another.  Mask warps, four for the chunk's first 128 rows and eight for its last (which
// have 2.6 times as much of the mask), hold C.B^T and form the A operand in tensor memory, a half of the steps at a time, so that the MMAs
// of one half run while the other is formed; they are a head ahead of the output warps, four per row block, which finish the accumulators.
// A warp has rows 32 (w % 4) .. of its block -- its tensor-memory lanes.  Mask warps have four 32-column ranges of C.B^T in either block,
// which makes them one piece of code.  Then one warp for TMA loads and stores, one MMA warp per row block, one warp for the per-head scalars.
//   Y1 = C . H (A = C from shared memory), Y2 = (CB o L) . x (A from tensor memory), out = exp(dA_m) Y1 + Y2 + D x
// Tensor memory: rows 0-127: accumulators Y1 | Y2 [0, 128), A [128, 192); rows 128-255: [192, 320), A [320, 448).  While a unit
// starts, C.B^T in fp32 takes the place of a row block's regions (128 and 256 columns).
// Shared memory: C 64 KB, two stages of x 32 KB | H 16 KB | z 32 KB; the output tile replaces
// z in place and leaves through a TMA store.  While a unit starts, B lies in the x parts of the two stages.
//
// What bounds it: a head takes the output warps' pass over its accumulators (4200 cycles) plus the MMAs that wait for them (1400); the mask
// warps have a third of the time to spare.  269 us for the shape above (321 with twelve warps that did both, one after the other), 2.7 ms for
// 262144 steps of 128 heads (3.28).  C.B^T takes 64 registers of a thread, and shared memory leaves the L1 cache nothing, so a spilled
// register comes back from L2: the roles share the block's registers out between them (setmaxnreg).  What is still spilled, 72 bytes a
// thread, is the mask warps' (built with the bodies of the others taken out, 72; the output warps alone 0), who have time to spare.
// Instruction fetch is what bounds the roles themselves: loops are rolled, waits short, places advanced without divisions.  The output loop
// unrolled twice takes 273 us, eight times 320; with the next accumulators requested ahead 289.
//
// Decay mask, per thread one row m and ranges of 8 columns k:
//   L[m,k] = exp(dA_m - dA_ref) * (exp(dA_ref - dA_k) dt_k), ref = last column of the range
// with one exponential per row and range; the column factors are formed once per head by the scalar warp.  dA is
// non-increasing (A <= 0, dt >= 0), so both exponents are <= 0 below the diagonal; in the range that holds the diagonal the row
// factor is at most 2^kMaxDiagSpan and the columns past the diagonal meet a zero of C.B^T.  A 32-column range in which that
// fails (a steeper decay, or dA not monotone) is done element by element: exp(min(dA_m - dA_k, 0)) dt_k.
// Both exponents are differences of the same rounded products dA log2 e, so that those of a step's weight on itself cancel exactly: the
// products are kept from being contracted into the differences, which would leave a residue of half an ulp of dA.
// The factors are rounded to the input dtype and applied with packed 16-bit multiplies.
constexpr float kMaxDiagSpan = 100.f;
constexpr int kMaskWarps0 = 4, kMaskWarps1 = 8, kRowWarps = 4;      // that form the A operand, per row block; that finish the outputs of a row block
constexpr int kOutWarp = kMaskWarps0 + kMaskWarps1, kHelperWarp = kOutWarp + 2 * kRowWarps, kOutThreads = (kHelperWarp + 4) * 32;
constexpr int kMaskRegs = 104, kOutRegs = 64, kHelperRegs = 40, kOutLaunchRegs = 80;       // of a thread, by role; as the block is launched
static_assert(kMaskRegs * kOutWarp + kOutRegs * 2 * kRowWarps + kHelperRegs * 4 <= kOutLaunchRegs * kOutThreads / 32, "an increase would wait for ever");
constexpr uint32_t kAcc0 = 0, kA0 = 128, kAcc1 = 192, kA1 = 320;       // places in tensor memory
struct OutCfg {
    static constexpr uint32_t kC = 4 * 16384, kH = 2 * 8192, kStage = 32768 + kH + 32768;
    static constexpr uint32_t kScal = 1024 + 128 + 64;  // column factors, 32 refs, then flags
    static constexpr uint32_t kSmem = kC + 2 * kStage + 2 * kScal + 256;
};
static_assert(OutCfg::kSmem <= 227 * 1024, "shared memory");
enum { kStOutUnit = 21, kStOutCb, kStOutCbRead, kStOutStage, kStOutGate, kStOutA, kStOutAcc, kStOutAccFree, kStOutScal, kStOutScalFree, kStOutTile, kStOutAFree };
enum { kBarCb = 0, kBarCbRead = 2, kBarAcc = 4, kBarAccFree = 6, kBarXh = 8, kBarZ = 10, kBarScal = 12, kBarScalFree = 14, kBarOut = 16, kBarUnit = 20,
       kBarA = 21, kBarAFree = 25, kBars = 29 };

// Place of a (unit, head) pair; advanced without divisions.  Every role of the kernel walks the same list.
struct OutWalk {
    int b, c, g, hv, h;             // batch row, chunk, group; head inside the group; head
    bool enter;                     // first pair of this CTA in the unit (b, c, g)
    __device__ __forceinline__ OutWalk(int it, int ngroups, int nchunks, int hpu)
    {
        const int u = it / hpu, bc = u / ngroups;
        hv = it - u * hpu;
        g = u - bc * ngroups;
        b = bc / nchunks;
        c = bc - b * nchunks;
        h = g * hpu + hv;
        enter = true;
    }
    __device__ __forceinline__ void step(int ngroups, int nchunks, int hpu)
    {
        enter = false;
        ++h;
        if (++hv == hpu) {
            hv = 0;
            enter = true;
            if (++g == ngroups) {
                g = 0;
                h = 0;
                if (++c == nchunks) { c = 0; ++b; }
            }
        }
    }
    __device__ __forceinline__ int row_blocks(int seqlen) const { return seqlen - c * kQ > 128 ? 2 : 1; }     // that hold steps of the sequence
};

// DM: no D, one per head, one per column of a head.  Z: with a gate.
enum { kNoD, kHeadD, kColumnD };
template <typename T, int DM, bool Z>
__global__ void __launch_bounds__(kOutThreads, 1)
ssd_tc_output_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_C, const __grid_constant__ CUtensorMap tm_B,
                     const __grid_constant__ CUtensorMap tm_H, const __grid_constant__ CUtensorMap tm_z, const __grid_constant__ CUtensorMap tm_out,
                     const float *dtb, const float *dAb, const float *Dp, int nchunks, int nheads, int ngroups, int seqlen, int total_items, int h_np, const uint8_t *seq_start, const uint8_t *seq_carry, int *status)
{
    using Cfg = OutCfg;
    extern __shared__ __align__(1024) uint8_t sm[];
    uint8_t *Cs = sm;                                           // [row block][state half] tiles of [128][64]
    uint8_t *stages = sm + Cfg::kC;
    auto st_x = [&](int s) { return stages + s * Cfg::kStage; };
    auto st_H = [&](int s) { return stages + s * Cfg::kStage + 32768; };
    auto st_z = [&](int s) { return stages + s * Cfg::kStage + 32768 + Cfg::kH; };
    uint8_t *scal = stages + 2 * Cfg::kStage;
    uint64_t *bars = reinterpret_cast<uint64_t *>(scal + 2 * Cfg::kScal);
    // Barriers.  [row block]: C.B^T formed / read, accumulators complete / read; [stage]: x and H, z landed; scalars in place / read;
    // output tile complete (stage * 2 + row block); C and B of a unit landed; A in place / read (row block * 2 + half of the steps)
    uint64_t *b_cb = bars + kBarCb, *b_cbread = bars + kBarCbRead, *b_acc = bars + kBarAcc, *b_accfree = bars + kBarAccFree, *b_xh = bars + kBarXh,
             *b_z = bars + kBarZ, *b_scal = bars + kBarScal, *b_scalfree = bars + kBarScalFree, *b_out = bars + kBarOut, *b_unit = bars + kBarUnit,
             *b_A = bars + kBarA, *b_Afree = bars + kBarAFree;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + kBars);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int hpu = nheads / ngroups;                           // heads of a group
    const int it0 = (int)((int64_t)total_items * blockIdx.x / gridDim.x), count = (int)((int64_t)total_items * (blockIdx.x + 1) / gridDim.x) - it0;
    if (threadIdx.x == kHelperWarp * 32) {
        for (int i = 0; i < 2; ++i) {
            const int warps = i ? kMaskWarps1 : kMaskWarps0;
            mbar_init(&b_cb[i], 1);
            mbar_init(&b_cbread[i], warps);
            mbar_init(&b_acc[i], 1);
            mbar_init(&b_accfree[i], kRowWarps);
            mbar_init(&b_xh[i], 1);
            mbar_init(&b_z[i], 1);
            mbar_init(&b_scal[i], 1);
            mbar_init(&b_scalfree[i], kMaskWarps0 + kMaskWarps1);
            mbar_init(&b_out[2 * i], kRowWarps);
            mbar_init(&b_out[2 * i + 1], kRowWarps);
        }
        for (int i = 0; i < 4; ++i) {
            mbar_init(&b_A[i], i < 2 ? kMaskWarps0 : kMaskWarps1);
            mbar_init(&b_Afree[i], 1);
        }
        mbar_init(b_unit, 1);
        mbar_fence_init();
        if (smem_u32(sm) & 1023u) atomicCAS(status, 0, kStSmemAlign);   // the swizzled tiles assume a 1 KB aligned base
    }
    if (warp == kHelperWarp + 1) tmem_alloc(tmem_slot, 512);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    const bool aligned = (smem_u32(sm) & 1023u) == 0;
    pdl_trigger();
    pdl_wait();

    constexpr uint32_t kBarOff = Cfg::kC + 2 * Cfg::kStage + 2 * Cfg::kScal;
    if (!aligned) {
        // nothing runs (the status says so)
    } else if (warp < kOutWarp) {
        // ------------------------------------------------------------------ mask: A = CB o L
        registers_up<kMaskRegs>();
        constexpr int NR = 4;                                // 32-column ranges of the mask per thread
        const int rb = warp < kMaskWarps0 ? 0 : 1;           // my row block
        const int rq = warp & 3, cq_ = rb ? (warp - kMaskWarps0) >> 2 : 0;       // my rows of it, my half of the columns
        const uint32_t tlane_ = tmem + ((uint32_t)(rq * 32) << 16), smem_ = smem_u32(sm);
        const int r = rb * 128 + rq * 32 + lane;             // my row of the chunk
        bool ok = true;
        uint32_t cb[NR][16];                                 // my ranges of C.B^T, packed, masked
        const float *dA = dAb;                               // of the current (batch row, head, chunk)
        float dA_next = 0.f;
        int left = 0;                                        // heads left in the unit
        bool rows = true;                                    // the chunk reaches my block
        int nunits = 0, item = 0;

#pragma unroll 1
        for (int seq = 0; seq < count; ++seq) {
            // everything below is derived from these three; hidden from the compiler, which would otherwise keep dozens of addresses
            // and range numbers over the loop -- in spilled registers
            uint32_t smb = smem_, tlane = tlane_;
            int cq = cq_;
            asm volatile("" : "+r"(smb), "+r"(tlane), "+r"(cq));
            auto bar = [&](int k) { return smb + kBarOff + 8 * k; };
            // range t of mine: columns 32 j .. of the chunk (one tile of 128 columns, or a half of each of two)
            auto range = [&](int t) { return rb ? (t >> 1) * 4 + 2 * cq + (t & 1) : t; };
            if (left == 0) {
                // a new unit: C.B^T moves from tensor memory into registers
                const OutWalk w(it0 + seq, ngroups, nchunks, hpu);
                left = hpu - w.hv;
                rows = rb < w.row_blocks(seqlen);
                dA = dAb + (((int64_t)w.b * nheads + w.h) * nchunks + w.c) * kQ;
                int lo = 0;                                  // first column of my row's sequence inside the chunk
                if (rows) {
                    if (seq_start) lo = seq_start[((int64_t)w.b * nchunks + w.c) * kQ + r];
                    dA_next = dA[r];
                }
                // (every unit completes these barriers once, whatever its row blocks, so that nobody falls a phase behind)
                ok = __all_sync(0xffffffffu, mbar_wait(bar(kBarCb + rb), nunits & 1, status, kStOutCb));      // tcgen05.ld is warp-collective
                ++nunits;
                if (!ok) break;
                if (rows) {
                    tc_fence_after_sync();
                    const uint32_t from = tlane + (rb ? kAcc1 : kAcc0);
#pragma unroll
                    for (int t = 0; t < NR; ++t) {
                        // columns [lo, m] of the chunk stay
                        const int k0 = 32 * range(t), first = lo - k0, last = r - k0;
                        uint32_t keep = last < 0 ? 0u : last >= 31 ? ~0u : (2u << last) - 1u;
                        if (first > 0) keep &= first > 31 ? 0u : ~0u << first;
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            uint32_t v[8];
                            tmem_ld8_issue(from + k0 + 8 * e, v);
                            tmem_ld_wait(v);
#pragma unroll
                            for (int i = 0; i < 8; ++i) v[i] = keep >> (8 * e + i) & 1u ? v[i] : 0u;
#pragma unroll
                            for (int i = 0; i < 4; ++i) cb[t][4 * e + i] = Pack2<T>::pack(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
                        }
                    }
                    tc_fence_before_sync();
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(kBarCbRead + rb));
                // the A operand of the lower row block takes the place of C.B^T: no warp may write it while another still reads
                if (rb) ok = __all_sync(0xffffffffu, mbar_wait(bar(kBarCbRead + rb), (nunits - 1) & 1, status, kStOutCbRead));
                if (!ok) break;
            }
            const int s = seq & 1;
            const uint32_t sc = smb + Cfg::kC + 2 * Cfg::kStage + s * Cfg::kScal;
            ok = __all_sync(0xffffffffu, mbar_wait(bar(kBarScal + s), (seq >> 1) & 1, status, kStOutScal));
            if (!ok) break;
            --left;
            if (!rows) {                                     // no rows here in this chunk
                if (lane == 0) mbar_arrive(bar(kBarScalFree + s));
                continue;
            }
            const float dAm = __fmul_rn(dA_next, kLog2e);
            if (left) dA_next = dA[(int64_t)nchunks * kQ + r];                           // a whole head ahead of its use
            const uint32_t flags = __float_as_uint(lds32(sc + 1024 + 128));
            const uint32_t A = tlane + (rb ? kA1 : kA0);
#pragma unroll
            for (int t = 0; t < NR; ++t) {
                if ((t & 1) == 0) {      // half of the reduction: its MMAs run while the other half is formed, and before that the ones that read what is there now
                    if (item) ok = __all_sync(0xffffffffu, mbar_wait(bar(kBarAFree + 2 * rb + t / 2), (item - 1) & 1, status, kStOutAFree));
                    if (!ok) break;
                    tc_fence_after_sync();
                }
                const int j = range(t);
                const uint32_t dst = A + 16 * j, ck = sc + 128 * j;
                // (every branch goes one way for the whole warp: tcgen05.ld and .st are warp-collective)
                if (j - 4 * rb > rq) {                       // wholly past the diagonal
                    const uint32_t none[8] = {};
                    tmem_st8_issue(dst, none);
                    tmem_st8_issue(dst + 8, none);
                } else if ((flags >> (4 * j)) & 1) {
                    float f[4];
                    lds128f(sc + 1024 + 16 * j, f);
#pragma unroll
                    for (int g = 0; g < 4; ++g) f[g] = ex2(fminf(__fsub_rn(dAm, f[g]), kMaxDiagSpan));         // (a range past the diagonal only has to stay finite)
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        uint64_t c[8];
#pragma unroll
                        for (int i = 0; i < 4; ++i) lds_pair2(ck + 64 * half + 16 * i, c[2 * i], c[2 * i + 1]);
                        uint32_t a[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const float fg = f[2 * half + i / 4];
                            float l0, l1;
                            unpack2(mul2(pack2(fg, fg), c[i]), l0, l1);
                            if constexpr (Fmt<T>::v == 0) l0 = fminf(l0, 65504.f), l1 = fminf(l1, 65504.f);      // half precision: a factor past the diagonal must not become infinite
                            a[i] = Pack2<T>::mul(cb[t][8 * half + i], Pack2<T>::pack(l0, l1));
                        }
                        tmem_st8_issue(dst + 8 * half, a);
                    }
                } else {
                    // rare: a range that the factorised mask cannot do has its decays formed element by element, parked where its A words go
                    // (in a rolled loop, so that it costs neither registers nor instruction cache)
#pragma unroll 1
                    for (int i = 0; i < 16; ++i) {
                        const float2 d = *reinterpret_cast<const float2 *>(dA + 32 * j + 2 * i), w = *reinterpret_cast<const float2 *>(dtb + (dA - dAb) + 32 * j + 2 * i);
                        const float l0 = ex2(fminf(fmaf(d.x, -kLog2e, dAm), 0.f)) * w.x, l1 = ex2(fminf(fmaf(d.y, -kLog2e, dAm), 0.f)) * w.y;
                        __syncwarp();
                        tmem_st1_issue(dst + i, Pack2<T>::pack(l0, l1));
                    }
                    tmem_st_wait();
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        uint32_t a[8];
                        tmem_ld8_issue(dst + 8 * half, a);
                        tmem_ld_wait(a);
#pragma unroll
                        for (int i = 0; i < 8; ++i) a[i] = Pack2<T>::mul(cb[t][8 * half + i], a[i]);
                        tmem_st8_issue(dst + 8 * half, a);
                    }
                }
                if (t & 1) {
                    tmem_st_wait();
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar(kBarA + 2 * rb + t / 2));
                }
            }
            if (!ok) break;
            if (lane == 0) mbar_arrive(bar(kBarScalFree + s));
            dA += (int64_t)nchunks * kQ;
            ++item;
        }
    } else if (warp < kHelperWarp) {
        // ------------------------------------------------------------------ outputs: out = exp(dA_m) Y1 + Y2 + D x, gated
        registers_down<kOutRegs>();
        const int rb = (warp - kOutWarp) >> 2, rq = warp & 3;
        const uint32_t acc = tmem + ((uint32_t)(rq * 32) << 16) + (rb ? kAcc1 : kAcc0), smb = smem_u32(sm);
        const int r = rb * 128 + rq * 32 + lane;             // my row of the chunk
        auto bar = [&](int k) { return smb + kBarOff + 8 * k; };
        const float *dA = dAb;                               // of the current head
        [[maybe_unused]] const float *Dv = Dp;
        float dA_next = 0.f, D_next = 0.f;
        int left = 0, item = 0;
        bool carry = true, rows = true, ok = true;           // my row continues the sequence that ended the previous chunk; the chunk reaches my block
#pragma unroll 1
        for (int seq = 0; seq < count; ++seq) {
            if (left == 0) {
                const OutWalk w(it0 + seq, ngroups, nchunks, hpu);
                left = hpu - w.hv;
                rows = rb < w.row_blocks(seqlen);
                dA = dAb + (((int64_t)w.b * nheads + w.h) * nchunks + w.c) * kQ + r;
                if constexpr (DM != kNoD) Dv = Dp + (int64_t)w.h * (DM == kColumnD ? kP : 1);
                if (rows) {
                    if (seq_start) {
                        const int64_t bc = (int64_t)w.b * nchunks + w.c;
                        carry = seq_start[bc * kQ + r] == 0 && seq_carry[bc] != 0;
                    }
                    dA_next = *dA;
                    if constexpr (DM == kHeadD) D_next = *Dv;
                }
            }
            --left;
            if (!rows) continue;
            const int s = seq & 1, sph = (seq >> 1) & 1;
            const float rs = carry ? ex2(dA_next * kLog2e) : 0.f, Dh = D_next;
            if (left) {                                      // a whole head ahead of their use
                dA_next = dA[(int64_t)nchunks * kQ];
                if constexpr (DM == kHeadD) D_next = Dv[1];
            }
            dA += (int64_t)nchunks * kQ;
            const uint32_t row = smb + Cfg::kC + s * Cfg::kStage + r * 128;
            // The product first: x is there when it is, and so are the gates of all heads before.  A warp that came past the heads of a chunk
            // without rows of its block may be many phases ahead of the gate's barrier, whose parity alone does not tell it that.
            ok = mbar_wait(bar(kBarAcc + rb), item & 1, status, kStOutAcc) && mbar_wait(bar(kBarZ + s), sph, status, kStOutGate);
            ok = __all_sync(0xffffffffu, ok);                // tcgen05.ld is warp-collective
            ++item;
            if (!ok) break;
            tc_fence_after_sync();
            const uint64_t rs2 = pack2(rs, rs), D2 = pack2(Dh, Dh);
#pragma unroll 1
            for (int e8 = 0; e8 < 8; ++e8) {
                uint32_t y1[8], y2[8];
                tmem_ld8_issue(acc + e8 * 8, y1);
                tmem_ld8_issue(acc + 64 + e8 * 8, y2);
                const uint32_t xaddr = row + (uint32_t)((e8 ^ (r & 7)) << 4), zaddr = xaddr + 32768 + Cfg::kH;
                uint4 xv = make_uint4(0, 0, 0, 0), zv = make_uint4(0, 0, 0, 0);
                if constexpr (DM != kNoD) xv = lds128(xaddr);
                if constexpr (Z) zv = lds128(zaddr);
                tmem_ld_wait(y1, y2);
                uint64_t y[4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    y[i] = fma2(rs2, pack2(__uint_as_float(y1[2 * i]), __uint_as_float(y1[2 * i + 1])),
                                pack2(__uint_as_float(y2[2 * i]), __uint_as_float(y2[2 * i + 1])));
                if (e8 == 7) {
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar(kBarAccFree + rb));
                }
                if constexpr (DM != kNoD) {
                    const uint32_t xe[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 f = Pack2<T>::unpack(xe[i]);
                        uint64_t d2 = D2;
                        if constexpr (DM == kColumnD) {
                            const int pc = e8 * 8 + 2 * i;
                            d2 = pack2(Dv[pc], Dv[pc + 1]);
                        }
                        y[i] = fma2(pack2(f.x, f.y), d2, y[i]);
                    }
                }
                if constexpr (Z) {
                    const uint32_t ze[4] = {zv.x, zv.y, zv.z, zv.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 f = Pack2<T>::unpack(ze[i]);
                        if constexpr (Fmt<T>::v == 1) {      // bfloat16 output: one MUFU per gate value is accurate enough
                            const uint64_t h2 = mul2(pack2(f.x, f.y), pack2(0.5f, 0.5f));
                            float h0, h1;
                            unpack2(h2, h0, h1);
                            y[i] = mul2(y[i], fma2(h2, pack2(tanh_approx(h0), tanh_approx(h1)), h2));
                        } else {
                            y[i] = mul2(y[i], pack2(fast_silu(f.x), fast_silu(f.y)));
                        }
                    }
                }
                uint32_t o[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float a0, a1;
                    unpack2(y[i], a0, a1);
                    o[i] = Pack2<T>::pack(a0, a1);
                }
                sts128(zaddr, make_uint4(o[0], o[1], o[2], o[3]));
            }
            if constexpr (DM != kNoD) Dv += DM == kColumnD ? kP : 1;
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(kBarOut + 2 * s + rb));
        }
    } else {
        registers_down<kHelperRegs>();
        if (warp == kHelperWarp + 1 || warp == kHelperWarp + 2) {
            // ------------------------------------------------------------------ MMAs of one row block
            const int rb = (int)warp_uniform(warp) - (kHelperWarp + 1);
            OutWalk w(it0, ngroups, nchunks, hpu);
            auto step = [&] { w.step(ngroups, nchunks, hpu); };
            const uint32_t tm = warp_uniform(tmem), acc = tm + (rb ? kAcc1 : kAcc0);
            auto wait = [&](uint64_t *bar, int phase, int code) { return __all_sync(0xffffffffu, mbar_wait(bar, phase & 1, status, code)) != 0; };
            bool ok = true, rows = true;
            int nunits = 0, item = 0;
            const uint32_t idesc_cb = instr_desc_f16(128, 128, Fmt<T>::v, 0, 0) + ((uint32_t)(rb ? 128 >> 3 : 0) << 17),      // N = 128 or 256
                           idesc_y1 = instr_desc_f16(128, 64, Fmt<T>::v, 0, h_np ? 1 : 0), idesc_y2 = instr_desc_f16(128, 64, Fmt<T>::v, 0, 1);
            const uint32_t step_H = h_np ? 128 : 2;              // states along the rows of the tile, or along its columns
            const uint64_t desc_C = smem_desc_sw128(smem_u32(Cs) + rb * 2 * 16384, 16, 1024), desc_x = smem_desc_sw128(smem_u32(st_x(0)), 16, 1024),
                           desc_H = smem_desc_sw128(smem_u32(st_H(0)), 16, 1024);
#pragma unroll 1
            for (int seq = 0; seq < count && ok; ++seq, step()) {
                if (w.enter) {
                    rows = rb < w.row_blocks(seqlen);
                    ok = wait(b_unit, nunits, kStOutUnit);
                    ++nunits;
                    if (!ok) break;
                    if (rows) {
                        if (item) ok = wait(&b_accfree[rb], item - 1, kStOutAccFree);
                        if (!ok) break;
                        tc_fence_after_sync();
                        if (elect_one()) {
#pragma unroll 1
                            for (int kb = 0; kb < 2; ++kb)      // B lies in the x parts of the stages
                                mma_steps_ss(4, acc, desc_C + kb * (16384 / 16), 2, desc_x + kb * (Cfg::kStage / 16), 2, idesc_cb, kb > 0);
                            mma_commit(&b_cb[rb]);
                        }
                    } else if (lane == 0) {
                        mbar_arrive(&b_cb[rb]);
                    }
                    __syncwarp();
                    ok = wait(&b_cbread[rb], nunits - 1, kStOutCbRead);
                    if (!ok) break;
                    tc_fence_after_sync();
                }
                if (!rows) continue;
                const int s = seq & 1;
                const uint64_t off = s * (Cfg::kStage / 16);
                ok = wait(&b_xh[s], seq >> 1, kStOutStage) && (item == 0 || wait(&b_accfree[rb], item - 1, kStOutAccFree));
                if (!ok) break;
                tc_fence_after_sync();
                if (elect_one()) {
#pragma unroll 1
                    for (int kb = 0; kb < 2; ++kb)
                        mma_steps_ss(4, acc, desc_C + kb * (16384 / 16), 2, desc_H + off + kb * (8192 / 16), step_H, idesc_y1, kb > 0);
                }
                __syncwarp();
#pragma unroll 1
                for (int half = 0; half < 2; ++half) {
                    ok = wait(&b_A[2 * rb + half], item, kStOutA);
                    if (!ok) break;
                    tc_fence_after_sync();
                    if (elect_one()) {
                        const int steps = 4 * (rb + 1);
                        mma_steps_ts(steps, acc + 64, tm + (rb ? kA1 : kA0) + half * steps * 8, desc_x + off + half * steps * 128, 128, idesc_y2, half > 0);
                        mma_commit(&b_Afree[2 * rb + half]);
                        if (half) mma_commit(&b_acc[rb]);
                    }
                    __syncwarp();
                }
                ++item;
                if (!ok) break;
                __syncwarp();
            }
        } else if (warp == kHelperWarp) {
            // ------------------------------------------------------------------ TMA loads and stores
            if (lane == 0) {
                OutWalk w(it0, ngroups, nchunks, hpu);
                auto step = [&] { w.step(ngroups, nchunks, hpu); };
                bool ok = true;
                uint32_t outs = 0;                   // parities of the next completion of each b_out
                struct Pending { int b, h, t, nrb; } pend[2] = {};
                int nunits_requested = 0, seq = 0, done = 0;         // units requested; heads requested, finished
                // Heads leave in the order in which they came: the one in stage s has its output tiles stored as they are completed.  Then the
                // next head's x and H may take the place of its own at once; z, whose place the output tiles have, when these have been read.
                // A new unit starts when no head is in flight: C goes to its place, B to the x parts of the stages.
#pragma unroll 1
                while (ok) {
                    const bool have = seq < count;
                    const int keep = have && !w.enter ? 1 : 0;       // heads that may stay in flight before the next request
                    if (done + keep < seq) {
                        const int s = done & 1;
#pragma unroll 1
                        for (int rb = 0; rb < pend[s].nrb && ok; ++rb) {
                            const int k = 2 * s + rb;
                            ok = mbar_wait(&b_out[k], (outs >> k) & 1, status, kStOutTile);
                            outs ^= 1u << k;
                            if (ok) {
                                tma_store_4d(&tm_out, st_z(s) + rb * 16384, 0, pend[s].h, pend[s].t + rb * 128, pend[s].b);
                                tma_store_commit();
                            }
                        }
                        ++done;
                        continue;
                    }
                    if (!have) break;
                    const int s = seq & 1, nrb = w.row_blocks(seqlen);
                    if (w.enter) {
                        ++nunits_requested;
                        mbar_expect_tx(b_unit, nrb * 2 * 16384 + 2 * 32768);
#pragma unroll 1
                        for (int kb = 0; kb < 2; ++kb) {
#pragma unroll 1
                            for (int rb = 0; rb < nrb; ++rb) tma_load_4d(Cs + (rb * 2 + kb) * 16384, &tm_C, b_unit, kb * 64, w.g, w.c * kQ + rb * 128, w.b);
                            tma_load_4d(st_x(kb), &tm_B, b_unit, kb * 64, w.g, w.c * kQ, w.b);
                        }
#pragma unroll 1
                        for (int rb = 0; rb < 2 && ok; ++rb) ok = mbar_wait(&b_cb[rb], (nunits_requested - 1) & 1, status, kStOutCb);        // B has been read
                        if (!ok) break;
                    }
                    mbar_expect_tx(&b_xh[s], 32768 + Cfg::kH);
                    tma_load_4d(st_x(s), &tm_x, &b_xh[s], 0, w.h, w.c * kQ, w.b);
                    const int uh = (w.b * nchunks + w.c) * nheads + w.h;
                    if (h_np) tma_load_3d(st_H(s), &tm_H, &b_xh[s], 0, 0, uh);                     // [n][p] tile
                    else
#pragma unroll 1
                        for (int kb = 0; kb < 2; ++kb) tma_load_3d(st_H(s) + kb * 8192, &tm_H, &b_xh[s], kb * 64, 0, uh);   // columns n of the [p][n] state
                    tma_store_wait_read();
                    if (Z) {
                        mbar_expect_tx(&b_z[s], 32768);
                        tma_load_4d(st_z(s), &tm_z, &b_z[s], 0, w.h, w.c * kQ, w.b);
                    } else {
                        mbar_arrive(&b_z[s]);                        // the place is free
                    }
                    pend[s] = {w.b, w.h, w.c * kQ, nrb};
                    ++seq;
                    step();
                }
                tma_store_wait_read();
                if (!ok) {
                    // gave up: nothing may still be landing in this CTA's shared memory when it exits
                    if (nunits_requested) mbar_wait(b_unit, (nunits_requested - 1) & 1, status, kStOutUnit);
#pragma unroll 1
                    for (int k = seq > 2 ? seq - 2 : 0; k < seq; ++k) {
                        mbar_wait(&b_xh[k & 1], (k >> 1) & 1, status, kStOutStage);
                        if (Z) mbar_wait(&b_z[k & 1], (k >> 1) & 1, status, kStOutGate);
                    }
                }
            }
        } else {
            // ------------------------------------------------------------------ per-head scalars
            OutWalk w(it0, ngroups, nchunks, hpu);
            bool ok = true;
            float4 dA[2], dt[2];                     // of my eight steps: one range of the factorised mask
            auto request = [&]() {
                const int64_t o = (((int64_t)w.b * nheads + w.h) * nchunks + w.c) * kQ + 8 * lane;
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    dA[i] = *reinterpret_cast<const float4 *>(dAb + o + 4 * i);
                    dt[i] = *reinterpret_cast<const float4 *>(dtb + o + 4 * i);
                }
            };
            if (count > 0) request();
#pragma unroll 1
            for (int seq = 0; seq < count && ok; ++seq) {
                const int s = seq & 1;
                float *ck = reinterpret_cast<float *>(scal + s * Cfg::kScal), *ref = ck + 256;
                if (seq >= 2) ok = __all_sync(0xffffffffu, mbar_wait(&b_scalfree[s], ((seq >> 1) - 1) & 1, status, kStOutScalFree));
                if (!ok) break;
                const float a[8] = {dA[0].x, dA[0].y, dA[0].z, dA[0].w, dA[1].x, dA[1].y, dA[1].z, dA[1].w};
                const float end = __fmul_rn(a[7], kLog2e);
                float before = __shfl_up_sync(0xffffffffu, a[7], 1);                 // dA of the step before mine
                if (lane == 0) before = a[0];
                bool mono = true;
#pragma unroll
                for (int i = 0; i < 8; ++i) mono = mono && a[i] <= (i ? a[i - 1] : before) + 2e-6f * fabsf(i ? a[i - 1] : before);      // rounding of the sums aside
                auto factor = [&](int i, float t) { return ex2(__fsub_rn(end, __fmul_rn(a[i], kLog2e))) * t; };
                *reinterpret_cast<float4 *>(ck + 8 * lane) = make_float4(factor(0, dt[0].x), factor(1, dt[0].y), factor(2, dt[0].z), factor(3, dt[0].w));
                *reinterpret_cast<float4 *>(ck + 8 * lane + 4) = make_float4(factor(4, dt[1].x), factor(5, dt[1].y), factor(6, dt[1].z), factor(7, dt[1].w));
                ref[lane] = end;
                // bit 4 j: the ranges of columns 32 j .. 32 j + 31 may use the factorised mask
                uint32_t flags = __ballot_sync(0xffffffffu, a[0] * kLog2e - end <= kMaxDiagSpan);
                flags &= flags >> 1;
                flags &= flags >> 2;
                if (!__all_sync(0xffffffffu, mono)) flags = 0;
                if (lane == 0) reinterpret_cast<uint32_t *>(ref)[32] = flags;
                __syncwarp();
                if (lane == 0) mbar_arrive(&b_scal[s]);
                w.step(ngroups, nchunks, hpu);
                if (seq + 1 < count) request();
            }
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == kHelperWarp + 1) tmem_dealloc(tmem, 512);
}

// ====================================================================================== incoming state
// Sequence split, OUTPUT half: the LOCAL half stored the entering states of the range as if nothing came in.
// Adds prefix_decay[c] * S_in to each of them (16-bit [n][p] tiles) and forms the range's end state
// range_decay * S_in + S_local.  grid (ceil(nchunks / kFixChunks), nheads, batch), 256 threads; the incoming
// state of the (batch, head) is transposed once into shared memory.  Chunks whose share has decayed to nothing
// are left alone, which for fast-decaying heads is all but the first few.
constexpr int kFixChunks = 8;
template <typename T>
__global__ void __launch_bounds__(256) ssd_incoming_state_kernel(T *prev16, const float *s_in, const float *prefix_decay, const float *s_local,
                                                                  const float *range_decay, float *final_states, int nchunks, int nheads)
{
    __shared__ float sin_np[kN * (kP + 1)];      // [n][p], padded
    __shared__ float wmax[8];
    const int h = blockIdx.y, b = blockIdx.z;
    const int64_t bh = (int64_t)b * nheads + h;
    const float *src = s_in + bh * (kP * kN);
    if (blockIdx.x > 0 && prefix_decay[bh * nchunks + blockIdx.x * kFixChunks] == 0.f) return;   // decayed to zero before this CTA's chunks
    float amax = 0.f;
    for (int e = threadIdx.x; e < kP * kN; e += 256) {
        const float v = src[e];
        sin_np[(e % kN) * (kP + 1) + e / kN] = v;    // src is [p][n]
        amax = fmaxf(amax, fabsf(v));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = amax;
    if (blockIdx.x == 0 && final_states) {
        const float d = range_decay[bh];
        for (int e = threadIdx.x; e < kP * kN; e += 256) final_states[bh * (kP * kN) + e] = fmaf(d, src[e], s_local[bh * (kP * kN) + e]);
    }
    __syncthreads();
    float smax = wmax[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) smax = fmaxf(smax, wmax[i]);
    const int c0 = blockIdx.x * kFixChunks;
    for (int c = c0; c < min(c0 + kFixChunks, nchunks); ++c) {
        const float pd = prefix_decay[bh * nchunks + c];
        // the prefix decay only shrinks along the range: once the whole share is below the smallest normal number
        // nothing is left to add (infinities and NaNs in S_in still go through)
        if (pd * smax < 1.1754944e-38f) break;
        T *tile = prev16 + (((int64_t)b * nchunks + c) * nheads + h) * (kP * kN);
        for (int v = threadIdx.x; v < kP * kN / 8; v += 256) {      // 8 consecutive p of one n per step
            const int n = v / (kP / 8), p = (v % (kP / 8)) * 8;
            uint4 raw = *reinterpret_cast<const uint4 *>(tile + n * kP + p);
            uint32_t *w = reinterpret_cast<uint32_t *>(&raw);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float2 f = Pack2<T>::unpack(w[q]);
                w[q] = Pack2<T>::pack(fmaf(pd, sin_np[n * (kP + 1) + p + 2 * q], f.x), fmaf(pd, sin_np[n * (kP + 1) + p + 2 * q + 1], f.y));
            }
            *reinterpret_cast<uint4 *>(tile + n * kP + p) = raw;
        }
    }
}

bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
// TMA can walk a (batch, time, row, element) tensor of 16-bit values: strides in steps of 16 bytes, none of them 0 (a tensor
// expanded over a dimension).
bool rows_for_tma(const void *p, const int64_t *s)
{
    for (int i = 0; i < 3; ++i)
        if (s[i] <= 0 || s[i] % 8) return false;
    return aligned16(p);
}

// ====================================================================================== end states of packed sequences
// One CTA per (head, sequence): S^T[n,p] = sum over the sequence's steps in the chunk of its last token, plus the state entering that
// chunk if the sequence began earlier.  bf16 inputs: the weighted x rows are cut into three bf16 values, so that the fp32 result keeps
// fp32 products; B is exact as it is.  (Half precision would need its B cut as well: ssd_split.cu does that.)  The small products have
// a sum of their own, which keeps the tensor core's rounding of sums out of them.  Tiles of ROWS rows that hold no step of the sequence are
// skipped.  A CTA is a chain of copy, cut and MMAs per tile between two ends: tiles of 64 rows let four CTAs share an SM, which pays where
// there are that many (40 sequences x 48 heads: 130 us a call with 128 rows, 113 with 64; x 128 heads 318 / 292; 20 x 64 407 / 370; 23 x 80 185 / 184),
// tiles of 128 make the chain shorter (3 x 24: 44 / 48; 5 x 32: 284 / 293; 8 x 80 336 / 338).  2500 us with one thread per element (23 x 80).
constexpr int kVarThreads = 288;
template <int ROWS> constexpr uint32_t kVarTile = ROWS * 128;                            // [rows][64]
template <int ROWS> constexpr uint32_t kVarSmem = 5 * kVarTile<ROWS> + 64 + 1024;        // of B two, of x three parts
template <int ROWS>
__global__ void __launch_bounds__(kVarThreads, ROWS == 64 ? 4 : 2) ssd_tc_varlen_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_B,
                                                                    const float *dtb, const float *dAb, const int32_t *cu_seqlens, float *varlen,
                                                                    const __nv_bfloat16 *prev16, int prev_np, int nchunks, int nheads, int heads_per_group,
                                                                    int seqlen, int *status)
{
    using T = __nv_bfloat16;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *sm = align1024(smem_raw);
    uint8_t *Bs = sm, *xs = sm + 2 * kVarTile<ROWS>;
    uint64_t *bars = reinterpret_cast<uint64_t *>(xs + 3 * kVarTile<ROWS>);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 3);
    const int h = blockIdx.x, sq = blockIdx.y;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int start = cu_seqlens[sq], end = cu_seqlens[sq + 1];
    const bool empty = end <= start || end > seqlen || start < 0;
    const int c = empty ? 0 : (end - 1) / kQ, t0 = c * kQ;
    const int k0 = max(start - t0, 0), k1 = empty ? 0 : end - t0;     // rows [k0, k1) of the chunk
    if (threadIdx.x == 256) {
        mbar_init(&bars[0], 1);      // tiles landed
        mbar_init(&bars[1], 8);      // rows weighted
        mbar_init(&bars[2], 1);      // MMAs done
        mbar_fence_init();
    }
    if (warp == 8) tmem_alloc(tmem_slot, 128);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    pdl_wait();
    const float *dAc = dAb + ((int64_t)h * nchunks + c) * kQ, *dtc = dtb + ((int64_t)h * nchunks + c) * kQ;
    const float dA_end = empty ? 0.f : dAc[k1 - 1];
    // my part of the state that enters the chunk (a row of its [n][p] tile; asked for now, needed last)
    const int n = (warp & 3) * 32 + lane, p0 = ((warp >> 2) & 1) * 32;
    const bool entering = !empty && start < t0 && warp < 8;
    const T *H = prev16 + ((int64_t)c * nheads + h) * (kP * kN);
    uint4 hv[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) hv[q] = entering && prev_np ? reinterpret_cast<const uint4 *>(H + n * 64 + p0)[q] : make_uint4(0, 0, 0, 0);
    bool ok = true;
    int round = 0;
#pragma unroll 1
    for (int r_first = 0; r_first < kQ && ok; r_first += ROWS) {
        if (k1 <= r_first || k0 >= r_first + ROWS) continue;
        if (warp == 8) {
            if (lane == 0) {
                mbar_expect_tx(&bars[0], 3 * kVarTile<ROWS>);
                tma_load_4d(xs, &tm_x, &bars[0], 0, h, t0 + r_first, 0);
                for (int kb = 0; kb < 2; ++kb) tma_load_4d(Bs + kb * kVarTile<ROWS>, &tm_B, &bars[0], kb * 64, h / heads_per_group, t0 + r_first, 0);
            }
            __syncwarp();
            ok = __all_sync(0xffffffffu, mbar_wait(&bars[1], round & 1, status, kStBarScaled) && mbar_wait(&bars[0], round & 1, status, kStBarB));
            tc_fence_after_sync();
            const uint32_t idesc = instr_desc_f16(128, 64, 1, 1, 1), tm = warp_uniform(tmem);
            const uint64_t dB = smem_desc_sw128(smem_u32(Bs), kVarTile<ROWS>, 1024), dx = smem_desc_sw128(smem_u32(xs), 16, 1024);
            if (elect_one()) {
                if (ok) {
#pragma unroll 1
                    for (int part = 0; part < 3; ++part)
                        mma_steps_ss(ROWS / 16, part ? tm + 64 : tm, dB, 128, dx + part * (kVarTile<ROWS> / 16), 128, idesc, round > 0 || part == 2);
                }
                mma_commit(&bars[2]);
            }
            __syncwarp();
            ok = __all_sync(0xffffffffu, mbar_wait(&bars[2], round & 1, status, kStBarDone)) && ok;
        } else {
            constexpr int TPR = 256 / ROWS, NC = 8 / TPR;       // threads per row, and 16-byte chunks of each
            const int r = threadIdx.x / TPR, k = r_first + r, cq = (threadIdx.x % TPR) * NC;
            const bool mine = k >= k0 && k < k1;
            const float w = mine ? __expf(fminf(dA_end - dAc[k], 0.f)) * dtc[k] : 0.f;
            ok = mbar_wait(&bars[0], round & 1, status, kStBarX);
            // where B is infinite the later parts of x, which may have the other sign or be zero, are made tiny and of the first one's
            bool bad = false;
            if (ok) {
#pragma unroll
                for (int ch = 0; ch < 2 * NC; ++ch) {
                    const uint4 v = lds128(smem_u32(Bs) + (ch / NC) * kVarTile<ROWS> + r * 128 + (((cq + ch % NC) ^ (r & 7)) << 4));
                    const uint32_t m = __vmaxu2(__vmaxu2(v.x & 0x7fff7fffu, v.y & 0x7fff7fffu), __vmaxu2(v.z & 0x7fff7fffu, v.w & 0x7fff7fffu));
                    bad = bad || (m & 0xffffu) >= 0x7f80u || (m >> 16) >= 0x7f80u;
                }
            }
            bad = __shfl_xor_sync(0xffffffffu, bad, 1) || bad;
            if (TPR == 4) bad = __shfl_xor_sync(0xffffffffu, bad, 2) || bad;
            if (ok) {
#pragma unroll
                for (int ch = 0; ch < NC; ++ch) {
                    const uint32_t off = r * 128 + (((cq + ch) ^ (r & 7)) << 4);
                    if (!mine) {        // steps of other sequences count for nothing, infinite B included
                        sts128(smem_u32(Bs) + off, make_uint4(0, 0, 0, 0));
                        sts128(smem_u32(Bs) + kVarTile<ROWS> + off, make_uint4(0, 0, 0, 0));
                    }
                    const uint4 v = mine ? lds128(smem_u32(xs) + off) : make_uint4(0, 0, 0, 0);
                    const uint32_t e[4] = {v.x, v.y, v.z, v.w};
                    uint32_t part[3][4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const float2 f = Pack2<T>::unpack(e[q]);
                        float a0 = f.x * w, a1 = f.y * w;
#pragma unroll
                        for (int p = 0; p < 3; ++p) {
                            part[p][q] = bad && p > 0 ? (part[0][q] & 0x80008000u) | 0x01000100u : Pack2<T>::pack(a0, a1);
                            const float2 g = Pack2<T>::unpack(part[p][q]);
                            a0 = isinf(g.x) ? 0.f : a0 - g.x;
                            a1 = isinf(g.y) ? 0.f : a1 - g.y;
                        }
                    }
#pragma unroll
                    for (int p = 0; p < 3; ++p) sts128(smem_u32(xs) + p * kVarTile<ROWS> + off, make_uint4(part[p][0], part[p][1], part[p][2], part[p][3]));
                }
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars[1]);
            ok = mbar_wait(&bars[2], round & 1, status, kStBarDone) && ok;
        }
        ++round;
    }
    if (warp < 8) {
        tc_fence_after_sync();
        const bool formed = round > 0 && __all_sync(0xffffffffu, ok);        // tcgen05.ld is warp-collective
        const float carry = __expf(dA_end);
        float *dst = varlen + (((int64_t)sq * nheads + h) * kP + p0) * kN + n;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            float v[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = 0.f;
            if (formed) {
                const uint32_t at = tmem + ((uint32_t)((warp & 3) * 32) << 16) + p0 + 16 * q;
                float rest[16];
                tmem_ld16(at, v);
                tmem_ld16(at + 64, rest);
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] += rest[j];
            }
            const uint32_t hw[8] = {hv[2 * q].x, hv[2 * q].y, hv[2 * q].z, hv[2 * q].w, hv[2 * q + 1].x, hv[2 * q + 1].y, hv[2 * q + 1].z, hv[2 * q + 1].w};
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                if (entering) {
                    const float2 f = Pack2<T>::unpack(hw[j >> 1]);
                    v[j] = fmaf(prev_np ? (j & 1 ? f.y : f.x) : to_float(H[(p0 + 16 * q + j) * kN + n]), carry, v[j]);
                }
                dst[(16 * q + j) * kN] = v[j];
            }
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 8) tmem_dealloc(tmem, 128);
}

// ====================================================================================== host
// (rank-4) map of a (batch, seqlen, rows, inner) tensor with boxes of 64 inner elements x `steps` steps
bool map_rows(CUtensorMap *m, int fmt, const void *p, const int64_t *st, int inner, int rows, const mb200_ssd_args &a, uint32_t steps)
{
    const uint64_t d[4] = {(uint64_t)inner, (uint64_t)rows, (uint64_t)a.seqlen, (uint64_t)a.batch};
    const uint64_t s[3] = {(uint64_t)st[2] * 2, (uint64_t)st[1] * 2, (uint64_t)st[0] * 2};
    const uint32_t bx[4] = {64, 1, steps, 1};
    return encode_16bit(m, fmt, p, 4, d, s, bx);
}

// The stages of a call follow one another at once: each starts, sets up its barriers, tensor memory and first loads while the one before
// drains, and waits for it (pdl_wait) before it reads what that wrote.  Every stage waits, so the last has waited for all.  Only where
// the output stage has at most kEarlyItems (chunk, head) pairs per SM.  Early / in turn, us, bf16, by pairs per SM: 2 39.9 / 46.1, 9 87 / 93,
// 17 143 / 150, 35 250 / 257, 69 439 / 447, 104 640 / 647, 138 834 / 840; from 208 on (1210 / 1212, 277: 1650 / 1673, 415: 2533 / 2484, 886:
// 5155 / 5186) it is lost in runs that differ by up to 4 %.
constexpr int kEarlyItems = 128;
struct TcCall {
    char *base;
    float *dtb, *dAb;
    void *prev16;
    int *status;
    int nc, hpg;
    bool early;
};
TcCall tc_call(const mb200_ssd_args &a, const SsdScratch &lay)
{
    TcCall k;
    k.base = static_cast<char *>(a.scratch);
    k.dtb = reinterpret_cast<float *>(k.base + lay.off_dt);
    k.dAb = reinterpret_cast<float *>(k.base + lay.off_dA);
    k.prev16 = k.base + lay.off_prev16;
    k.status = ssd_status_word(a, lay);
    k.nc = lay.nchunks;
    k.hpg = a.nheads / a.ngroups;
    k.early = (int64_t)a.batch * k.nc * a.nheads <= (int64_t)kEarlyItems * sm_count(a.device);
    return k;
}

// The entering states as the state-stream kernel stores them: [n][p] tiles of 128 x 64.
bool map_states_np(CUtensorMap *m, int fmt, const TcCall &k, const mb200_ssd_args &a)
{
    const uint64_t d[3] = {kP, kN, (uint64_t)a.batch * k.nc * a.nheads};
    const uint64_t s[2] = {2 * kP, 2 * kP * kN};
    const uint32_t bx[3] = {kP, kN, 1};
    return encode_16bit(m, fmt, k.prev16, 3, d, s, bx);
}

template <typename T>
int run_chunk_state(const mb200_ssd_args &a, const SsdScratch &lay, cudaStream_t stream)
{
    const TcCall k = tc_call(a, lay);
    CUtensorMap tx, tB;
    if (!map_rows(&tx, Fmt<T>::v, a.x, a.x_stride, a.headdim, a.nheads, a, 256) || !map_rows(&tB, Fmt<T>::v, a.B, a.B_stride, a.dstate, a.ngroups, a, 256))
        return fail(MB200_ERR_LAUNCH, "ssd: tensor map for x or B failed");
    constexpr int smem = 3 * 32768 + 256 + 1024;
    ensure_dynamic_smem(reinterpret_cast<const void *>(&ssd_tc_chunk_state_kernel<T>), smem, a.device);
    ssd_tc_chunk_state_kernel<T><<<dim3(a.nheads, k.nc, a.batch), kStateThreads, smem, stream>>>(
        tx, tB, k.dtb, k.dAb, reinterpret_cast<float *>(k.base + lay.off_states), k.nc, a.nheads, k.hpg, a.seq_idx, a.seqlen,
        k.status);
    MB200_CHECK_LAUNCH("ssd chunk_state (tensor core)");
    return MB200_OK;
}

template <typename T>
int run_state_stream(const mb200_ssd_args &a, const SsdScratch &lay, cudaStream_t stream)
{
    const TcCall k = tc_call(a, lay);
    CUtensorMap tx, tB, tHs;
    if (!map_rows(&tx, Fmt<T>::v, a.x, a.x_stride, a.headdim, a.nheads, a, 128) || !map_rows(&tB, Fmt<T>::v, a.B, a.B_stride, a.dstate, a.ngroups, a, 128) ||
        !map_states_np(&tHs, Fmt<T>::v, k, a))
        return fail(MB200_ERR_LAUNCH, "ssd: tensor map for x, B or the states failed");
    // whole operator: from initial_states, entering states stored.  LOCAL half of a sequence split: from a zero
    // state, entering states stored as they are without the incoming state, plus what the OUTPUT half needs to
    // add that state's share later.
    const bool whole = (a.phases & MB200_SSD_PHASE_OUTPUT) != 0;
    float *aux_prefix = whole ? nullptr : reinterpret_cast<float *>(k.base + lay.off_aux);
    float *aux_state = whole ? nullptr : reinterpret_cast<float *>(k.base + lay.off_aux_state);
    float *aux_decay = whole ? nullptr : reinterpret_cast<float *>(k.base + lay.off_aux_decay);
    const float *init = whole ? a.initial_states : nullptr;
    // Two heads of a group per CTA share the B tile (a fifth less shared-memory and L2 traffic per head), but a
    // CTA then runs 1.6x as long, so only whole waves of such CTAs pay; what is left over runs as pairs if that is
    // more than half a wave and as single heads otherwise.
    const int sms = sm_count(a.device);
    const int64_t pairs = k.hpg % 2 == 0 ? (int64_t)a.batch * (a.nheads / 2) : 0;
    int64_t paired = pairs / sms * sms;
    if (pairs - paired > sms / 2) paired = pairs;
    auto go = [&](auto heads_tag, int64_t units, int64_t unit0) {
        constexpr int HEADS = decltype(heads_tag)::value;
        ensure_dynamic_smem(reinterpret_cast<const void *>(&ssd_tc_state_stream_kernel<T, HEADS>), (int)StreamCfg<HEADS>::kSmem, a.device);
        launch_dependent_if(k.early, ssd_tc_state_stream_kernel<T, HEADS>, dim3((unsigned)units), kStreamThreads, StreamCfg<HEADS>::kSmem, stream,
            tx, tB, tHs, k.dtb, k.dAb, init, a.final_states, a.range_decay, aux_prefix, aux_state, aux_decay, 1, k.nc, a.nheads, k.hpg,
            (int)unit0, a.seq_idx, a.seqlen, k.status);
    };
    if (paired > 0) go(std::integral_constant<int, 2>{}, paired, 0);
    const int64_t singles = (int64_t)a.batch * a.nheads - 2 * paired;
    if (singles > 0) go(std::integral_constant<int, 1>{}, singles, 2 * paired);
    MB200_CHECK_LAUNCH("ssd state stream (tensor core)");
    return MB200_OK;
}

template <typename T>
int run_output(const mb200_ssd_args &a, const SsdScratch &lay, bool h_np, cudaStream_t stream)
{
    const TcCall k = tc_call(a, lay);
    constexpr int fmt = Fmt<T>::v;
    CUtensorMap tx, tC, tB, tH, tz, tout;
    bool ok = map_rows(&tx, fmt, a.x, a.x_stride, a.headdim, a.nheads, a, 256) && map_rows(&tB, fmt, a.B, a.B_stride, a.dstate, a.ngroups, a, 256) &&
              map_rows(&tC, fmt, a.C, a.C_stride, a.dstate, a.ngroups, a, 128) && map_rows(&tout, fmt, a.out, a.out_stride, a.headdim, a.nheads, a, 128);
    if (a.z) ok = ok && map_rows(&tz, fmt, a.z, a.z_stride, a.headdim, a.nheads, a, 256);
    else tz = tx;
    if (h_np) {
        ok = ok && map_states_np(&tH, fmt, k, a);
    } else {
        const uint64_t d[3] = {kN, kP, (uint64_t)a.batch * k.nc * a.nheads};
        const uint64_t s[2] = {2 * kN, 2 * kN * kP};
        const uint32_t bx[3] = {64, 64, 1};
        ok = ok && encode_16bit(&tH, fmt, k.prev16, 3, d, s, bx);
    }
    if (!ok) return fail(MB200_ERR_LAUNCH, "ssd: a tensor map of the output stage failed");
    const int64_t items = (int64_t)a.batch * k.nc * a.nheads;
    const int grid = (int)std::min<int64_t>(items, sm_count(a.device));
    const uint8_t *seq_start = a.seq_idx ? reinterpret_cast<const uint8_t *>(k.base + lay.off_seq_start) : nullptr;
    const uint8_t *seq_carry = reinterpret_cast<const uint8_t *>(k.base + lay.off_seq_carry);
    auto go = [&](auto dm, auto with_z) -> int {
        auto kernel = ssd_tc_output_kernel<T, decltype(dm)::value, decltype(with_z)::value>;
        // its warps would wait for ever for registers that the block was not launched with
        static std::atomic<bool> enough{false};              // (a query that failed is made again by the next call)
        if (!enough.load(std::memory_order_relaxed)) {
            cudaFuncAttributes at;
            const cudaError_t e = cudaFuncGetAttributes(&at, reinterpret_cast<const void *>(kernel));
            if (e != cudaSuccess) {
                cudaGetLastError();                          // (it is not the next launch's)
                return fail(MB200_ERR_LAUNCH, "ssd: attributes of the output kernel: %s", cudaGetErrorString(e));
            }
            if (at.numRegs < kOutLaunchRegs) return fail(MB200_ERR_LAUNCH, "ssd: output kernel built with too few registers (%d)", at.numRegs);
            enough.store(true, std::memory_order_relaxed);
        }
        ensure_dynamic_smem(reinterpret_cast<const void *>(kernel), (int)OutCfg::kSmem, a.device);
        launch_dependent_if(k.early, kernel, dim3(grid), kOutThreads, OutCfg::kSmem, stream, tx, tC, tB, tH, tz, tout, k.dtb, k.dAb, a.D, k.nc, a.nheads, a.ngroups, a.seqlen,
                            (int)items, h_np ? 1 : 0, seq_start, seq_carry, k.status);
        return MB200_OK;
    };
    auto with_d = [&](auto dm) { return a.z ? go(dm, std::true_type{}) : go(dm, std::false_type{}); };
    if (int rc = !a.D ? with_d(std::integral_constant<int, kNoD>{}) : a.D_has_hdim ? with_d(std::integral_constant<int, kColumnD>{}) : with_d(std::integral_constant<int, kHeadD>{}))
        return rc;
    MB200_CHECK_LAUNCH("ssd output (tensor core)");
    return MB200_OK;
}

int run_varlen(const mb200_ssd_args &a, const SsdScratch &lay, bool h_np, cudaStream_t stream)
{
    const TcCall k = tc_call(a, lay);
    auto go = [&](auto rows_c) -> int {
        constexpr int ROWS = decltype(rows_c)::value;
        CUtensorMap tx, tB;
        if (!map_rows(&tx, 1, a.x, a.x_stride, a.headdim, a.nheads, a, ROWS) || !map_rows(&tB, 1, a.B, a.B_stride, a.dstate, a.ngroups, a, ROWS))
            return fail(MB200_ERR_LAUNCH, "ssd: tensor map for x or B failed");
        ensure_dynamic_smem(reinterpret_cast<const void *>(&ssd_tc_varlen_kernel<ROWS>), (int)kVarSmem<ROWS>, a.device);
        launch_dependent(ssd_tc_varlen_kernel<ROWS>, dim3(a.nheads, a.num_seqs), kVarThreads, kVarSmem<ROWS>, stream, tx, tB, k.dtb, k.dAb, a.cu_seqlens, a.varlen_states,
                         static_cast<const __nv_bfloat16 *>(k.prev16), h_np ? 1 : 0, k.nc, a.nheads, a.nheads / a.ngroups, a.seqlen, k.status);
        MB200_CHECK_LAUNCH("ssd varlen states (tensor core)");
        return MB200_OK;
    };
    return (int64_t)a.nheads * a.num_seqs > 8 * sm_count(a.device) ? go(std::integral_constant<int, 64>{}) : go(std::integral_constant<int, 128>{});
}

// f(element type of the call)
template <class F> int with_type(const mb200_ssd_args &a, F f) { return a.io_dtype == MB200_BF16 ? f(__nv_bfloat16{}) : f(__half{}); }

}  // namespace

bool ssd_tc_shape(const mb200_ssd_args &a)
{
    if (a.io_dtype != MB200_BF16 && a.io_dtype != MB200_F16) return false;
    return a.headdim == kP && a.dstate == kN && a.chunk_size == kQ;
}

bool ssd_tc_local_eligible(const mb200_ssd_args &a)
{
    if (!ssd_tc_shape(a)) return false;
    if (!rows_for_tma(a.x, a.x_stride) || !rows_for_tma(a.B, a.B_stride)) return false;
    const int64_t nc = (a.seqlen + kQ - 1) / kQ;
    if ((int64_t)a.batch * nc * a.nheads > INT32_MAX || nc > 65535) return false;
    return encode_fn() != nullptr;
}

bool ssd_tc_cb_eligible(const mb200_ssd_args &a) { return a.C && rows_for_tma(a.C, a.C_stride); }

bool ssd_tc_output_eligible(const mb200_ssd_args &a)
{
    if (!ssd_tc_cb_eligible(a)) return false;
    if (!a.out || !rows_for_tma(a.out, a.out_stride)) return false;
    return !a.z || rows_for_tma(a.z, a.z_stride);
}

// One head of one batch row per CTA: worth it once those fill half of the SMs, or when there are so few chunks that walking them in
// order takes no longer than the launch of the separate recurrence.
bool ssd_tc_stream_eligible(const mb200_ssd_args &a)
{
    return (int64_t)a.batch * a.nheads >= kStreamMinUnits || a.seqlen <= 8 * kQ;
}

int ssd_tc_chunk_state(const mb200_ssd_args &a, const SsdScratch &lay, cudaStream_t stream)
{
    return with_type(a, [&](auto t) { return run_chunk_state<decltype(t)>(a, lay, stream); });
}

int ssd_tc_output(const mb200_ssd_args &a, const SsdScratch &lay, bool states_np, cudaStream_t stream)
{
    return with_type(a, [&](auto t) { return run_output<decltype(t)>(a, lay, states_np, stream); });
}

int ssd_tc_varlen(const mb200_ssd_args &a, const SsdScratch &lay, bool states_np, cudaStream_t stream) { return run_varlen(a, lay, states_np, stream); }

template <typename T>
int run_incoming(const mb200_ssd_args &a, const SsdScratch &lay, cudaStream_t stream)
{
    char *base = static_cast<char *>(a.scratch);
    const float *aux_state = reinterpret_cast<const float *>(base + lay.off_aux_state);
    const float *aux_decay = reinterpret_cast<const float *>(base + lay.off_aux_decay);
    const int64_t PN = (int64_t)kP * kN;
    if (!a.initial_states) {       // nothing came in: the entering states stand, the end state is the local one
        if (a.final_states) {
            const cudaError_t e = cudaMemcpyAsync(a.final_states, aux_state, sizeof(float) * (size_t)a.batch * a.nheads * PN,
                                                  cudaMemcpyDeviceToDevice, stream);
            if (e != cudaSuccess) return fail(MB200_ERR_LAUNCH, "ssd: copying the range state: %s", cudaGetErrorString(e));
        }
        return MB200_OK;
    }
    ssd_incoming_state_kernel<T><<<dim3((lay.nchunks + kFixChunks - 1) / kFixChunks, a.nheads, a.batch), 256, 0, stream>>>(
        reinterpret_cast<T *>(base + lay.off_prev16), a.initial_states, reinterpret_cast<const float *>(base + lay.off_aux), aux_state,
        aux_decay, a.final_states, lay.nchunks, a.nheads);
    MB200_CHECK_LAUNCH("ssd incoming state");
    return MB200_OK;
}

int ssd_tc_apply_incoming(const mb200_ssd_args &a, const SsdScratch &lay, cudaStream_t stream)
{
    return a.io_dtype == MB200_BF16 ? run_incoming<__nv_bfloat16>(a, lay, stream) : run_incoming<__half>(a, lay, stream);
}

int ssd_tc_state_stream(const mb200_ssd_args &a, const SsdScratch &lay, cudaStream_t stream)
{
    return with_type(a, [&](auto t) { return run_state_stream<decltype(t)>(a, lay, stream); });
}

}  // namespace mb200

