// Stages of the SSD chunked forward for 16-bit inputs of every shape, on the tensor cores with products as exact as fp32's.
//
// ssd_tc.cu serves 16-bit calls of headdim 64, dstate 128 and chunk 256 with 16-bit operands throughout: weights, decays and entering
// states are rounded to the input type.  Here nothing but the result is.  An fp32 operand -- C.B^T times its decay, a weighted x, an
// entering state -- is cut into bf16 values that add up to it (three hold all 24 bits), and a half-precision input into two, so that
// tcgen05.mma of bf16 operands forms the products, which it adds in fp32; terms below 2^-24 of a product are left out.  bf16 has
// fp32's range: nothing overflows that fp32 holds, whatever the input type.  Against 64 bits, 2 x 1500 steps of 16 heads of 64 x 64:
// end states 1.6e-6 to 3.4e-6, outputs 1.66e-3 (bf16) and 2.07e-4 (fp16), which is their own rounding; the fp32 kernels of ssd.cu gave the
// same to within 1 %, operands rounded to 16 bits 1.7e-3 / 2.1e-4 and 2.4e-3 / 3.0e-4.
//
// Every kernel is one tile loop: 256 threads fetch the next 64 steps of the reduction into registers while the tensor core works on the
// last ones, form the operand values, cut them and store them to 128-byte-swizzled shared memory.  The tensor core is idle most of
// the time; what bounds these kernels is that element-wise work and the latencies between it, which two to four CTAs per SM share.
// Rows are read with plain loads, so any stride and alignment goes.
// 2 x 1500 steps of 48 half-precision heads of 64 x 64, us: chunk states 28, C.B^T 5, outputs 69; the fp32 kernels took 318 for the call.
#include <type_traits>

#include "ssd_common.cuh"
#include "tc_sm100.cuh"

namespace mb200 {
namespace {

using namespace tc;

constexpr int kThreads = 256;
constexpr uint32_t kTileA = 16384, kTileB = 8192;       // bytes of one part of a 128 x 64 and of a 64 x 64 operand
constexpr int kParts = 3;                               // of an fp32 value
template <typename T> constexpr int kInParts = std::is_same<T, __half>::value ? 2 : 1;       // of an input value

enum { kStSplitState = 51, kStSplitCb, kStSplitScan };

__device__ __forceinline__ void sts128(uint32_t addr, uint32_t x, uint32_t y, uint32_t z, uint32_t w)
{
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
// Cuts eight values into NP bf16 parts and stores part p at addr + p * stride.  Each part is what is left rounded to bf16, so that the
// rest is exact and three parts hold all of it.  Values that bf16 would round to infinity, and infinities, are cut by truncation
// instead, which leaves infinities in the first part.
template <int NP>
__device__ __noinline__ void store_parts_large(uint32_t addr, uint32_t stride, float v0, float v1, float v2, float v3, float v4, float v5, float v6, float v7)
{
    float v[8] = {v0, v1, v2, v3, v4, v5, v6, v7};
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t top = __float_as_uint(v[i]) & 0xffff0000u;
            if (i & 1) w[i / 2] |= top;
            else w[i / 2] = top >> 16;
            v[i] = v[i] == __uint_as_float(top) ? 0.f : v[i] - __uint_as_float(top);
        }
        sts128(addr + p * stride, w[0], w[1], w[2], w[3]);
    }
}
template <int NP>
__device__ __forceinline__ void store_parts(uint32_t addr, uint32_t stride, float (&v)[8])
{
    uint32_t w[4];
    auto round8 = [&] {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
            w[i] = *reinterpret_cast<const uint32_t *>(&h);
        }
    };
    round8();
    const auto abs2 = [](uint32_t u) { u &= 0x7fff7fffu; return *reinterpret_cast<const __nv_bfloat162 *>(&u); };
    const __nv_bfloat162 most = __hmax2(__hmax2(abs2(w[0]), abs2(w[1])), __hmax2(abs2(w[2]), abs2(w[3])));
    const uint32_t top = *reinterpret_cast<const uint32_t *>(&most);
    if ((top & 0xffffu) == 0x7f80u || (top >> 16) == 0x7f80u) {          // an infinity
        store_parts_large<NP>(addr, stride, v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7]);
        return;
    }
    sts128(addr, w[0], w[1], w[2], w[3]);
#pragma unroll
    for (int p = 1; p < NP; ++p) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            v[2 * i] -= __uint_as_float(w[i] << 16);
            v[2 * i + 1] -= __uint_as_float(w[i] & 0xffff0000u);
        }
        round8();
        sts128(addr + p * stride, w[0], w[1], w[2], w[3]);
    }
}
__device__ __noinline__ void store_first(uint32_t addr, uint32_t stride, float v0, float v1, float v2, float v3, float v4, float v5, float v6, float v7)
{
    const float v[8] = {v0, v1, v2, v3, v4, v5, v6, v7};
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
        w[i] = *reinterpret_cast<const uint32_t *>(&h);
    }
    sts128(addr, w[0], w[1], w[2], w[3]);
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = (w[i] & 0x80008000u) | 0x01000100u;
    for (int p = 1; p < kParts; ++p) sts128(addr + p * stride, w[0], w[1], w[2], w[3]);
}
template <typename T> __device__ __forceinline__ void widen8(const uint4 &raw, float (&v)[8])
{
    const T *e = reinterpret_cast<const T *>(&raw);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = to_float(e[i]);
}
// Eight input values as they are: bf16 unchanged, half precision in two parts.
template <typename T> __device__ __forceinline__ void store_input(uint32_t addr, uint32_t stride, const uint4 &raw)
{
    if constexpr (kInParts<T> == 1) {
        sts128(addr, raw.x, raw.y, raw.z, raw.w);
    } else {
        float v[8];
        widen8<T>(raw, v);
        store_parts<2>(addr, stride, v);
    }
}

// An infinity (or a NaN) among eight inputs.  Times the first part of an operand it gives what it should, but the later parts may have the
// other sign or be zero: where one turns up they are left out, or made tiny and of the first part's sign.
template <typename T> __device__ __forceinline__ bool not_finite(const uint4 &r)
{
    constexpr uint32_t kInf = std::is_same<T, __half>::value ? 0x7c00u : 0x7f80u;
    const uint32_t m = __vmaxu2(__vmaxu2(r.x & 0x7fff7fffu, r.y & 0x7fff7fffu), __vmaxu2(r.z & 0x7fff7fffu, r.w & 0x7fff7fffu));
    return (m & 0xffffu) >= kInf || (m >> 16) >= kInf;
}

// Eight elements that follow each other in memory, zeros from `n` on; `vec`: they start on a 16-byte boundary.  What is not whole stays out
// of line: a kernel has two dozen such loads.
template <typename T> __device__ __noinline__ uint4 load8_ragged(const T *p, int n)
{
    uint4 r = make_uint4(0, 0, 0, 0);
    T *e = reinterpret_cast<T *>(&r);
#pragma unroll
    for (int i = 0; i < 8; ++i)
        if (i < n) e[i] = p[i];
    return r;
}
template <typename T> __device__ __forceinline__ uint4 load8(const T *p, bool vec, int n)
{
    static_assert(sizeof(T) == 2, "16-bit inputs");
    if (n <= 0) return make_uint4(0, 0, 0, 0);
    return vec && n >= 8 ? *reinterpret_cast<const uint4 *>(p) : load8_ragged(p, n);
}
__device__ __noinline__ float4 load4_ragged(const float *p, int n)
{
    return make_float4(n > 0 ? p[0] : 0.f, n > 1 ? p[1] : 0.f, n > 2 ? p[2] : 0.f, n > 3 ? p[3] : 0.f);
}
__device__ __forceinline__ float4 load4(const float *p, bool vec, int n)
{
    if (n <= 0) return make_float4(0.f, 0.f, 0.f, 0.f);
    return vec && n >= 4 ? *reinterpret_cast<const float4 *>(p) : load4_ragged(p, n);
}
__device__ __forceinline__ void load8(const float *p, bool vec, int n, float4 &lo, float4 &hi)
{
    lo = load4(p, vec, n);
    hi = load4(p + 4, vec, n - 4);
}
template <typename T> __device__ __forceinline__ bool rows16(const T *p, int64_t stride)
{
    return (reinterpret_cast<uintptr_t>(p) & 15) == 0 && stride % 8 == 0;
}
// byte offset of 16-byte chunk `chunk` of row `row` in a tile of 128-byte rows
__device__ __forceinline__ uint32_t sw128(int row, int chunk) { return row * 128 + ((chunk ^ (row & 7)) << 4); }

// The products of one 64-step tile, parts against parts: D += A B, those of the first parts to `d`, the others to `rest`; of `na` parts of A
// and `nb` of B, without those below 2^-24.  Called by a whole warp.
__device__ __forceinline__ void multiply(int na, int nb, uint32_t d, uint32_t rest, uint64_t a, uint32_t step_a, uint64_t b, uint32_t step_b, uint32_t idesc,
                                         bool accumulate)
{
    if (elect_one()) {
        mma_steps_ss(4, d, a, step_a, b, step_b, idesc, accumulate);
        bool more = accumulate || rest == d;
#pragma unroll 1
        for (int i = 0; i < na; ++i)
#pragma unroll 1
            for (int j = i == 0 ? 1 : 0; j < nb && i + j < max(na, nb); ++j) {
                mma_steps_ss(4, rest, a + i * (kTileA / 16), step_a, b + j * (kTileB / 16), step_b, idesc, more);
                more = true;
            }
    }
    __syncwarp();
}

// What the kernels share: a pair of operand tiles, the barrier that the MMAs of a step arrive on, and tensor memory.
struct Tile {
    uint32_t a, b, tmem;
    uint64_t *bar;
    int *status, code;
    int issued = 0;
    bool ok = true;
    // (all threads; `cols` columns of tensor memory)
    __device__ __forceinline__ void open(uint8_t *smem, uint32_t bytes_a, uint32_t bytes_b, int cols, int *status_, int code_)
    {
        a = smem_u32(smem);
        b = a + bytes_a;
        bar = reinterpret_cast<uint64_t *>(smem + bytes_a + bytes_b);
        uint32_t *slot = reinterpret_cast<uint32_t *>(bar + 1);
        status = status_;
        code = code_;
        if (threadIdx.x == 32) {
            mbar_init(bar, 1);
            mbar_fence_init();
            if (a & 1023u) atomicCAS(status, 0, code);      // the swizzled tiles assume a 1 KB aligned base
        }
        if (threadIdx.x < 32) tmem_alloc(slot, cols);
        tc_fence_before_sync();
        __syncthreads();
        tc_fence_after_sync();
        tmem = *slot;
    }
    // the operands of the last step have been read, and its products added
    __device__ __forceinline__ void drain()
    {
        if (issued > 0 && ok) ok = mbar_wait(bar, (issued - 1) & 1, status, code);
    }
    // the tiles are complete: `go` issues the products, told whether any thread raised its flag
    template <class F> __device__ __forceinline__ void step(bool flag, F go)
    {
        fence_proxy_async();
        const bool any = __syncthreads_or(flag);
        if (threadIdx.x < 32) {
            go(any);
            if (elect_one()) mma_commit(bar);
            __syncwarp();
        }
        ++issued;
    }
    __device__ __forceinline__ void close(int cols)
    {
        tc_fence_before_sync();
        __syncthreads();
        if (threadIdx.x < 32) tmem_dealloc(tmem, cols);
    }
};
constexpr uint32_t kTail = 16;                          // barrier and tensor-memory slot behind the tiles

__device__ __forceinline__ int seq_at(const mb200_ssd_args &a, int b, int t) { return a.seq_idx ? a.seq_idx[(int64_t)b * a.seqlen + t] : 0; }

// ====================================================================================== chunk states
// S^T[n,p] = sum_k B[k,n] (w_k x[k,p]), w_k = exp(min(dA_end - dA_k, 0)) dt_k; grid (64-column tiles of P x 128-state tiles, (batch, chunk)
// or sequence, heads).  PACKED: the state after the last token of a packed sequence -- its steps in the chunk of that token, plus the state
// entering the chunk if the sequence began earlier.
template <typename T> constexpr uint32_t kStateSmem = kInParts<T> * kTileA + kParts * kTileB + kTail;
template <typename T, bool PACKED>
__global__ void __launch_bounds__(kThreads, 3) ssd_split_state_kernel(const mb200_ssd_args a, const float *dtb, const float *dAb, const void *entering, SsdStates form,
                                                                      float *states, int nchunks, int *status)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    const int Q = a.chunk_size, P = a.headdim, N = a.dstate, tilesN = (N + 127) / 128;
    const int p0 = (blockIdx.x / tilesN) * 64, n0 = (blockIdx.x % tilesN) * 128, h = blockIdx.z, g = h / (a.nheads / a.ngroups);
    Tile t;
    t.open(smem, kInParts<T> * kTileA, kParts * kTileB, 128, status, kStSplitState);
    pdl_wait();
    int b, c, k0, k1;                               // my steps of the chunk: [k0, k1)
    bool carry = false;
    if constexpr (PACKED) {
        const int start = a.cu_seqlens[blockIdx.y], end = a.cu_seqlens[blockIdx.y + 1];
        const bool empty = end <= start || end > a.seqlen || start < 0;
        b = 0;
        c = empty ? 0 : (end - 1) / Q;
        k0 = empty ? 0 : max(start - c * Q, 0);
        k1 = empty ? 0 : end - c * Q;
        carry = !empty && start < c * Q;
    } else {
        b = blockIdx.y / nchunks;
        c = blockIdx.y % nchunks;
        k0 = 0;
        k1 = min(Q, a.seqlen - c * Q);
    }
    const int64_t row = (((int64_t)b * a.nheads + h) * nchunks + c) * Q, t0 = (int64_t)c * Q;
    const float *dtc = dtb + row, *dAc = dAb + row;
    const float dA_end = PACKED ? (k1 > 0 ? dAc[k1 - 1] : 0.f) : dAc[Q - 1];
    const T *x = static_cast<const T *>(a.x) + (int64_t)b * a.x_stride[0] + t0 * a.x_stride[1] + (int64_t)h * a.x_stride[2] + p0;
    const T *B = static_cast<const T *>(a.B) + (int64_t)b * a.B_stride[0] + t0 * a.B_stride[1] + (int64_t)g * a.B_stride[2] + n0;
    const bool vx = rows16(x, a.x_stride[1]), vB = rows16(B, a.B_stride[1]), wide = N - n0 > 64;
    const int seq_last = PACKED || k1 == 0 ? 0 : seq_at(a, b, c * Q + k1 - 1);      // only steps of the chunk's last sequence reach its end state
    const int c8 = threadIdx.x & 7, r0 = threadIdx.x >> 3;      // my eight columns; rows r0 and r0 + 32 of a tile
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n = n0 + (warp & 3) * 32 + lane, p = p0 + (warp >> 2) * 32;           // my state index and the first of my 32 columns
    const int64_t hc = (int64_t)c * a.nheads + h;
    uint4 in[4] = {};                               // my part of an [n][p] tile of entering states: asked for now, needed last
    if (PACKED && carry && form == SsdStates::np16 && n < N) {
#pragma unroll
        for (int i = 0; i < 4; ++i) in[i] = reinterpret_cast<const uint4 *>(static_cast<const T *>(entering) + (hc * N + n) * P + p)[i];
    }

    uint4 xr[2], Br[4];
    float w[2];
    const bool whole = vx && vB && P - p0 >= 64 && N - n0 >= (wide ? 128 : 64) && (PACKED || !a.seq_idx);
    auto fetch = [&](int k) {
        if (whole && k + 64 <= k1) {                // no edge, nothing to look at
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int kk = k + r0 + 32 * i;
                const T *Bk = B + (int64_t)kk * a.B_stride[1] + 8 * c8;
                xr[i] = *reinterpret_cast<const uint4 *>(x + (int64_t)kk * a.x_stride[1] + 8 * c8);
                Br[i] = *reinterpret_cast<const uint4 *>(Bk);
                if (wide) Br[2 + i] = *reinterpret_cast<const uint4 *>(Bk + 64);
                w[i] = __expf(fminf(dA_end - dAc[kk], 0.f)) * dtc[kk];
            }
            return;
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int kk = k + r0 + 32 * i;
            bool on = kk < k1;
            if (!PACKED && a.seq_idx) on = on && seq_at(a, b, c * Q + kk) == seq_last;
            xr[i] = load8(x + (int64_t)kk * a.x_stride[1] + 8 * c8, vx, on ? P - p0 - 8 * c8 : 0);
            w[i] = on ? __expf(fminf(dA_end - dAc[kk], 0.f)) * dtc[kk] : 0.f;
            const T *Bk = B + (int64_t)kk * a.B_stride[1] + 8 * c8;
            Br[i] = load8(Bk, vB, kk < k1 ? N - n0 - 8 * c8 : 0);
            if (wide) Br[2 + i] = load8(Bk + 64, vB, kk < k1 ? N - n0 - 64 - 8 * c8 : 0);
        }
    };
    if (k0 < k1) fetch(k0);
    constexpr uint32_t idesc = instr_desc_f16(128, 64, 1, 1, 1);
#pragma unroll 1
    for (int k = k0; k < k1; k += 64) {
        t.drain();
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const uint32_t o = sw128(r0 + 32 * i, c8);
            float v[8];
            widen8<T>(xr[i], v);
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] *= w[i];
            const bool bad = not_finite<T>(Br[i]) || (wide && not_finite<T>(Br[2 + i]));
            if (__ballot_sync(0xffffffffu, bad) & 0xffu << (lane & 24)) store_first(t.b + o, kTileB, v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7]);     // in my row
            else store_parts<kParts>(t.b + o, kTileB, v);
            store_input<T>(t.a + o, kTileA, Br[i]);                             // states n0 .. n0 + 63, then the other 64
            if (wide) store_input<T>(t.a + 8192 + o, kTileA, Br[2 + i]);
        }
        t.step(false, [&](bool) {
            // the tensor core adds to a sum with less care than fp32 rounding: the small products have one of their own (with one for
            // all, end states were 8 to 15 % further from 64 bits than the fp32 kernels' in chunks of 128; with two 1 to 2 %)
            const uint32_t acc = warp_uniform(t.tmem);
            multiply(kInParts<T>, kParts, acc, acc + 64, smem_desc_sw128(t.a, 8192, 1024), 128, smem_desc_sw128(t.b, 16, 1024), 128, idesc, k > k0);
        });
        if (k + 64 < k1) fetch(k + 64);
    }
    t.drain();
    float v[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = 0.f;
    if (__all_sync(0xffffffffu, t.ok && t.issued > 0)) {        // tcgen05.ld is warp-collective
        tc_fence_after_sync();
        const uint32_t at = t.tmem + ((uint32_t)((warp & 3) * 32) << 16) + (warp >> 2) * 32;
        float rest[32];
        tmem_ld32(at, v);
        tmem_ld32(at + 64, rest);
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] += rest[j];
    }
    if (n < N) {
        const int64_t slot = PACKED ? (int64_t)blockIdx.y * a.nheads + h : ((int64_t)b * nchunks + c) * a.nheads + h;
        float *S = states + slot * P * N + n;
        const float decay = carry ? __expf(dA_end) : 0.f;
        const T *tile = reinterpret_cast<const T *>(in);
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            if (p + j >= P) continue;
            if (PACKED && carry) {
                const int64_t e = (hc * P + p + j) * N + n;
                const float was = form == SsdStates::np16 ? to_float(tile[j]) : form == SsdStates::pn16 ? to_float(static_cast<const T *>(entering)[e])
                                                                                                        : static_cast<const float *>(entering)[e];
                v[j] = fmaf(was, decay, v[j]);
            }
            S[(int64_t)(p + j) * N] = v[j];
        }
    }
    t.close(128);
}

// ====================================================================================== C.B^T
// CB[m,k] = C_m . B_k, fp32, in tiles of 128 x 64 that reach the diagonal or lie below it; pairs of different sequences get 0.  The
// products of two inputs are exact in the input type.  grid (row blocks x column tiles, batch x chunks, groups)
constexpr uint32_t kCbSmem = kTileA + kTileB + kTail;
template <typename T>
__global__ void __launch_bounds__(kThreads, 4) ssd_split_cb_kernel(const mb200_ssd_args a, float *cb, int nchunks, int *status)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    const int Q = a.chunk_size, N = a.dstate, tilesK = (Q + 63) / 64;
    const int m0 = (blockIdx.x / tilesK) * 128, k0 = (blockIdx.x % tilesK) * 64;
    const int b = blockIdx.y / nchunks, c = blockIdx.y % nchunks, g = blockIdx.z, len = min(Q, a.seqlen - c * Q);
    if (k0 >= m0 + 128 || m0 >= len || k0 >= len) return;
    Tile t;
    t.open(smem, kTileA, kTileB, 64, status, kStSplitCb);
    pdl_wait();
    const int64_t t0 = (int64_t)c * Q;
    const T *C = static_cast<const T *>(a.C) + (int64_t)b * a.C_stride[0] + (t0 + m0) * a.C_stride[1] + (int64_t)g * a.C_stride[2];
    const T *B = static_cast<const T *>(a.B) + (int64_t)b * a.B_stride[0] + (t0 + k0) * a.B_stride[1] + (int64_t)g * a.B_stride[2];
    const bool vC = rows16(C, a.C_stride[1]), vB = rows16(B, a.B_stride[1]), whole = vC && vB && m0 + 128 <= len && k0 + 64 <= len;
    const int c8 = threadIdx.x & 7, r0 = threadIdx.x >> 3;
    uint4 Cr[4], Br[2];
    auto fetch = [&](int n) {
        if (whole && n + 64 <= N) {
#pragma unroll
            for (int i = 0; i < 4; ++i) Cr[i] = *reinterpret_cast<const uint4 *>(C + (int64_t)(r0 + 32 * i) * a.C_stride[1] + n + 8 * c8);
#pragma unroll
            for (int i = 0; i < 2; ++i) Br[i] = *reinterpret_cast<const uint4 *>(B + (int64_t)(r0 + 32 * i) * a.B_stride[1] + n + 8 * c8);
            return;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) Cr[i] = load8(C + (int64_t)(r0 + 32 * i) * a.C_stride[1] + n + 8 * c8, vC, m0 + r0 + 32 * i < len ? N - n - 8 * c8 : 0);
#pragma unroll
        for (int i = 0; i < 2; ++i) Br[i] = load8(B + (int64_t)(r0 + 32 * i) * a.B_stride[1] + n + 8 * c8, vB, k0 + r0 + 32 * i < len ? N - n - 8 * c8 : 0);
    };
    fetch(0);
    constexpr uint32_t idesc = instr_desc_f16(128, 64, std::is_same<T, __half>::value ? 0 : 1, 0, 0);
#pragma unroll 1
    for (int n = 0; n < N; n += 64) {
        t.drain();
#pragma unroll
        for (int i = 0; i < 4; ++i) sts128(t.a + sw128(r0 + 32 * i, c8), Cr[i].x, Cr[i].y, Cr[i].z, Cr[i].w);
#pragma unroll
        for (int i = 0; i < 2; ++i) sts128(t.b + sw128(r0 + 32 * i, c8), Br[i].x, Br[i].y, Br[i].z, Br[i].w);
        t.step(false, [&](bool) {
            const uint32_t acc = warp_uniform(t.tmem);
            multiply(1, 1, acc, acc, smem_desc_sw128(t.a, 16, 1024), 2, smem_desc_sw128(t.b, 16, 1024), 2, idesc, n > 0);
        });
        if (n + 64 < N) fetch(n + 64);
    }
    t.drain();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, m = m0 + (warp & 3) * 32 + lane, k = k0 + (warp >> 2) * 32;
    if (__all_sync(0xffffffffu, t.ok)) {
        float v[32];
        tc_fence_after_sync();
        tmem_ld32(t.tmem + ((uint32_t)((warp & 3) * 32) << 16) + (warp >> 2) * 32, v);
        if (m < Q) {
            if (a.seq_idx) {
                const int mine = m < len ? seq_at(a, b, c * Q + m) : 0;
#pragma unroll
                for (int j = 0; j < 32; ++j)
                    if (!(m < len && k + j < len && mine == seq_at(a, b, c * Q + k + j))) v[j] = 0.f;
            }
            float *out = cb + ((((int64_t)b * nchunks + c) * a.ngroups + g) * Q + m) * Q + k;
            const bool vec = Q % 4 == 0;
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
                if (vec && k + j + 4 <= Q) *reinterpret_cast<float4 *>(out + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
                else
#pragma unroll
                    for (int e = j; e < j + 4; ++e)
                        if (k + e < Q) out[e] = v[e];
            }
        }
    }
    t.close(64);
}

// ====================================================================================== chunk outputs
// y[m,p] = exp(dA_m) C_m . H[p] + sum_{k <= m} CB[m,k] exp(min(dA_m - dA_k, 0)) dt_k x[k,p] + D x[m,p], then y silu(z).
// grid (row blocks of 128, heaviest first, x 64-column tiles of P, batch x chunks, heads).  Two CTAs of 126 registers per SM: three of 80
// spill, and took 76 us where this takes 69 (the half-precision call above); a second pair of tiles left L1 so little that C.B^T, which
// every head reads again, came from L2 each time (72 -> 81 us in bf16); one CTA per SM that keeps C.B^T in tensor memory while the heads
// pass took 78, with all its warps in step 85.
// The result is rounded to the input type.  For bf16 two parts, 16 to 17 bits of an operand, leave its error what all three give.
template <typename T> constexpr int kOutParts = std::is_same<T, __half>::value ? 3 : 2;
template <typename T> constexpr uint32_t kScanA = kOutParts<T> * kTileA;
template <typename T> constexpr uint32_t kScanB = kOutParts<T> * kTileB;
template <typename T>
__global__ void __launch_bounds__(kThreads, 2) ssd_split_scan_kernel(const mb200_ssd_args a, const float *dtb, const float *dAb, const float *states, const float *cb,
                                                                     int nchunks, int *status)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    const int Q = a.chunk_size, P = a.headdim, N = a.dstate, tilesP = (P + 63) / 64;
    const int m0 = ((Q + 127) / 128 - 1 - blockIdx.x / tilesP) * 128, p0 = (blockIdx.x % tilesP) * 64;
    const int b = blockIdx.y / nchunks, c = blockIdx.y % nchunks, h = blockIdx.z, g = h / (a.nheads / a.ngroups);
    const int len = min(Q, a.seqlen - c * Q);
    if (m0 >= len) return;
    Tile t;
    t.open(smem, kScanA<T>, kScanB<T>, 128, status, kStSplitScan);
    pdl_wait();
    const int64_t row = (((int64_t)b * a.nheads + h) * nchunks + c) * Q, t0 = (int64_t)c * Q;
    const float *dAc = dAb + row, *dtc = dtb + row;
    const T *x = static_cast<const T *>(a.x) + (int64_t)b * a.x_stride[0] + t0 * a.x_stride[1] + (int64_t)h * a.x_stride[2] + p0;
    const T *C = static_cast<const T *>(a.C) + (int64_t)b * a.C_stride[0] + (t0 + m0) * a.C_stride[1] + (int64_t)g * a.C_stride[2];
    const float *H = states + (((int64_t)b * nchunks + c) * a.nheads + h) * (int64_t)P * N + (int64_t)p0 * N;
    const float *cbm = cb + ((((int64_t)b * nchunks + c) * a.ngroups + g) * Q + m0) * Q;
    const bool vx = rows16(x, a.x_stride[1]), vC = rows16(C, a.C_stride[1]), vN = N % 4 == 0, vQ = Q % 4 == 0;
    const int kend = min(m0 + 128, len);
    // dA and dt of the steps my rows look back on
    float *col = reinterpret_cast<float *>(smem + kScanA<T> + kScanB<T> + kTail);
    const int cols = (kend + 63) / 64 * 64;
    for (int k = threadIdx.x; k < cols; k += kThreads) {
        col[k] = k < kend ? dAc[k] : 0.f;
        col[cols + k] = k < kend ? dtc[k] : 0.f;
    }
    const int c8 = threadIdx.x & 7, r0 = threadIdx.x >> 3;      // my eight columns; rows r0 + 32 i of a tile
    float dm[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) dm[i] = m0 + r0 + 32 * i < len ? dAc[m0 + r0 + 32 * i] : 0.f;

    // whole tiles need no look at any edge
    const bool whole_rows = m0 + 128 <= len, whole_cols = P - p0 >= 64;
    union { uint4 u[8]; float4 f[8]; } A;           // C rows, or CB rows in two halves
    union { uint4 u[4]; float4 f[4]; } Bq;          // H rows in two halves, or x rows
    auto fetch_states = [&](int n) {
        if (vC && vN && whole_rows && whole_cols && n + 64 <= N) {
#pragma unroll
            for (int i = 0; i < 4; ++i) A.u[i] = *reinterpret_cast<const uint4 *>(C + (int64_t)(r0 + 32 * i) * a.C_stride[1] + n + 8 * c8);
#pragma unroll
            for (int i = 0; i < 4; ++i) Bq.f[i] = reinterpret_cast<const float4 *>(H + (int64_t)(r0 + 32 * (i / 2)) * N + n + 8 * c8)[i & 1];
            return;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) A.u[i] = load8(C + (int64_t)(r0 + 32 * i) * a.C_stride[1] + n + 8 * c8, vC, m0 + r0 + 32 * i < len ? N - n - 8 * c8 : 0);
#pragma unroll
        for (int i = 0; i < 2; ++i)
            load8(H + (int64_t)(r0 + 32 * i) * N + n + 8 * c8, vN, p0 + r0 + 32 * i < P ? N - n - 8 * c8 : 0, Bq.f[2 * i], Bq.f[2 * i + 1]);
    };
    auto fetch_steps = [&](int k) {
        if (vx && vQ && whole_rows && whole_cols) {        // (then kend is a multiple of 64 as well)
#pragma unroll
            for (int i = 0; i < 8; ++i) A.f[i] = reinterpret_cast<const float4 *>(cbm + (int64_t)(r0 + 32 * (i / 2)) * Q + k + 8 * c8)[i & 1];
#pragma unroll
            for (int i = 0; i < 2; ++i) Bq.u[i] = *reinterpret_cast<const uint4 *>(x + (int64_t)(k + r0 + 32 * i) * a.x_stride[1] + 8 * c8);
            return;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
            load8(cbm + (int64_t)(r0 + 32 * i) * Q + k + 8 * c8, vQ, m0 + r0 + 32 * i < len ? kend - k - 8 * c8 : 0, A.f[2 * i], A.f[2 * i + 1]);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int kk = k + r0 + 32 * i;
            Bq.u[i] = load8(x + (int64_t)kk * a.x_stride[1] + 8 * c8, vx, kk < kend ? P - p0 - 8 * c8 : 0);
        }
    };
    fetch_states(0);
    // contribution of the state entering the chunk: C . H, into the first 64 columns
    constexpr uint32_t idesc_h = instr_desc_f16(128, 64, 1, 0, 0), idesc_x = instr_desc_f16(128, 64, 1, 0, 1);
#pragma unroll 1
    for (int n = 0; n < N; n += 64) {
        t.drain();
        bool bad = false;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            bad = bad || not_finite<T>(A.u[i]);
            store_input<T>(t.a + sw128(r0 + 32 * i, c8), kTileA, A.u[i]);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float4 lo = Bq.f[2 * i], hi = Bq.f[2 * i + 1];
            float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
            store_parts<kOutParts<T>>(t.b + sw128(r0 + 32 * i, c8), kTileB, v);
        }
        t.step(bad, [&](bool any) {
            const uint32_t acc = warp_uniform(t.tmem);
            multiply(kInParts<T>, any ? 1 : kOutParts<T>, acc, acc, smem_desc_sw128(t.a, 16, 1024), 2, smem_desc_sw128(t.b, 16, 1024), 2, idesc_h, n > 0);
        });
        if (n + 64 < N) fetch_states(n + 64);
        else fetch_steps(0);
    }
    // the steps of the chunk up to the diagonal, into the other 64
#pragma unroll 1
    for (int k = 0; k < kend; k += 64) {
        t.drain();
        uint64_t dk[4], tk[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            dk[e] = *reinterpret_cast<const uint64_t *>(col + k + 8 * c8 + 2 * e);
            tk[e] = *reinterpret_cast<const uint64_t *>(col + cols + k + 8 * c8 + 2 * e);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t to = t.a + sw128(r0 + 32 * i, c8);
            if (m0 + 32 * i + 31 < k) {             // these rows are above the diagonal
#pragma unroll
                for (int p = 0; p < kOutParts<T>; ++p) sts128(to + p * kTileA, 0u, 0u, 0u, 0u);
                continue;
            }
            const float4 lo = A.f[2 * i], hi = A.f[2 * i + 1];
            const uint64_t cbv[4] = {pack2(lo.x, lo.y), pack2(lo.z, lo.w), pack2(hi.x, hi.y), pack2(hi.z, hi.w)};
            float v[8];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float d0, d1;
                unpack2(sub2(pack2(dm[i], dm[i]), dk[e]), d0, d1);
                unpack2(mul2(pack2(fminf(d0, 0.f), fminf(d1, 0.f)), pack2(kLog2e, kLog2e)), d0, d1);
                unpack2(mul2(mul2(cbv[e], pack2(ex2(d0), ex2(d1))), tk[e]), v[2 * e], v[2 * e + 1]);
            }
            if (k + 64 > m0) {
                const int past = m0 + r0 + 32 * i - (k + 8 * c8);       // columns up to the diagonal
#pragma unroll
                for (int e = 0; e < 8; ++e) v[e] = e <= past ? v[e] : 0.f;
            }
            store_parts<kOutParts<T>>(to, kTileA, v);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) store_input<T>(t.b + sw128(r0 + 32 * i, c8), kTileB, Bq.u[i]);
        t.step(not_finite<T>(Bq.u[0]) || not_finite<T>(Bq.u[1]), [&](bool any) {
            const uint32_t acc = warp_uniform(t.tmem) + 64;
            multiply(any ? 1 : kOutParts<T>, kInParts<T>, acc, acc, smem_desc_sw128(t.a, 16, 1024), 2, smem_desc_sw128(t.b, 16, 1024), 128, idesc_x, k > 0);
        });
        if (k + 64 < kend) fetch_steps(k + 64);
    }
    // x and z of my rows are on their way while the last products are formed
    const T *z = a.z ? static_cast<const T *>(a.z) + (int64_t)b * a.z_stride[0] + t0 * a.z_stride[1] + (int64_t)h * a.z_stride[2] + p0 : nullptr;
    const bool vz = z && rows16(z, a.z_stride[1]);
    const int left = P - p0 - 8 * c8;
    uint4 xm[4], zm[4];
    if (whole_rows && whole_cols && vx && (!z || vz)) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int64_t m = m0 + r0 + 32 * i;
            if (a.D) xm[i] = *reinterpret_cast<const uint4 *>(x + m * a.x_stride[1] + 8 * c8);
            if (z) zm[i] = *reinterpret_cast<const uint4 *>(z + m * a.z_stride[1] + 8 * c8);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int64_t m = m0 + r0 + 32 * i;
            if (a.D) xm[i] = load8(x + m * a.x_stride[1] + 8 * c8, vx, m < len ? left : 0);
            if (z) zm[i] = load8(z + m * a.z_stride[1] + 8 * c8, vz, m < len ? left : 0);
        }
    }
    t.drain();
    if (__syncthreads_and(t.ok)) {
        // from tensor memory, where a thread has a row, to shared memory, so that eight lanes store a row's 64 columns together
        tc_fence_after_sync();
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, lm = (warp & 3) * 32 + lane, m = m0 + lm;
        float sc = m < len ? __expf(dAc[m]) : 0.f;
        // the entering state belongs to the sequence that ends the previous chunk
        if (a.seq_idx && m < len && seq_at(a, b, c * Q + m) != (c > 0 ? seq_at(a, b, c * Q - 1) : 0)) sc = 0.f;
        auto place = [&](int r, int chunk) { return reinterpret_cast<float4 *>(smem + r * 256 + ((chunk ^ (r & 7)) << 4)); };
#pragma unroll
        for (int j = (warp >> 2) * 32; j < (warp >> 2) * 32 + 32; j += 8) {
            uint32_t y1[8], y2[8];
            const uint32_t at = t.tmem + ((uint32_t)((warp & 3) * 32) << 16) + j;
            tmem_ld8_issue(at, y1);
            tmem_ld8_issue(at + 64, y2);
            tmem_ld_wait(y1, y2);
            float y[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) y[e] = fmaf(sc, __uint_as_float(y1[e]), __uint_as_float(y2[e]));
            *place(lm, j / 4) = make_float4(y[0], y[1], y[2], y[3]);
            *place(lm, j / 4 + 1) = make_float4(y[4], y[5], y[6], y[7]);
        }
        __syncthreads();
        T *out = static_cast<T *>(a.out) + (int64_t)b * a.out_stride[0] + t0 * a.out_stride[1] + (int64_t)h * a.out_stride[2] + p0 + 8 * c8;
        const bool vo = rows16(out, a.out_stride[1]);
        float Dv[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) Dv[e] = !a.D ? 0.f : !a.D_has_hdim ? a.D[h] : e < left ? a.D[(int64_t)h * P + p0 + 8 * c8 + e] : 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = r0 + 32 * i;
            if (m0 + r >= len || left <= 0) continue;
            const float4 lo = *place(r, 2 * c8), hi = *place(r, 2 * c8 + 1);
            float y[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w}, f[8];
            if (a.D) {
                widen8<T>(xm[i], f);
#pragma unroll
                for (int e = 0; e < 8; ++e) y[e] = fmaf(f[e], Dv[e], y[e]);
            }
            if (z) {
                widen8<T>(zm[i], f);
#pragma unroll
                for (int e = 0; e < 8; ++e) y[e] *= fast_silu(f[e]);
            }
            uint4 o;
            T *oe = reinterpret_cast<T *>(&o);
#pragma unroll
            for (int e = 0; e < 8; ++e) oe[e] = from_float<T>(y[e]);
            T *om = out + (int64_t)(m0 + r) * a.out_stride[1];
            if (vo && left >= 8) {
                *reinterpret_cast<uint4 *>(om) = o;
            } else {
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    if (e < left) om[e] = oe[e];
            }
        }
    }
    t.close(128);
}

struct Buffers {
    float *dt, *dA, *states, *cb;
    int *status;
    Buffers(const mb200_ssd_args &a, const SsdScratch &lay)
    {
        char *base = static_cast<char *>(a.scratch);
        dt = reinterpret_cast<float *>(base + lay.off_dt);
        dA = reinterpret_cast<float *>(base + lay.off_dA);
        states = reinterpret_cast<float *>(base + lay.off_states);
        cb = reinterpret_cast<float *>(base + lay.off_cb);
        status = ssd_status_word(a, lay);
    }
};
// f(element type of the call)
template <class F> int with_type(const mb200_ssd_args &a, F f) { return a.io_dtype == MB200_BF16 ? f(__nv_bfloat16{}) : f(__half{}); }

template <bool PACKED> int run_states(const mb200_ssd_args &a, const SsdScratch &lay, SsdStates form, cudaStream_t stream)
{
    return with_type(a, [&](auto tag) -> int {
        using T = decltype(tag);
        const Buffers s(a, lay);
        const void *entering = static_cast<const char *>(a.scratch) + (form == SsdStates::pn32 ? lay.off_states : lay.off_prev16);
        const unsigned tiles = (unsigned)((a.headdim + 63) / 64 * ((a.dstate + 127) / 128));
        ensure_dynamic_smem(reinterpret_cast<const void *>(&ssd_split_state_kernel<T, PACKED>), (int)kStateSmem<T>, a.device);
        launch_dependent(ssd_split_state_kernel<T, PACKED>, dim3(tiles, PACKED ? a.num_seqs : a.batch * lay.nchunks, a.nheads), kThreads, kStateSmem<T>, stream, a, s.dt, s.dA,
                         entering, form, PACKED ? a.varlen_states : s.states, lay.nchunks, s.status);
        MB200_CHECK_LAUNCH("ssd states (split products)");
        return MB200_OK;
    });
}

}  // namespace

int ssd_split_states(const mb200_ssd_args &a, const SsdScratch &lay, cudaStream_t stream) { return run_states<false>(a, lay, SsdStates::pn32, stream); }
int ssd_split_varlen(const mb200_ssd_args &a, const SsdScratch &lay, SsdStates entering, cudaStream_t stream) { return run_states<true>(a, lay, entering, stream); }

int ssd_split_cb(const mb200_ssd_args &a, const SsdScratch &lay, cudaStream_t stream)
{
    return with_type(a, [&](auto tag) -> int {
        using T = decltype(tag);
        const Buffers s(a, lay);
        ensure_dynamic_smem(reinterpret_cast<const void *>(&ssd_split_cb_kernel<T>), (int)kCbSmem, a.device);
        const unsigned tiles = (unsigned)((a.chunk_size + 127) / 128 * ((a.chunk_size + 63) / 64));
        launch_dependent(ssd_split_cb_kernel<T>, dim3(tiles, a.batch * lay.nchunks, a.ngroups), kThreads, kCbSmem, stream, a, s.cb, lay.nchunks, s.status);
        MB200_CHECK_LAUNCH("ssd C.B^T (split products)");
        return MB200_OK;
    });
}

int ssd_split_scan(const mb200_ssd_args &a, const SsdScratch &lay, cudaStream_t stream)
{
    return with_type(a, [&](auto tag) -> int {
        using T = decltype(tag);
        const Buffers s(a, lay);
        const uint32_t smem = kScanA<T> + kScanB<T> + kTail + 2 * ((a.chunk_size + 63) / 64 * 64) * (uint32_t)sizeof(float);
        ensure_dynamic_smem(reinterpret_cast<const void *>(&ssd_split_scan_kernel<T>), (int)smem, a.device);
        const unsigned tiles = (unsigned)((a.chunk_size + 127) / 128 * ((a.headdim + 63) / 64));
        launch_dependent(ssd_split_scan_kernel<T>, dim3(tiles, a.batch * lay.nchunks, a.nheads), kThreads, smem, stream, a, s.dt, s.dA, s.states, s.cb, lay.nchunks, s.status);
        MB200_CHECK_LAUNCH("ssd outputs (split products)");
        return MB200_OK;
    });
}

}  // namespace mb200
