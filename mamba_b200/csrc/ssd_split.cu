// Stages of the SSD chunked forward for every shape and type, on the tensor cores with operands in parts.
//
// ssd_tc.cu serves 16-bit calls of headdim 64, dstate 128 and chunk 256 with 16-bit operands throughout: weights, decays and entering states
// are rounded to the input type.  Here an fp32 operand -- an fp32 input, C.B^T times its decay, a weighted x, an entering state -- is cut
// into bf16 values that add up to it, and a half-precision input into two, so that tcgen05.mma of bf16 operands forms the products, which it
// adds in fp32.  Three parts hold all 24 bits, and terms below 2^-24 of a product are left out: so chunk states, C.B^T, and the outputs of
// half precision and fp32.  bf16 outputs take two parts, 16 to 17 bits, of their entering states and decayed C.B^T, so that about 2^-17 of an
// operand is left out of a result with 8 bits.  bf16 has fp32's range: nothing overflows that fp32 holds, whatever the input type.  The
// tensor core cuts its sums off where fp32 arithmetic rounds.  Sums that leave a 16-bit call in fp32 have the small products in a sum of
// their own; in fp32 calls the tensor core adds the products of 64 steps only, the small ones first, and fp32 additions do the rest: without
// decays, where the sums are the whole error, states of 256 steps are 2.3e-7 from 64 bits, outputs 2.6e-7 (4.0e-7 and 6.4e-7 with two sums
// over all steps, 3.3e-7 and 4.3e-7 with tiles of fp32 FMAs; 2 x 2048 steps of 8 heads of 64 x 64: 44.4 us for 43.6).  Against 64 bits, 2 x
// 1500 steps of 16 heads of 64 x 64, four seeds: outputs 1.66e-3 (bf16) and 2.08e-4 (fp16), which is their own rounding, 2.3e-7 to 7.9e-7 in
// fp32 (tiles of fp32 FMAs: 6.7e-7 to 14e-7); end states 1.3e-7 to 1.7e-6 (1.6e-6 to 4.7e-6).  Operands rounded to 16 bits: outputs 2.4e-3
// and 3.0e-4, end states 1.7e-3 and 2.1e-4.
//
// A tile loop: 256 threads fetch the next 64 steps of the reduction while the tensor core works on the last ones, form the operand values,
// cut them and store them.  The tensor core is idle most of the time; what bounds these kernels is that element-wise work and the latencies
// between it, which two to four CTAs per SM share.  Rows are read with plain loads, so any stride and alignment goes.
// 2 x 1500 steps of 48 half-precision heads of 64 x 64, us: chunk states and C.B^T 23, outputs 67; fp32 FMAs took 318 for the call.
#include <algorithm>
#include <cfloat>
#include <type_traits>

#include "ssd_common.cuh"
#include "tc_sm100.cuh"

namespace mb200 {
namespace {

using namespace tc;

constexpr int kThreads = 256;
constexpr uint32_t kTileA = 16384, kTileB = 8192;       // bytes of one part of a 128 x 64 and of a 64 x 64 operand
constexpr int kParts = 3;                               // of an fp32 value
// of an input value
template <typename T> constexpr int kInParts = std::is_same<T, __nv_bfloat16>::value ? 1 : std::is_same<T, __half>::value ? 2 : kParts;

// fp32 operands are cut times 2^17: a value down to the smallest normal number then has all its parts among bf16's numbers, whose smallest is
// 2^-133 (as they are, one of 1e-36 kept 10 bits).  Sums come out times 2^34.  What becomes too large for that, an operand or a sum, is left
// to fp32 FMAs like what cannot be cut at all.
constexpr float kLift = 0x1p17f, kDrop = 0x1p-34f;

// The next tile is requested before the barrier that completes this one, whose cutting takes no time in bf16, or behind it (a call of 2 x 3000
// steps of 32 heads of 128 x 128 in bf16 173 us behind, 168 before; of 2 x 1500 of 48 half-precision heads of 64 x 64 90.6 / 97.5, of 2 x 2048
// of 8 fp32 heads 40.5 / 41.4).
template <typename T> constexpr bool kEarly = kInParts<T> == 1;

enum { kStSplitState = 51, kStSplitCb, kStSplitScan };

__device__ __forceinline__ void sts128(uint32_t addr, uint32_t x, uint32_t y, uint32_t z, uint32_t w)
{
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}

// Eight elements of an input row, as they lie in memory.
template <typename T> struct Raw8 { uint4 q[sizeof(T) / 2]; };
template <typename T> __device__ __forceinline__ void widen8(const Raw8<T> &raw, float (&v)[8])
{
    const T *e = reinterpret_cast<const T *>(&raw);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = to_float(e[i]);
}
// Eight elements that follow each other in memory, zeros from `n` on; `vec`: they start on a 16-byte boundary.  What is not whole stays out
// of line: a kernel has two dozen such loads.
template <typename T> __device__ __noinline__ Raw8<T> load8_ragged(const T *p, int n)
{
    Raw8<T> r = {};
    T *e = reinterpret_cast<T *>(&r);
#pragma unroll
    for (int i = 0; i < 8; ++i)
        if (i < n) e[i] = p[i];
    return r;
}
template <typename T> __device__ __forceinline__ Raw8<T> load8_whole(const T *p) { return *reinterpret_cast<const Raw8<T> *>(p); }
template <typename T> __device__ __forceinline__ Raw8<T> load8(const T *p, bool vec, int n)
{
    if (n <= 0) return Raw8<T>{};
    return vec && n >= 8 ? load8_whole(p) : load8_ragged(p, n);
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
template <typename T> __device__ __forceinline__ bool rows16(const T *p, int64_t stride)
{
    return (reinterpret_cast<uintptr_t>(p) & 15) == 0 && stride * (int64_t)sizeof(T) % 16 == 0;
}

// Cuts a pair of values into NP packed bf16 parts.  Each part is what is left rounded to bf16, so that the rest is exact and three parts
// hold all of it.
template <int NP> __device__ __forceinline__ void cut2(uint64_t v, uint32_t (&w)[NP])
{
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        float a, b;
        unpack2(v, a, b);
        const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
        w[p] = *reinterpret_cast<const uint32_t *>(&h);
        if (p + 1 < NP) v = sub2(v, pack2(__uint_as_float(w[p] << 16), __uint_as_float(w[p] & 0xffff0000u)));
    }
}
// Finds what the cut cannot do: infinities and NaNs, and values that bf16 rounds to infinity.  (An infinity in the first part of an operand
// would meet the later parts of the other, which may have the other sign or be zero.)  A tile that holds one is left out by the tensor core
// and added with fp32 FMAs at the end.  Fed with packed first parts, or packed 16-bit inputs: 0 x v is NaN for those.
template <typename T> struct Finite {
    using H2 = typename std::conditional<std::is_same<T, __half>::value, __half2, __nv_bfloat162>::type;
    uint32_t sum = 0;
    __device__ __forceinline__ void feed(uint32_t w)
    {
        const uint32_t zero = 0;
        const H2 r = __hfma2(*reinterpret_cast<const H2 *>(&w), *reinterpret_cast<const H2 *>(&zero), *reinterpret_cast<const H2 *>(&sum));
        sum = *reinterpret_cast<const uint32_t *>(&r);
    }
    __device__ __forceinline__ bool bad() const { return (sum & 0x7fff7fffu) != 0; }
};
__device__ __forceinline__ uint64_t lift2(float a, float b) { return mul2(pack2(a, b), pack2(kLift, kLift)); }
// Eight values in NP parts, part p at addr + p * stride.
template <int NP, bool LIFT = false> __device__ __forceinline__ bool store_parts(uint32_t addr, uint32_t stride, const float (&v)[8])
{
    uint32_t w[4][NP];
    Finite<__nv_bfloat16> f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        cut2<NP>(LIFT ? lift2(v[2 * i], v[2 * i + 1]) : pack2(v[2 * i], v[2 * i + 1]), w[i]);
        f.feed(w[i][0]);
    }
#pragma unroll
    for (int p = 0; p < NP; ++p) sts128(addr + p * stride, w[0][p], w[1][p], w[2][p], w[3][p]);
    return f.bad();
}
// Eight input values: bf16 as they are, half precision in two parts, fp32 in three.  Says whether one of them is none that can be cut.
template <typename T> __device__ __forceinline__ bool store_input(uint32_t addr, uint32_t stride, const Raw8<T> &raw)
{
    if constexpr (kInParts<T> == 1) {
        const uint4 q = raw.q[0];
        sts128(addr, q.x, q.y, q.z, q.w);
        Finite<T> f;
        f.feed(q.x); f.feed(q.y); f.feed(q.z); f.feed(q.w);
        return f.bad();
    } else {
        float v[8];
        widen8<T>(raw, v);
        return store_parts<kInParts<T>, sizeof(T) == 4>(addr, stride, v);
    }
}
// byte offset of 16-byte chunk `chunk` of row `row` in a tile of 128-byte rows
__device__ __forceinline__ uint32_t sw128(int row, int chunk) { return row * 128 + ((chunk ^ (row & 7)) << 4); }

// The products of one 64-step tile, parts against parts: D += A B, those of the first parts to `d`, the others to `rest`; of `na` parts of A
// and `nb` of B, without those below 2^-24.  Called by a whole warp.
__device__ __forceinline__ void multiply(int na, int nb, uint32_t d, uint32_t rest, uint64_t a, uint32_t step_a, uint64_t b, uint32_t step_b, uint32_t idesc,
                                         bool accumulate, uint32_t part_b = kTileB)
{
    if (elect_one()) {
        mma_steps_ss(4, d, a, step_a, b, step_b, idesc, accumulate);
        bool more = accumulate || rest == d;
#pragma unroll 1
        for (int i = 0; i < na; ++i)
#pragma unroll 1
            for (int j = i == 0 ? 1 : 0; j < nb && i + j < max(na, nb); ++j) {
                mma_steps_ss(4, rest, a + i * (kTileA / 16), step_a, b + j * (part_b / 16), step_b, idesc, more);
                more = true;
            }
    }
    __syncwarp();
}

// The same of fp32 operands, into a sum of the tile's own.  The small products come first, so that only the last ones meet a large sum.
__device__ __forceinline__ void multiply_tile(uint32_t d, uint64_t a, uint32_t step_a, uint64_t b, uint32_t step_b, uint32_t idesc, uint32_t part_b = kTileB)
{
    if (elect_one()) {
        bool more = false;
#pragma unroll 1
        for (int s = kParts - 1; s >= 0; --s)
#pragma unroll 1
            for (int i = 0; i <= s; ++i) {
                mma_steps_ss(4, d, a + i * (kTileA / 16), step_a, b + (s - i) * (part_b / 16), step_b, idesc, more);
                more = true;
            }
    }
    __syncwarp();
}
// Tensor memory: a tile's (lifted) products join the sum over the tiles (`first`: begin it), times `scale`; `cols` columns of my row.  The next
// MMAs may follow a barrier.
__device__ __forceinline__ void fold(uint32_t tile, uint32_t sum, int cols, bool on, bool first, float scale = 1.f)
{
#pragma unroll 1
    for (int j = 0; j < cols; j += 16) {
        uint32_t x[2][8], y[2][8];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            tmem_ld8_issue(tile + j + 8 * i, x[i]);
            tmem_ld8_issue(sum + j + 8 * i, y[i]);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            tmem_ld_wait(x[i], y[i]);
#pragma unroll
            for (int e = 0; e < 8; ++e) y[i][e] = __float_as_uint(fmaf(on ? __uint_as_float(x[i][e]) : 0.f, kDrop, first ? 0.f : __uint_as_float(y[i][e])) * scale);
            tmem_st8_issue(sum + j + 8 * i, y[i]);
        }
    }
    tmem_st_wait();
    tc_fence_before_sync();
}

__device__ __forceinline__ bool finite(float v) { return fabsf(v) <= FLT_MAX; }

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
    // the tiles are complete: `go` issues the products, unless a thread has found what cannot be cut (then it returns false)
    template <class F> __device__ __forceinline__ bool step(bool bad, F go)
    {
        fence_proxy_async();
        if (__syncthreads_or(bad)) return false;
        if (threadIdx.x < 32) {
            go();
            if (elect_one()) mma_commit(bar);
            __syncwarp();
        }
        ++issued;
        return true;
    }
    __device__ __forceinline__ void close(int cols)
    {
        tc_fence_before_sync();
        __syncthreads();
        if (threadIdx.x < 32) tmem_dealloc(tmem, cols);
    }
};
constexpr int kSlice = 16;                              // of what is left to the FMAs, along the reduction
constexpr uint32_t kTail = 16;                          // barrier and tensor-memory slot behind the tiles

__device__ __forceinline__ int seq_at(const mb200_ssd_args &a, int b, int t) { return a.seq_idx ? a.seq_idx[(int64_t)b * a.seqlen + t] : 0; }

// ====================================================================================== chunk states
// S^T[n,p] = sum_k B[k,n] (w_k x[k,p]), w_k = exp(min(dA_end - dA_k, 0)) dt_k.  A unit is 64 columns of a head; a CTA has U units that follow
// each other in a group, and 128 states, of a (batch, chunk) or sequence.  PACKED: the state after the last token of a packed sequence -- its
// steps in the chunk of that token, plus the state entering the chunk if the sequence began earlier.
// Two units share B: fetched, cut, stored and read by the tensor core once.  That pays where B is cut, as soon as single units would not all
// fit the GPU at once (2 x 1500 steps of 48 half-precision heads of 64 x 64: 29 us with one, 23 with two; a call of 2 x 3000 of 32 fp32 heads
// of 64 x 128 181.3 / 179.9, of 128 x 128 336 / 326); in bf16, whose B is stored as it is, two CTAs per SM lose what it saves (2 x 3000 of 32 heads of 128 x 128:
// 52 / 57), and so do the short sums of packed sequences (46 / 54).
template <typename T, int U> constexpr uint32_t kStateB = kParts * U * kTileB;
template <typename T, int U> constexpr uint32_t kStateSmem = kInParts<T> * kTileA + kStateB<T, U> + kTail;      // and the weights of the chunk's steps:
template <int U> inline uint32_t state_weight_bytes(const mb200_ssd_args &a) { return U * ((a.chunk_size + 31) / 32 * 32) * 4; }
// Rare: the states of a CTA some of whose tiles the tensor core has left out: those are added with fp32 FMAs, 16 steps at a time in the place
// of the operands.  (It finds everything by itself and ends the work on these states, so that the kernel keeps nothing for it.)
template <typename T, bool PACKED, int U>
__device__ __noinline__ void finish_left_out_states(const mb200_ssd_args a, const float *dAb, const void *entering, SsdStates form, float *states, int nchunks, int tile, int chunk_or_seq,
                                                    int g, uint8_t *smem, uint32_t tmem, uint32_t skipped, bool formed)
{
    const int Q = a.chunk_size, P = a.headdim, N = a.dstate, tilesN = (N + 127) / 128, tilesP = (P + 63) / 64, units = a.nheads / a.ngroups * tilesP;
    const int unit0 = (tile / tilesN) * U, n0 = (tile % tilesN) * 128;
    const int start = PACKED ? a.cu_seqlens[chunk_or_seq] : 0, end = PACKED ? a.cu_seqlens[chunk_or_seq + 1] : 0;
    const int b = PACKED ? 0 : chunk_or_seq / nchunks, c = PACKED ? (end - 1) / Q : chunk_or_seq % nchunks;
    const int k0 = PACKED ? max(start - c * Q, 0) : 0, k1 = PACKED ? end - c * Q : min(Q, a.seqlen - c * Q);
    const bool carry = PACKED && start < c * Q;
    const int64_t t0 = (int64_t)c * Q;
    const float *const weights = reinterpret_cast<const float *>(smem + kInParts<T> * kTileA + kStateB<T, U> + kTail);
    const int ranges = (Q + 31) / 32 * 32, seq_last = PACKED ? 0 : seq_at(a, b, c * Q + k1 - 1);
    auto head = [&](int u) { return g * (a.nheads / a.ngroups) + min(unit0 + u, units - 1) / tilesP; };
    auto first_col = [&](int u) { return min(unit0 + u, units - 1) % tilesP * 64; };
    auto x_at = [&](int u, int k, int p) {
        return to_float(static_cast<const T *>(a.x)[(int64_t)b * a.x_stride[0] + (t0 + k) * a.x_stride[1] + (int64_t)head(u) * a.x_stride[2] + p]);
    };
    auto B_at = [&](int k, int n) { return to_float(static_cast<const T *>(a.B)[(int64_t)b * a.B_stride[0] + (t0 + k) * a.B_stride[1] + (int64_t)g * a.B_stride[2] + n]); };
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n = n0 + (warp & 3) * 32 + lane, mine = U == 2 ? warp >> 2 : 0;
    const int h = head(mine), col0 = U == 2 ? mine * 64 : (warp >> 2) * 32;             // my columns of the sums
    const bool live = n < N && unit0 + mine < units;
    float *const Bs = reinterpret_cast<float *>(smem), *const xs = Bs + kSlice * 128;
    tc_fence_after_sync();
#pragma unroll 1
    for (int half = 0; half < U; ++half) {          // 32 columns each
        const int p = first_col(mine) + col0 - mine * 64 + 32 * half;
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = 0.f;
        if (formed) {                               // (of fp32 operands the sum over the tiles)
            const uint32_t at = tmem + ((uint32_t)((warp & 3) * 32) << 16) + col0 + 32 * half;
            float rest[32];
            tmem_ld32(at, v);
            tmem_ld32(at + 64 * U, rest);
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = sizeof(T) == 2 ? v[j] + rest[j] : rest[j];
        }
        bool fits = true;
#pragma unroll
        for (int j = 0; j < 32; ++j) fits = fits && finite(v[j]);
        const bool again = sizeof(T) == 4 && live && !fits;  // the lifted sums did not: all of it by FMAs
        if (again) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = 0.f;
        }
        const bool every = __syncthreads_or(again);
#pragma unroll 1
        for (int k = k0; k < k1; k += kSlice) {
            const bool out = skipped >> (k - k0) / 64 & 1;
            if (!out && !every) continue;
            __syncthreads();
            const int s = threadIdx.x >> 4, kk = k + s, col = threadIdx.x & 15;
#pragma unroll
            for (int e = 0; e < 128; e += 16) Bs[s * 128 + e + col] = kk < k1 && n0 + e + col < N ? B_at(kk, n0 + e + col) : 0.f;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int pu = first_col(u) + col;
#pragma unroll
                for (int e = 0; e < 64; e += 16) xs[(s * U + u) * 64 + e + col] = kk < k1 && pu + e < P ? x_at(u, kk, pu + e) * weights[u * ranges + kk] : 0.f;
            }
            __syncthreads();
            if (!out && !again) continue;
#pragma unroll 1
            for (int i = 0; i < kSlice && k + i < k1; ++i) {
                if (!PACKED && a.seq_idx && seq_at(a, b, c * Q + k + i) != seq_last) continue;
                const float Bn = Bs[i * 128 + n - n0], *xk = xs + i * 64 * U + col0 + 32 * half;
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = fmaf(xk[j], Bn, v[j]);
            }
        }
        if (!live) continue;
        const float decay = carry ? __expf(dAb[(((int64_t)b * a.nheads + h) * nchunks + c) * Q + k1 - 1]) : 0.f;
        const int64_t slot = PACKED ? (int64_t)chunk_or_seq * a.nheads + h : ((int64_t)b * nchunks + c) * a.nheads + h, hc = (int64_t)c * a.nheads + h;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            if (p + j >= P) continue;
            if (carry) {
                const int64_t e = form == SsdStates::np16 ? (hc * N + n) * P + p + j : (hc * P + p + j) * N + n;
                v[j] = fmaf(form == SsdStates::pn32 ? static_cast<const float *>(entering)[e] : to_float(static_cast<const T *>(entering)[e]), decay, v[j]);
            }
            states[(slot * P + p + j) * N + n] = v[j];
        }
    }
}
template <typename T, bool PACKED, int U>
__device__ __forceinline__ void split_state(uint8_t *smem, int tile, int chunk_or_seq, int g, const mb200_ssd_args &a, const float *dtb, const float *dAb, const void *entering,
                                            SsdStates form, float *states, int nchunks, int *status)
{
    const int Q = a.chunk_size, P = a.headdim, N = a.dstate, tilesN = (N + 127) / 128, tilesP = (P + 63) / 64, hpg = a.nheads / a.ngroups;
    const int unit0 = (tile / tilesN) * U, n0 = (tile % tilesN) * 128;
    Tile t;
    t.open(smem, kInParts<T> * kTileA, kStateB<T, U>, 128 * U, status, kStSplitState);
    pdl_wait();
    int b, c, k0, k1;                               // my steps of the chunk: [k0, k1)
    bool carry = false;
    if constexpr (PACKED) {
        const int start = a.cu_seqlens[chunk_or_seq], end = a.cu_seqlens[chunk_or_seq + 1];
        const bool empty = end <= start || end > a.seqlen || start < 0;
        b = 0;
        c = empty ? 0 : (end - 1) / Q;
        k0 = empty ? 0 : max(start - c * Q, 0);
        k1 = empty ? 0 : end - c * Q;
        carry = !empty && start < c * Q;
    } else {
        b = chunk_or_seq / nchunks;
        c = chunk_or_seq % nchunks;
        k0 = 0;
        k1 = min(Q, a.seqlen - c * Q);
    }
    const int64_t t0 = (int64_t)c * Q;
    // of each unit (one past the group's last is the last again, and stores nothing)
    int h[U], p0[U];
    const float *dtc[U], *dAc[U];
    float dA_end[U];
    const T *x[U];
    bool vx = true, whole_p = true;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int unit = min(unit0 + u, hpg * tilesP - 1);
        h[u] = g * hpg + unit / tilesP;
        p0[u] = unit % tilesP * 64;
        const int64_t row = (((int64_t)b * a.nheads + h[u]) * nchunks + c) * Q;
        dtc[u] = dtb + row;
        dAc[u] = dAb + row;
        dA_end[u] = PACKED ? (k1 > 0 ? dAc[u][k1 - 1] : 0.f) : dAc[u][Q - 1];
        x[u] = static_cast<const T *>(a.x) + (int64_t)b * a.x_stride[0] + t0 * a.x_stride[1] + (int64_t)h[u] * a.x_stride[2] + p0[u];
        vx = vx && rows16(x[u], a.x_stride[1]);
        whole_p = whole_p && P - p0[u] >= 64;
    }
    const T *B = static_cast<const T *>(a.B) + (int64_t)b * a.B_stride[0] + t0 * a.B_stride[1] + (int64_t)g * a.B_stride[2] + n0;
    const bool vB = rows16(B, a.B_stride[1]), wide = N - n0 > 64;
    const int seq_last = PACKED || k1 == 0 ? 0 : seq_at(a, b, c * Q + k1 - 1);      // only steps of the chunk's last sequence reach its end state
    const int c8 = threadIdx.x & 7, r0 = threadIdx.x >> 3;      // my eight columns; rows r0 and r0 + 32 of a tile
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // results: my state index; one unit: half of its columns, two: all of one's
    const int n = n0 + (warp & 3) * 32 + lane, mine = U == 2 ? warp >> 2 : 0;
    const int my_h = U == 2 && mine ? h[U - 1] : h[0], p = (U == 2 && mine ? p0[U - 1] : p0[0]) + (U == 2 ? 0 : (warp >> 2) * 32);
    const int64_t hc = (int64_t)c * a.nheads + my_h;
    uint4 in[4 * U] = {};                           // my part of an [n][p] tile of entering states: asked for now, needed last
    if (sizeof(T) == 2 && PACKED && carry && form == SsdStates::np16 && n < N) {
#pragma unroll
        for (int i = 0; i < 4 * U; ++i) in[i] = reinterpret_cast<const uint4 *>(static_cast<const T *>(entering) + (hc * N + n) * P + p)[i];
    }

    // The weights: the distance of a step from the last of its 32 is summed within them and not taken from the chunk's sums, which are
    // rounded to 2^-24 of their size (end states of 2 x 1500 steps of 16 heads of 64 x 64 were 2.9e-6 from 64 bits with those, and are 0.2e-6 to
    // 1.0e-6).
    float *const weights = reinterpret_cast<float *>(smem + kInParts<T> * kTileA + kStateB<T, U> + kTail);
    const int ranges = (Q + 31) / 32 * 32;
    auto form_weights = [&] {
#pragma unroll
        for (int u = 0; u < U; ++u)
            for (int k = (k0 & ~31) + (int)threadIdx.x; k < ((k1 + 31) & ~31); k += kThreads) {         // (a warp has a range of 32)
                const float end = k1 > 0 ? dAc[u][min(k | 31, k1 - 1)] : 0.f, dt = k >= k0 && k < k1 ? dtc[u][k] : 0.f;
                float after = dt * a.A[h[u]];
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const float far = __shfl_down_sync(0xffffffffu, after, o);
                    if (lane + o < 32) after += far;
                }
                after = __shfl_down_sync(0xffffffffu, after, 1);
                const bool on = PACKED || !a.seq_idx || (k < k1 && seq_at(a, b, c * Q + k) == seq_last);
                weights[u * ranges + k] = on ? __expf(fminf(dA_end[u] - end + (lane < 31 ? after : 0.f), 0.f)) * dt : 0.f;
            }
    };
    Raw8<T> xr[U][2], Br[4];
    const bool whole = vx && vB && whole_p && N - n0 >= (wide ? 128 : 64) && (PACKED || !a.seq_idx);
    auto fetch = [&](int k) {
        if (whole && k + 64 <= k1) {                // no edge, nothing to look at
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int kk = k + r0 + 32 * i;
                const T *Bk = B + (int64_t)kk * a.B_stride[1] + 8 * c8;
                Br[i] = load8_whole(Bk);
                if (wide) Br[2 + i] = load8_whole(Bk + 64);
#pragma unroll
                for (int u = 0; u < U; ++u) xr[u][i] = load8_whole(x[u] + (int64_t)kk * a.x_stride[1] + 8 * c8);
            }
            return;
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int kk = k + r0 + 32 * i;
            bool on = kk < k1;
            if (!PACKED && a.seq_idx) on = on && seq_at(a, b, c * Q + kk) == seq_last;
#pragma unroll
            for (int u = 0; u < U; ++u) xr[u][i] = load8(x[u] + (int64_t)kk * a.x_stride[1] + 8 * c8, vx, on ? P - p0[u] - 8 * c8 : 0);
            const T *Bk = B + (int64_t)kk * a.B_stride[1] + 8 * c8;
            Br[i] = load8(Bk, vB, kk < k1 ? N - n0 - 8 * c8 : 0);
            if (wide) Br[2 + i] = load8(Bk + 64, vB, kk < k1 ? N - n0 - 64 - 8 * c8 : 0);
        }
    };
    if (k0 < k1) fetch(k0);
    form_weights();
    __syncthreads();
    constexpr uint32_t idesc = instr_desc_f16(128, 64 * U, 1, 1, 1);
    uint32_t skipped = 0;                           // tiles left for the FMAs
    const uint32_t mine_at = t.tmem + ((uint32_t)((warp & 3) * 32) << 16) + (U == 2 ? mine * 64 : (warp >> 2) * 32);       // my columns of the sums
    int folded = 0;                                 // fp32: tiles whose products have joined the sum
    auto fold_last = [&] {
        if (sizeof(T) == 2 || t.issued == folded) return;
        tc_fence_after_sync();
        fold(mine_at, mine_at + 64 * U, 32 * U, true, folded == 0);
        folded = t.issued;
    };
#pragma unroll 1
    for (int k = k0, i64 = 0; k < k1; k += 64, ++i64) {
        t.drain();
        fold_last();
        bool bad = false;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const uint32_t o = sw128(r0 + 32 * i, c8);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                float v[8];
                widen8<T>(xr[u][i], v);
                const int kk = k + r0 + 32 * i;
                float w = kk < k1 ? weights[u * ranges + kk] : 0.f;
                if (sizeof(T) == 4) w *= kLift;
#pragma unroll
                for (int e = 0; e < 8; ++e) v[e] *= w;
                bad = store_parts<kParts>(t.b + u * kTileB + o, U * kTileB, v) || bad;
            }
            bad = store_input<T>(t.a + o, kTileA, Br[i]) || bad;                // states n0 .. n0 + 63, then the other 64
            if (wide) bad = store_input<T>(t.a + 8192 + o, kTileA, Br[2 + i]) || bad;
        }
        if (kEarly<T> && k + 64 < k1) fetch(k + 64);
        const bool first = t.issued == 0;
        if (!t.step(bad, [&] {
            // (16 bits: with one sum for large and small products end states were 8 to 15 % further from 64 bits than tiles of fp32 FMAs in chunks
            // of 128; with two 1 to 2 %)
            const uint32_t acc = warp_uniform(t.tmem);
            const uint64_t da = smem_desc_sw128(t.a, 8192, 1024), db = smem_desc_sw128(t.b, kTileB, 1024);
            if constexpr (sizeof(T) == 4) {
                tc_fence_after_sync();
                multiply_tile(acc, da, 128, db, 128, idesc, U * kTileB);
            } else {
                multiply(kInParts<T>, kParts, acc, acc + 64 * U, da, 128, db, 128, idesc, !first, U * kTileB);
            }
        })) skipped |= 1u << i64;
        if (!kEarly<T> && k + 64 < k1) fetch(k + 64);
    }
    t.drain();
    const bool formed = __all_sync(0xffffffffu, t.ok && t.issued > 0);
    const bool live = n < N && unit0 + mine < hpg * tilesP;
    const float my_end = U == 2 && mine ? dA_end[U - 1] : dA_end[0], decay = carry ? __expf(my_end) : 0.f;
    const T *my_x = U == 2 && mine ? x[U - 1] : x[0];
    const int my_p0 = U == 2 && mine ? p0[U - 1] : p0[0];
    const int64_t slot = PACKED ? (int64_t)chunk_or_seq * a.nheads + my_h : ((int64_t)b * nchunks + c) * a.nheads + my_h;
    if (skipped) {
        fold_last();
        finish_left_out_states<T, PACKED, U>(a, dAb, entering, form, states, nchunks, tile, chunk_or_seq, g, smem, t.tmem, skipped, formed);
        t.close(128 * U);
        return;
    }
    tc_fence_after_sync();
#pragma unroll
    for (int half = 0; half < U; ++half) {          // 32 columns each
        const int pc = p + 32 * half;
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = 0.f;
        if (formed) {                               // tcgen05.ld is warp-collective
            float rest[32];
            tmem_ld32(mine_at + 32 * half, v);
            tmem_ld32(mine_at + 32 * half + 64 * U, rest);
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = sizeof(T) == 2 ? v[j] + rest[j] : fmaf(t.issued > folded ? v[j] : 0.f, kDrop, folded > 0 ? rest[j] : 0.f);
        }
        if (!live) continue;
        if constexpr (sizeof(T) == 4) {
            bool fits = true;
#pragma unroll
            for (int j = 0; j < 32; ++j) fits = fits && finite(v[j]);
            if (!fits) {                            // the lifted sums did not: all of it by FMAs
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = 0.f;
#pragma unroll 1
                for (int k = k0; k < k1; ++k) {
                    if (!PACKED && a.seq_idx && seq_at(a, b, c * Q + k) != seq_last) continue;
                    const float wk = weights[mine * ranges + k], Bn = to_float(B[(int64_t)k * a.B_stride[1] + n - n0]);
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        if (pc + j < P) v[j] = fmaf(to_float(my_x[(int64_t)k * a.x_stride[1] + pc - my_p0 + j]) * wk, Bn, v[j]);
                }
            }
        }
        float *S = states + slot * P * N + n;
        const T *tile_in = reinterpret_cast<const T *>(in) + 32 * half;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            if (pc + j >= P) continue;
            if (PACKED && carry) {
                const int64_t e = (hc * P + pc + j) * N + n;
                const float was = form == SsdStates::np16 ? to_float(tile_in[j]) : form == SsdStates::pn16 ? to_float(static_cast<const T *>(entering)[e])
                                                                                                           : static_cast<const float *>(entering)[e];
                v[j] = fmaf(was, decay, v[j]);
            }
            S[(int64_t)(pc + j) * N] = v[j];
        }
    }
    t.close(128 * U);
}

// ====================================================================================== C.B^T
// CB[m,k] = C_m . B_k, fp32, in tiles of 128 x 64 that reach the diagonal or lie below it; pairs of different sequences get 0.  The
// products of two inputs are exact in the input type.  A CTA has one tile of a (batch, chunk) and a group.
template <typename T> constexpr int kCbParts = sizeof(T) == 2 ? 1 : kParts;
template <typename T> constexpr uint32_t kCbSmem = kCbParts<T> * (kTileA + kTileB) + kTail;
template <typename T>
__device__ __forceinline__ void split_cb(uint8_t *smem, int tile, int chunk, int g, const mb200_ssd_args &a, float *cb, int nchunks, int *status)
{
    const int Q = a.chunk_size, N = a.dstate, tilesK = (Q + 63) / 64;
    const int m0 = (tile / tilesK) * 128, k0 = (tile % tilesK) * 64;
    const int b = chunk / nchunks, c = chunk % nchunks, len = min(Q, a.seqlen - c * Q);
    if (k0 >= m0 + 128 || m0 >= len || k0 >= len) return;
    Tile t;
    constexpr int kSums = sizeof(T) == 2 ? 64 : 128;     // columns of tensor memory: in fp32 the products of a tile, and the sum over the tiles
    t.open(smem, kCbParts<T> * kTileA, kCbParts<T> * kTileB, kSums, status, kStSplitCb);
    pdl_wait();
    const int64_t t0 = (int64_t)c * Q;
    const T *C = static_cast<const T *>(a.C) + (int64_t)b * a.C_stride[0] + (t0 + m0) * a.C_stride[1] + (int64_t)g * a.C_stride[2];
    const T *B = static_cast<const T *>(a.B) + (int64_t)b * a.B_stride[0] + (t0 + k0) * a.B_stride[1] + (int64_t)g * a.B_stride[2];
    const bool vC = rows16(C, a.C_stride[1]), vB = rows16(B, a.B_stride[1]), whole = vC && vB && m0 + 128 <= len && k0 + 64 <= len;
    const int c8 = threadIdx.x & 7, r0 = threadIdx.x >> 3;
    Raw8<T> Cr[4], Br[2];
    auto fetch = [&](int n) {
        if (whole && n + 64 <= N) {
#pragma unroll
            for (int i = 0; i < 4; ++i) Cr[i] = load8_whole(C + (int64_t)(r0 + 32 * i) * a.C_stride[1] + n + 8 * c8);
#pragma unroll
            for (int i = 0; i < 2; ++i) Br[i] = load8_whole(B + (int64_t)(r0 + 32 * i) * a.B_stride[1] + n + 8 * c8);
            return;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) Cr[i] = load8(C + (int64_t)(r0 + 32 * i) * a.C_stride[1] + n + 8 * c8, vC, m0 + r0 + 32 * i < len ? N - n - 8 * c8 : 0);
#pragma unroll
        for (int i = 0; i < 2; ++i) Br[i] = load8(B + (int64_t)(r0 + 32 * i) * a.B_stride[1] + n + 8 * c8, vB, k0 + r0 + 32 * i < len ? N - n - 8 * c8 : 0);
    };
    fetch(0);
    constexpr uint32_t idesc = instr_desc_f16(128, 64, std::is_same<T, __half>::value ? 0 : 1, 0, 0);
    bool all = true;                                // no tile left for the FMAs
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, m = m0 + (warp & 3) * 32 + lane, k = k0 + (warp >> 2) * 32;
    const uint32_t mine_at = t.tmem + ((uint32_t)((warp & 3) * 32) << 16) + (warp >> 2) * 32;                // my columns of the sums
#pragma unroll 1
    for (int n = 0; n < N; n += 64) {
        t.drain();
        if (sizeof(T) == 4 && n > 0 && all) {
            tc_fence_after_sync();
            fold(mine_at, mine_at + 64, 32, true, n == 64);
        }
        bool bad = false;
        auto store = [&](uint32_t to, uint32_t stride, const Raw8<T> &r) {
            if constexpr (sizeof(T) == 2) sts128(to, r.q[0].x, r.q[0].y, r.q[0].z, r.q[0].w);        // one product, exact: nothing to look for
            else bad = store_input<T>(to, stride, r) || bad;
        };
#pragma unroll
        for (int i = 0; i < 4; ++i) store(t.a + sw128(r0 + 32 * i, c8), kTileA, Cr[i]);
#pragma unroll
        for (int i = 0; i < 2; ++i) store(t.b + sw128(r0 + 32 * i, c8), kTileB, Br[i]);
        if (kEarly<T> && n + 64 < N) fetch(n + 64);
        const bool first = t.issued == 0;
        all = t.step(bad, [&] {
            const uint32_t acc = warp_uniform(t.tmem);
            const uint64_t da = smem_desc_sw128(t.a, 16, 1024), db = smem_desc_sw128(t.b, 16, 1024);
            if constexpr (sizeof(T) == 4) {
                tc_fence_after_sync();
                multiply_tile(acc, da, 2, db, 2, idesc);
            } else {
                multiply(1, 1, acc, acc, da, 2, db, 2, idesc, !first);
            }
        }) && all;
        if (!kEarly<T> && n + 64 < N) fetch(n + 64);
    }
    t.drain();
    float v[32];
    if (sizeof(T) == 4 && !all) {                   // a tile could not be cut: fp32 FMAs, 16 states at a time in the place of the operands
        float *const Cs = reinterpret_cast<float *>(smem), *const Bs = Cs + kSlice * 132;
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = 0.f;
#pragma unroll 1
        for (int n = 0; n < N; n += kSlice) {
            const int s = threadIdx.x & 15, row = threadIdx.x >> 4;
            __syncthreads();
#pragma unroll
            for (int e = 0; e < 8; ++e) Cs[s * 132 + row + 16 * e] = n + s < N && m0 + row + 16 * e < len ? to_float(C[(int64_t)(row + 16 * e) * a.C_stride[1] + n + s]) : 0.f;
#pragma unroll
            for (int e = 0; e < 4; ++e) Bs[s * 68 + row + 16 * e] = n + s < N && k0 + row + 16 * e < len ? to_float(B[(int64_t)(row + 16 * e) * a.B_stride[1] + n + s]) : 0.f;
            __syncthreads();
#pragma unroll 1
            for (int i = 0; i < kSlice && n + i < N; ++i) {
                const float Cn = Cs[i * 132 + m - m0];
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = fmaf(Cn, Bs[i * 68 + k - k0 + j], v[j]);
            }
        }
    }
    if (__all_sync(0xffffffffu, t.ok)) {
        if (sizeof(T) == 2 || all) {
            tc_fence_after_sync();
            tmem_ld32(mine_at, v);
        }
        if (sizeof(T) == 4 && all) {
            float sum[32];
            tmem_ld32(mine_at + 64, sum);
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                v[j] = fmaf(v[j], kDrop, N > 64 ? sum[j] : 0.f);
                if (finite(v[j])) continue;             // (else the lifted sum did not fit)
                v[j] = 0.f;
#pragma unroll 1
                for (int n = 0; n < N && m < len && k + j < len; ++n)
                    v[j] = fmaf(to_float(C[(int64_t)(m - m0) * a.C_stride[1] + n]), to_float(B[(int64_t)(k + j - k0) * a.B_stride[1] + n]), v[j]);
            }
        }
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
    t.close(kSums);
}

// Both in one launch: the chunk states need what the launch before formed, C.B^T nothing, and its short CTAs fill the last wave of the other's.
// (states of PACKED sequences have a launch of their own, after the recurrence)
// None of these kernels lets the next one in early: 45 us for 48, 102 for 106 where they do not (2 x 2048 steps of 8 fp32 heads, 2 x 1500
// of 48 half-precision heads of 64 x 64).
template <typename T, bool PACKED, int U>
__global__ void __launch_bounds__(kThreads, sizeof(T) == 2 && U == 1 ? 3 : 2) ssd_split_first_kernel(const mb200_ssd_args a, const float *dtb, const float *dAb, const void *entering, SsdStates form,
                                                                                           float *states, float *cb, int state_ctas, int state_tiles, int cb_tiles, int nchunks, int *status)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    int i = blockIdx.x;
    if (i < state_ctas) {
        const int rows = PACKED ? a.num_seqs : a.batch * nchunks, tile = i % state_tiles;
        i /= state_tiles;
        split_state<T, PACKED, U>(smem, tile, i % rows, i / rows, a, dtb, dAb, entering, form, states, nchunks, status);
    } else if constexpr (!PACKED) {
        i -= state_ctas;
        const int rows = a.batch * nchunks, tile = i % cb_tiles;
        i /= cb_tiles;
        split_cb<T>(smem, tile, i % rows, i / rows, a, cb, nchunks, status);
    }
}

// ====================================================================================== chunk outputs
// y[m,p] = exp(dA_m) C_m . H[p] + sum_{k <= m} CB[m,k] exp(min(dA_m - dA_k, 0)) dt_k x[k,p] + D x[m,p], then y silu(z).
// grid (row blocks of 128, heaviest first, x 64-column tiles of P, batch x chunks, heads).  One kernel for 16-bit inputs, one for fp32.
// The result is rounded to the input type.  For bf16 two parts, 16 to 17 bits of an operand, leave its error what all three give.
template <typename T> constexpr int kOutParts = std::is_same<T, __nv_bfloat16>::value ? 2 : 3;

// Decays of the steps a block of rows looks back on, factorised: exp(dA_m - dA_k) dt_k = exp(dA_m - ref) (exp(ref - dA_k) dt_k), ref = dA of
// the last of 32 steps: an exponential per row and 32 columns instead of one per element.  dA does not increase (A <= 0, dt >= 0), so neither
// exponent is positive below the diagonal; in the range that holds it the first is bounded.  The two are multiplied with each other before
// CB, whose product with a column factor of 2^-100 may be subnormal; a column factor that is so itself (a step of almost no length) would
// lose bits as well.  A range for which one of these is not so has its decays formed one by one.
// In that range two exponents of up to 100 replace one that is small where the weight is large, so neither may lose what the other does not
// give back: the distance of a step from the range's last is summed within the range, not taken from the chunk's sums, which are rounded to
// 2^-24 of their size, and its rows use the same rounded distances as its columns, so that the exponents of a step's weight on itself cancel.
constexpr float kMaxSpan = 100.f;                       // (in powers of two) of the decays within 32 steps
inline uint32_t scan_decay_bytes(const mb200_ssd_args &a)
{
    const uint32_t blocks = (a.chunk_size + 127) / 128, states = (a.dstate + 63) / 64;
    return (3 * 128 * blocks + 1 + (2 * blocks + states + 31) / 32) * 4;
}
struct ScanDecays {
    float *ck, *dA, *rel;       // [step], to the end of the row block: column factors; dA (steps past the end have the last one's); powers of two that
                                // the step's state decays by to the last of its range
    uint32_t *plain;            // ranges that cannot be factorised, a bit each
    uint32_t *skip;             // tiles left for the FMAs, a bit each: of the states, then of the steps
    int cols;
    __device__ __forceinline__ ScanDecays(uint8_t *at, int cols_)
        : ck(reinterpret_cast<float *>(at)), dA(ck + cols_), rel(dA + cols_), plain(reinterpret_cast<uint32_t *>(rel + cols_)), skip(plain + 1), cols(cols_) {}
    // (all threads; a barrier after each)
    __device__ __forceinline__ void clear(int ntiles) const
    {
        for (int i = threadIdx.x; i < 1 + (ntiles + 31) / 32; i += blockDim.x) plain[i] = 0;
    }
    __device__ __forceinline__ void form(const float *dAc, const float *dtc, float A, int kend) const
    {
        const int lane = threadIdx.x & 31;
        for (int k = threadIdx.x; k < cols; k += blockDim.x) {              // (a warp has a range of 32)
            const float v = dAc[min(k, kend - 1)], dt = k < kend ? dtc[k] : 0.f, step = dt * A;
            float after = step;                         // the steps behind mine
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float far = __shfl_down_sync(0xffffffffu, after, o);
                if (lane + o < 32) after += far;
            }
            after = __shfl_down_sync(0xffffffffu, after, 1);
            const float down = lane < 31 ? after * kLog2e : 0.f, w = ex2(down) * dt;
            dA[k] = v;
            rel[k] = -down;
            ck[k] = w;
            const bool falls = __all_sync(0xffffffffu, step <= 0.f && v >= -FLT_MAX);
            const bool fits = __all_sync(0xffffffffu, down >= -kMaxSpan && (w >= FLT_MIN || dt == 0.f));
            if (lane == 0) {
                if (!falls) atomicOr(plain, ~0u);                            // then min(dA_m - dA_k, 0) may be 0 anywhere
                else if (!fits) atomicOr(plain, 1u << (k >> 5));
            }
        }
    }
    // exp(dA_m - ref) for a row `rel_m` before the last of its own range, ref = dA of the last of range `range`; rows before that range's only have
    // to stay finite
    __device__ __forceinline__ float row(float rel_m, float own_end, int range) const { return ex2(fminf(fmaf(own_end - dA[32 * range + 31], kLog2e, rel_m), kMaxSpan)); }
};
// Rare: the outputs of a CTA some of whose tiles the tensor core has left out.  The sums of 128 x 64 of them lie in shared memory; what those
// tiles contribute is added with fp32 FMAs, 16 states or steps at a time.  A thread has eight columns of rows r0 + 32 i.
constexpr uint32_t kLeftOutBytes = kSlice * (132 + 64) * 4;
__device__ __forceinline__ float4 *sum_chunk(uint8_t *sums, int r, int chunk) { return reinterpret_cast<float4 *>(sums + r * 256 + ((chunk ^ (r & 7)) << 4)); }
// (It finds everything by itself and ends the work on these outputs, so that the kernels keep nothing for it.  `lifted`: sums of lifted operands; eight that did not all fit are
// formed again from all tiles.)
template <typename T>
__device__ __noinline__ void finish_left_out(const mb200_ssd_args a, const float *dtb, const float *dAb, const float *states, const float *cb, int nchunks, int tile_cols, int p0,
                                          float *stage, uint8_t *sums, const uint32_t *skip, bool lifted)
{
    const int Q = a.chunk_size, P = a.headdim, N = a.dstate, m0 = ((Q + 127) / 128 - 1 - blockIdx.x / ((P + tile_cols - 1) / tile_cols)) * 128;
    const int b = blockIdx.y / nchunks, c = blockIdx.y % nchunks, h = blockIdx.z, g = h / (a.nheads / a.ngroups);
    const int len = min(Q, a.seqlen - c * Q), kend = min(m0 + 128, len), left = P - p0;
    const int64_t row = (((int64_t)b * a.nheads + h) * nchunks + c) * Q, t0 = (int64_t)c * Q;
    const float *dAc = dAb + row, *dtc = dtb + row;
    const T *x = static_cast<const T *>(a.x) + (int64_t)b * a.x_stride[0] + t0 * a.x_stride[1] + (int64_t)h * a.x_stride[2] + p0;
    const T *C = static_cast<const T *>(a.C) + (int64_t)b * a.C_stride[0] + (t0 + m0) * a.C_stride[1] + (int64_t)g * a.C_stride[2];
    const float *H = states + (((int64_t)b * nchunks + c) * a.nheads + h) * (int64_t)P * N + (int64_t)p0 * N;
    const float *cbm = cb + ((((int64_t)b * nchunks + c) * a.ngroups + g) * Q + m0) * Q;
    const int c8 = threadIdx.x & 7, r0 = threadIdx.x >> 3, nH = (N + 63) / 64, ntiles = nH + (kend + 63) / 64;
    float *const As = stage, *const Bs = As + kSlice * 132;
    uint32_t again = 0;                 // rows of mine whose sums did not fit
    for (int i = 0; i < 4 && lifted; ++i) {
        float4 *lo = sum_chunk(sums, r0 + 32 * i, 2 * c8), *hi = sum_chunk(sums, r0 + 32 * i, 2 * c8 + 1);
        if (finite(lo->x) && finite(lo->y) && finite(lo->z) && finite(lo->w) && finite(hi->x) && finite(hi->y) && finite(hi->z) && finite(hi->w)) continue;
        *lo = *hi = make_float4(0.f, 0.f, 0.f, 0.f);
        again |= 1u << i;
    }
    const bool every = __syncthreads_or(again);
    float acc[4][8] = {};
    bool scaled = false;
    auto scale = [&] {                  // the states' part is complete
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int m = m0 + r0 + 32 * i;
            const bool on = m < len && !(a.seq_idx && seq_at(a, b, c * Q + m) != (c > 0 ? seq_at(a, b, c * Q - 1) : 0));
            const float sc = on ? __expf(dAc[m]) : 0.f;
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[i][e] *= sc;
        }
        scaled = true;
    };
#pragma unroll 1
    for (int t = 0; t < ntiles; ++t) {
        const bool out = (skip[t >> 5] >> (t & 31)) & 1, steps = t >= nH;
        if (!out && !every) continue;
        if (steps && !scaled) scale();
        const uint32_t rows = out ? 15u : again;
        const int first = (steps ? t - nH : t) * 64, end = min(first + 64, steps ? kend : N);
#pragma unroll 1
        for (int k = first; k < end; k += kSlice) {
            __syncthreads();
            const int s = threadIdx.x & 15, kk = k + s, row = threadIdx.x >> 4;
#pragma unroll 1
            for (int r = row; r < 128; r += 16) {
                const int m = m0 + r;
                float v = 0.f;
                if (m < len && kk < end && (!steps || kk <= m))
                    v = steps ? cbm[(int64_t)r * Q + kk] * (__expf(fminf(dAc[m] - dAc[kk], 0.f)) * dtc[kk]) : to_float(C[r * a.C_stride[1] + kk]);
                As[s * 132 + r] = v;
            }
            if (steps) {
                const int ks = k + row;
#pragma unroll 1
                for (int p = s; p < 64; p += 16) Bs[row * 64 + p] = ks < end && p < left ? to_float(x[ks * a.x_stride[1] + p]) : 0.f;
            } else {
#pragma unroll 1
                for (int p = row; p < 64; p += 16) Bs[s * 64 + p] = kk < end && p < left ? H[(int64_t)p * N + kk] : 0.f;
            }
            __syncthreads();
#pragma unroll 1
            for (int i = 0; i < kSlice && k + i < end; ++i) {
                const float4 lo = *reinterpret_cast<const float4 *>(Bs + i * 64 + 8 * c8), hi = *reinterpret_cast<const float4 *>(Bs + i * 64 + 8 * c8 + 4);
                const float b[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (!(rows >> q & 1) || (steps && k + i > m0 + r0 + 32 * q)) continue;     // (nothing goes back in time, not as 0 x inf either)
                    const float w = As[i * 132 + r0 + 32 * q];
#pragma unroll
                    for (int e = 0; e < 8; ++e) acc[q][e] = fmaf(w, b[e], acc[q][e]);
                }
            }
        }
    }
    if (!scaled) scale();
    const T *z = a.z ? static_cast<const T *>(a.z) + (int64_t)b * a.z_stride[0] + t0 * a.z_stride[1] + (int64_t)h * a.z_stride[2] + p0 : nullptr;
    T *out = static_cast<T *>(a.out) + (int64_t)b * a.out_stride[0] + t0 * a.out_stride[1] + (int64_t)h * a.out_stride[2] + p0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = r0 + 32 * i;
        const int64_t m = m0 + r;
        const float *sum[2] = {&sum_chunk(sums, r, 2 * c8)->x, &sum_chunk(sums, r, 2 * c8 + 1)->x};
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int col = 8 * c8 + e;
            if (m >= len || col >= left) continue;
            float y = sum[e >> 2][e & 3] + acc[i][e];
            if (a.D) y = fmaf(to_float(x[m * a.x_stride[1] + col]), a.D[a.D_has_hdim ? (int64_t)h * P + p0 + col : h], y);
            if (z) y *= sizeof(T) == 2 ? fast_silu(to_float(z[m * a.z_stride[1] + col])) : silu(to_float(z[m * a.z_stride[1] + col]));
            out[m * a.out_stride[1] + col] = from_float<T>(y);
        }
    }
}

// ---- 16 bits
// Two CTAs of 121 to 128 registers per SM, of which no more than 12 bytes a thread are spilled: three CTAs of 80 registers spill, and took 76
// us where two took 69 and now take 67 (2 x 1500 steps of 48 half-precision heads of 64 x 64); a second pair of tiles left L1 so little that
// C.B^T, which every head reads again, came from L2 each time (72 -> 81 us in bf16); one CTA per SM that keeps C.B^T in tensor memory while
// the heads pass took 78, with all its warps in step 85.  A kernel laid out like the one for fp32 below, with a warp for the MMAs alone, took
// 68 there, but 175 for 155 us in bf16 (2 x 3000 steps of 32 heads of 128 x 128).
template <typename T> constexpr uint32_t kScan16A = kOutParts<T> * kTileA;
template <typename T, int W> constexpr uint32_t kScan16B = kOutParts<T> * W * kTileB;
static_assert(32768 + kLeftOutBytes <= kScan16A<__nv_bfloat16> + kScan16B<__nv_bfloat16, 1>, "sums and what is added to them");
// W: tiles of 64 columns that share A, whose forming is most of the work: two of a head that has them, where single ones would not all fit the
// GPU at once (a call of 2 x 3000 steps of 32 bf16 heads of 128 x 128: 204 us with one, 168 with two).
template <typename T, int W>
__global__ void __launch_bounds__(kThreads, 2) ssd_split_scan16_kernel(const mb200_ssd_args a, const float *dtb, const float *dAb, const float *states, const float *cb,
                                                                     int nchunks, int *status)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    const int Q = a.chunk_size, P = a.headdim, N = a.dstate, tilesP = (P + 64 * W - 1) / (64 * W);
    const int m0 = ((Q + 127) / 128 - 1 - blockIdx.x / tilesP) * 128, p0 = (blockIdx.x % tilesP) * 64 * W;
    const int b = blockIdx.y / nchunks, c = blockIdx.y % nchunks, h = blockIdx.z, g = h / (a.nheads / a.ngroups);
    const int len = min(Q, a.seqlen - c * Q);
    if (m0 >= len) return;
    Tile t;
    t.open(smem, kScan16A<T>, kScan16B<T, W>, 128 * W, status, kStSplitScan);
    pdl_wait();
    const int64_t row = (((int64_t)b * a.nheads + h) * nchunks + c) * Q, t0 = (int64_t)c * Q;
    const float *dAc = dAb + row, *dtc = dtb + row;
    const T *x = static_cast<const T *>(a.x) + (int64_t)b * a.x_stride[0] + t0 * a.x_stride[1] + (int64_t)h * a.x_stride[2] + p0;
    const T *C = static_cast<const T *>(a.C) + (int64_t)b * a.C_stride[0] + (t0 + m0) * a.C_stride[1] + (int64_t)g * a.C_stride[2];
    const float *H = states + (((int64_t)b * nchunks + c) * a.nheads + h) * (int64_t)P * N + (int64_t)p0 * N;
    const float *cbm = cb + ((((int64_t)b * nchunks + c) * a.ngroups + g) * Q + m0) * Q;
    const bool vx = rows16(x, a.x_stride[1]), vC = rows16(C, a.C_stride[1]), vN = N % 4 == 0, vQ = Q % 4 == 0;
    const int kend = min(m0 + 128, len);
    const ScanDecays decays(smem + kScan16A<T> + kScan16B<T, W> + kTail, m0 + 128);
    decays.clear((N + 63) / 64 + (kend + 63) / 64);
    __syncthreads();
    const int c8 = threadIdx.x & 7, r0 = threadIdx.x >> 3;      // my eight columns; rows r0 + 32 i of a tile
    // whole tiles need no look at any edge
    const bool whole_rows = m0 + 128 <= len, whole_cols = P - p0 >= 64 * W;
    union { Raw8<T> u[4]; float4 f[8]; } A;         // C rows, or CB rows in two halves
    union { Raw8<T> u[2 * W]; float4 f[4 * W]; } Bq;        // H rows in two halves, or x rows
    auto fetch_states = [&](int n) {
        if (vC && vN && whole_rows && whole_cols && n + 64 <= N) {
#pragma unroll
            for (int i = 0; i < 4; ++i) A.u[i] = load8_whole(C + (int64_t)(r0 + 32 * i) * a.C_stride[1] + n + 8 * c8);
#pragma unroll
            for (int i = 0; i < 4 * W; ++i) Bq.f[i] = reinterpret_cast<const float4 *>(H + (int64_t)(r0 + 32 * (i / 2)) * N + n + 8 * c8)[i & 1];
            return;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) A.u[i] = load8(C + (int64_t)(r0 + 32 * i) * a.C_stride[1] + n + 8 * c8, vC, m0 + r0 + 32 * i < len ? N - n - 8 * c8 : 0);
#pragma unroll
        for (int i = 0; i < 4 * W; ++i)
            Bq.f[i] = load4(H + (int64_t)(r0 + 32 * (i / 2)) * N + n + 8 * c8 + 4 * (i & 1), vN, p0 + r0 + 32 * (i / 2) < P ? N - n - 8 * c8 - 4 * (i & 1) : 0);
    };
    auto fetch_steps = [&](int k) {
        if (vx && vQ && whole_rows && whole_cols) {        // (then kend is a multiple of 64 as well)
#pragma unroll
            for (int i = 0; i < 8; ++i) A.f[i] = reinterpret_cast<const float4 *>(cbm + (int64_t)(r0 + 32 * (i / 2)) * Q + k + 8 * c8)[i & 1];
#pragma unroll
            for (int i = 0; i < 2 * W; ++i) Bq.u[i] = load8_whole(x + (int64_t)(k + r0 + 32 * (i & 1)) * a.x_stride[1] + 64 * (i >> 1) + 8 * c8);
            return;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
            A.f[i] = load4(cbm + (int64_t)(r0 + 32 * (i / 2)) * Q + k + 8 * c8 + 4 * (i & 1), vQ, m0 + r0 + 32 * (i / 2) < len ? kend - k - 8 * c8 - 4 * (i & 1) : 0);
#pragma unroll
        for (int i = 0; i < 2 * W; ++i) {
            const int kk = k + r0 + 32 * (i & 1), col = 64 * (i >> 1) + 8 * c8;
            Bq.u[i] = load8(x + (int64_t)kk * a.x_stride[1] + col, vx, kk < kend ? P - p0 - col : 0);
        }
    };
    fetch_states(0);
    const float Dh = a.D && !a.D_has_hdim ? a.D[h] : 0.f;
    decays.form(dAc, dtc, a.A[h], kend);
    __syncthreads();
    const uint32_t plains = *decays.plain;
    float rel[4], own_end[4];                       // of my rows
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        rel[i] = decays.rel[m0 + r0 + 32 * i];
        own_end[i] = decays.dA[m0 + 32 * i + 31];
    }
    const int nH = (N + 63) / 64;
    bool left_out = false;                          // tiles have been left for the FMAs (a bit each in the skip words)
    auto leave_out = [&](int tile) {
        left_out = true;
        if (threadIdx.x == 0) decays.skip[tile >> 5] |= 1u << (tile & 31);
    };
    // contribution of the state entering the chunk: C . H, into the first columns
    constexpr uint32_t idesc_h = instr_desc_f16(128, 64 * W, 1, 0, 0), idesc_x = instr_desc_f16(128, 64 * W, 1, 0, 1);
#pragma unroll 1
    for (int n = 0; n < N; n += 64) {
        t.drain();
        bool bad = false;
#pragma unroll
        for (int i = 0; i < 4; ++i) bad = store_input<T>(t.a + sw128(r0 + 32 * i, c8), kTileA, A.u[i]) || bad;
#pragma unroll
        for (int i = 0; i < 2 * W; ++i) {
            const float4 lo = Bq.f[2 * i], hi = Bq.f[2 * i + 1];
            const float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
            bad = store_parts<kOutParts<T>>(t.b + sw128(r0 + 32 * i, c8), W * kTileB, v) || bad;
        }
        auto next = [&] {
            if (n + 64 < N) fetch_states(n + 64);
            else fetch_steps(0);
        };
        if (kEarly<T>) next();
        const bool first = t.issued == 0;
        if (!t.step(bad, [&] {
            const uint32_t acc = warp_uniform(t.tmem);
            multiply(kInParts<T>, kOutParts<T>, acc, acc, smem_desc_sw128(t.a, 16, 1024), 2, smem_desc_sw128(t.b, 16, 1024), 2, idesc_h, !first, W * kTileB);
        })) leave_out(n >> 6);
        if (!kEarly<T>) next();
    }
    // the steps of the chunk up to the diagonal, into the others
    const int states_done = t.issued;
#pragma unroll 1
    for (int k = 0; k < kend; k += 64) {
        t.drain();
        uint64_t fk[4];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(decays.ck + k + 8 * c8 + 4 * q);
            fk[2 * q] = v.x;
            fk[2 * q + 1] = v.y;
        }
        const int range = (k >> 5) + (c8 >> 2);
        const bool plain = (plains >> range) & 1;
        bool bad = false;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t to = t.a + sw128(r0 + 32 * i, c8);
            if (m0 + 32 * i + 31 < k) {             // these rows are above the diagonal
#pragma unroll
                for (int p = 0; p < kOutParts<T>; ++p) sts128(to + p * kTileA, 0u, 0u, 0u, 0u);
                continue;
            }
            const float4 lo = A.f[2 * i], hi = A.f[2 * i + 1];
            uint64_t f[4] = {fk[0], fk[1], fk[2], fk[3]};
            float fm = decays.row(rel[i], own_end[i], range);
            if (plain) {
                const float dm = decays.dA[m0 + r0 + 32 * i];
                fm = 1.f;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int kk = k + 8 * c8 + 2 * e;
                    f[e] = pack2(kk < kend ? ex2(fminf(dm - decays.dA[kk], 0.f) * kLog2e) * dtc[kk] : 0.f,
                                 kk + 1 < kend ? ex2(fminf(dm - decays.dA[kk + 1], 0.f) * kLog2e) * dtc[kk + 1] : 0.f);
                }
            }
            const uint64_t cbv[4] = {pack2(lo.x, lo.y), pack2(lo.z, lo.w), pack2(hi.x, hi.y), pack2(hi.z, hi.w)};
            float v[8];
#pragma unroll
            for (int e = 0; e < 4; ++e) unpack2(mul2(cbv[e], mul2(f[e], pack2(fm, fm))), v[2 * e], v[2 * e + 1]);
            if (k + 64 > m0) {
                const int past = m0 + r0 + 32 * i - (k + 8 * c8);       // columns up to the diagonal
#pragma unroll
                for (int e = 0; e < 8; ++e) v[e] = e <= past ? v[e] : 0.f;
            }
            bad = store_parts<kOutParts<T>>(to, kTileA, v) || bad;
        }
#pragma unroll
        for (int i = 0; i < 2 * W; ++i) bad = store_input<T>(t.b + (i >> 1) * kTileB + sw128(r0 + 32 * (i & 1), c8), W * kTileB, Bq.u[i]) || bad;
        if (kEarly<T> && k + 64 < kend) fetch_steps(k + 64);
        const bool first = t.issued == states_done;
        if (!t.step(bad, [&] {
            const uint32_t acc = warp_uniform(t.tmem) + 64 * W;
            multiply(kOutParts<T>, kInParts<T>, acc, acc, smem_desc_sw128(t.a, 16, 1024), 2, smem_desc_sw128(t.b, kTileB, 1024), 128, idesc_x, !first, W * kTileB);
        })) leave_out(nH + (k >> 6));
        if (!kEarly<T> && k + 64 < kend) fetch_steps(k + 64);
    }
    // x and z of my rows are on their way while the last products are formed
    const T *z = a.z ? static_cast<const T *>(a.z) + (int64_t)b * a.z_stride[0] + t0 * a.z_stride[1] + (int64_t)h * a.z_stride[2] + p0 : nullptr;
    const bool vz = z && rows16(z, a.z_stride[1]);
    Raw8<T> xm[4], zm[4];
    auto request = [&](int w) {                     // of column tile w
        const int col = 64 * w + 8 * c8, left = P - p0 - col;
        if (whole_rows && whole_cols && vx && (!z || vz)) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int64_t m = m0 + r0 + 32 * i;
                if (a.D) xm[i] = load8_whole(x + m * a.x_stride[1] + col);
                if (z) zm[i] = load8_whole(z + m * a.z_stride[1] + col);
            }
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int64_t m = m0 + r0 + 32 * i;
                if (a.D) xm[i] = load8(x + m * a.x_stride[1] + col, vx, m < len ? left : 0);
                if (z) zm[i] = load8(z + m * a.z_stride[1] + col, vz, m < len ? left : 0);
            }
        }
    };
    request(0);
    t.drain();
    if (__syncthreads_and(t.ok)) {
        // from tensor memory, where a thread has a row, to shared memory, so that eight lanes store a row's 64 columns together
        tc_fence_after_sync();
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, lm = (warp & 3) * 32 + lane, m = m0 + lm;
        auto scale = [&](int m) {                   // the entering state belongs to the sequence that ends the previous chunk
            if (m >= len || (a.seq_idx && seq_at(a, b, c * Q + m) != (c > 0 ? seq_at(a, b, c * Q - 1) : 0))) return 0.f;
            return __expf(decays.dA[m]);
        };
        const float sc = scale(m);
        const bool any1 = states_done > 0, any2 = t.issued > states_done;        // sums that the tensor core has formed
        auto place = [&](int r, int chunk) { return sum_chunk(smem, r, chunk); };
        auto collect = [&](int w) {
#pragma unroll
            for (int j = (warp >> 2) * 32; j < (warp >> 2) * 32 + 32; j += 8) {
                uint32_t y1[8], y2[8];
                const uint32_t at = t.tmem + ((uint32_t)((warp & 3) * 32) << 16) + 64 * w + j;
                tmem_ld8_issue(at, y1);
                tmem_ld8_issue(at + 64 * W, y2);
                tmem_ld_wait(y1, y2);
                float y[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) y[e] = fmaf(sc, any1 ? __uint_as_float(y1[e]) : 0.f, any2 ? __uint_as_float(y2[e]) : 0.f);
                *place(lm, j / 4) = make_float4(y[0], y[1], y[2], y[3]);
                *place(lm, j / 4 + 1) = make_float4(y[4], y[5], y[6], y[7]);
            }
            __syncthreads();
        };
        if (left_out) {
#pragma unroll 1
            for (int w = 0; w < W; ++w) {
                if (w > 0) __syncthreads();
                collect(w);
                finish_left_out<T>(a, dtb, dAb, states, cb, nchunks, 64 * W, p0 + 64 * w, reinterpret_cast<float *>(smem + 32768), smem, decays.skip, false);
            }
        }
#pragma unroll 1
        for (int w = 0; w < W && !left_out; ++w) {
            const int col = 64 * w + 8 * c8, left = P - p0 - col;
            if (w > 0) {
                __syncthreads();
                request(w);
            }
            collect(w);
            T *out = static_cast<T *>(a.out) + (int64_t)b * a.out_stride[0] + t0 * a.out_stride[1] + (int64_t)h * a.out_stride[2] + p0 + col;
            const bool vo = rows16(out, a.out_stride[1]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = r0 + 32 * i;
                if (m0 + r >= len || left <= 0) continue;
                const float4 lo = *place(r, 2 * c8), hi = *place(r, 2 * c8 + 1);
                float y[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w}, f[8];
                if (a.D) {
                    widen8<T>(xm[i], f);
#pragma unroll
                    for (int e = 0; e < 8; ++e) y[e] = fmaf(f[e], !a.D_has_hdim ? Dh : e < left ? a.D[(int64_t)h * P + p0 + col + e] : 0.f, y[e]);
                }
                if (z) {
                    widen8<T>(zm[i], f);
#pragma unroll
                    for (int e = 0; e < 8; ++e) y[e] *= fast_silu(f[e]);
                }
                Raw8<T> o;
                T *oe = reinterpret_cast<T *>(&o);
#pragma unroll
                for (int e = 0; e < 8; ++e) oe[e] = from_float<T>(y[e]);
                T *om = out + (int64_t)(m0 + r) * a.out_stride[1];
                if (vo && left >= 8) {
                    *reinterpret_cast<Raw8<T> *>(om) = o;
                } else {
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        if (e < left) om[e] = oe[e];
                }
            }
        }
    }
    t.close(128 * W);
}


// ---- fp32
// Eight warps form the operands of a tile of 64 along the reduction -- first the states, then the steps of the chunk up to the diagonal --
// and the first issues its MMAs: the A operand (C, then CB with its decays) goes to tensor memory, B (H, then x) to shared memory.  A warp
// has rows 32 (w % 4) .. and one half of the 64 columns; tcgen05.st.16x128b gives a lane four of these rows, and four lanes a row's 16
// bytes, so that the loads fill whole sectors.  The order within a tile is free: a lane's four consecutive elements go to where its words
// are, and B's rows (or H's columns) follow.  (A ninth warp for the MMAs alone leaves a thread 96 registers for 128, because a quarter of the
// SM then has five warps: 28.0 us for 26.2.  With the 128 nothing is spilled.)
// What bounds it: a CTA is one pass through a chain of latencies -- launch, first loads, operands, MMAs, stores -- with three tiles in the
// middle, so everything that can be is requested at the start, and C.B^T two tiles ahead.  2 x 2048 steps of 8 heads of 64 x 64: 27 us (its
// start, which overlaps the recurrence, included), 2 x 3000 steps of 32 heads of 64 x 128 136; 64 x 64 tiles of packed fp32 FMAs took 54 and
// 245.
// Shared memory: B, then two stages of C.B^T, 4 KB a warp.  The sums leave through the first of them.
constexpr uint32_t kScanB = kParts * kTileB, kScanTiles = kScanB + 65536;
constexpr uint32_t kScanTail = 48;                      // barriers and tensor-memory slot behind the tiles
constexpr uint32_t kScanA = 128;                        // tensor memory: the sums of large and of small products, then A

// where step `k` of a tile lies along the reduction: a lane's elements 4 j .. 4 j + 3 of 16 are words j and 4 + j
__device__ __forceinline__ int place4(int k) { return (k & ~15) + ((k >> 1) & 1) * 8 + ((k >> 2) & 3) * 2 + (k & 1); }
__device__ __forceinline__ void tmem_st_16x128b(uint32_t taddr, uint32_t a, uint32_t b)
{
    asm volatile("tcgen05.st.sync.aligned.16x128b.x1.b32 [%0], {%1, %2};" ::"r"(taddr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ void tmem_st_16x128b_x4(uint32_t taddr, const uint32_t (&r)[8])
{
    asm volatile("tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
                 "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, bool in)      // zeros where not `in`
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
}

__global__ void __launch_bounds__(kThreads, 2) ssd_split_scan_kernel(const mb200_ssd_args a, const float *dtb, const float *dAb, const float *states, const float *cb,
                                                                         int nchunks, int *status)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    using T = float;
    constexpr int NP = kParts;
    const int Q = a.chunk_size, P = a.headdim, N = a.dstate, tilesP = (P + 63) / 64;
    const int m0 = ((Q + 127) / 128 - 1 - blockIdx.x / tilesP) * 128, p0 = (blockIdx.x % tilesP) * 64;
    const int b = blockIdx.y / nchunks, c = blockIdx.y % nchunks, h = blockIdx.z, g = h / (a.nheads / a.ngroups);
    const int len = min(Q, a.seqlen - c * Q);
    if (m0 >= len) return;
    const int kend = min(m0 + 128, len), ksteps = (kend + 63) / 64, nH = (N + 63) / 64, ntiles = nH + ksteps;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + kScanTiles), *done = full + 2;      // [tile & 1]: operands in place; their products added
    uint32_t *slot = reinterpret_cast<uint32_t *>(done + 2);
    const ScanDecays decays(smem + kScanTiles + kScanTail, m0 + 128);
    uint32_t *const skip = decays.skip;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&full[i], kThreads / 32);
            mbar_init(&done[i], 1);
        }
        mbar_fence_init();
        if (smem_u32(smem) & 1023u) atomicCAS(status, 0, kStSplitScan);             // the swizzled tiles assume a 1 KB aligned base
    }
    if (warp == 0) tmem_alloc(slot, 256);
    decays.clear(ntiles);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    pdl_wait();
    const uint32_t tmem = *slot, tiles = smem_u32(smem);
    const int64_t row = (((int64_t)b * a.nheads + h) * nchunks + c) * Q, t0 = (int64_t)c * Q;
    const float *dAc = dAb + row, *dtc = dtb + row;
    const T *x = static_cast<const T *>(a.x) + (int64_t)b * a.x_stride[0] + t0 * a.x_stride[1] + (int64_t)h * a.x_stride[2] + p0;
    const T *C = static_cast<const T *>(a.C) + (int64_t)b * a.C_stride[0] + (t0 + m0) * a.C_stride[1] + (int64_t)g * a.C_stride[2];
    const float *H = states + (((int64_t)b * nchunks + c) * a.nheads + h) * (int64_t)P * N + (int64_t)p0 * N;
    const float *cbm = cb + ((((int64_t)b * nchunks + c) * a.ngroups + g) * Q + m0) * Q;
    const bool vx = rows16(x, a.x_stride[1]), vC = rows16(C, a.C_stride[1]), vN = N % 2 == 0, vQ = Q % 4 == 0;
    const bool whole_rows = m0 + 128 <= len, whole_cols = P - p0 >= 64;
    const int j4 = lane & 3, rw = (warp & 3) * 32, ra = rw + (lane >> 2), ch = (warp >> 2) * 32;       // A: rows ra + 8 i, columns of half ch
    const int c8 = threadIdx.x & 7, r0 = threadIdx.x >> 3;                                             // B: rows r0 + 32 i, chunk c8

    Raw8<T> Cr[4];
    float2 Hr[2][4];
    auto fetch_states = [&](int n) {
        // a lane's elements of a row of C: 16 q + 4 j .. + 3; H's columns lie as they do
        const T *pC = C + (int64_t)ra * a.C_stride[1] + n + ch + 4 * j4;
        const float *pH = H + (int64_t)r0 * N + n + 16 * (c8 >> 1) + 2 * (c8 & 1);
        if (vC && vN && whole_rows && whole_cols && n + 64 <= N) {
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int q = 0; q < 2; ++q) Cr[r].q[q] = *reinterpret_cast<const uint4 *>(pC + (int64_t)(8 * r) * a.C_stride[1] + 16 * q);
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int j = 0; j < 4; ++j) Hr[r][j] = *reinterpret_cast<const float2 *>(pH + (int64_t)(32 * r) * N + 4 * j);
            return;
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const T *p = pC + (int64_t)(8 * r) * a.C_stride[1];
            const int left = m0 + ra + 8 * r < len ? N - (int)(p - (C + (int64_t)(ra + 8 * r) * a.C_stride[1])) : 0;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const float4 v = load4(p + 16 * q, vC, left - 16 * q);
                Cr[r].q[q] = *reinterpret_cast<const uint4 *>(&v);
            }
        }
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float *p = pH + (int64_t)(32 * r) * N + 4 * j;
                const int left = p0 + r0 + 32 * r < P ? N - (int)(p - (H + (int64_t)(r0 + 32 * r) * N)) : 0;
                Hr[r][j] = make_float2(left > 0 ? p[0] : 0.f, left > 1 ? p[1] : 0.f);
            }
    };
    Raw8<T> xr[2];
    auto fetch_x = [&](int k) {
        if (vx && whole_rows && whole_cols) {                // no edge, nothing to look at (kend is a multiple of 64 as well)
#pragma unroll
            for (int i = 0; i < 2; ++i) xr[i] = load8_whole(x + (int64_t)(k + r0 + 32 * i) * a.x_stride[1] + 8 * c8);
            return;
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int kk = k + r0 + 32 * i;
            xr[i] = load8(x + (int64_t)kk * a.x_stride[1] + 8 * c8, vx, kk < kend ? P - p0 - 8 * c8 : 0);
        }
    };
    // my warp's 32 x 32 of C.B^T: packets of a row, halves of odd rows swapped, so that a lane's reads below meet no conflict
    constexpr int kAhead = 2;                                // stages
    const uint32_t ring = tiles + kScanB + warp * 4096;
    auto request_cb = [&](int k) {
        const uint32_t to = ring + ((k >> 6) & 1) * 32768 + (lane >> 3) * 128;
        const uint32_t to0 = to + (((lane & 7) ^ ((lane >> 1) & 4)) << 4);                 // rows lane / 8 + 4 i: odd where lane / 8 is
        if (k < kend && m0 + rw + 31 >= k + ch) {            // (else my rows are above the diagonal)
            const int col = k + ch + 4 * (lane & 7), r = rw + (lane >> 3);
            const float *p = cbm + (int64_t)r * Q + col;
            if (vQ && whole_rows) {
#pragma unroll
                for (int i = 0; i < 8; ++i) cp_async16(to0 + 512 * i, p + (int64_t)(4 * i) * Q, true);
            } else {
#pragma unroll 1
                for (int i = 0; i < 8; ++i) {
                    const bool in = m0 + r + 4 * i < len && col < Q;
                    if (vQ) {
                        cp_async16(to0 + 512 * i, in ? p + (int64_t)(4 * i) * Q : cbm, in);
                    } else {
                        const float4 v = load4(p + (int64_t)(4 * i) * Q, false, in ? Q - col : 0);
                        sts128(to0 + 512 * i, __float_as_uint(v.x), __float_as_uint(v.y), __float_as_uint(v.z), __float_as_uint(v.w));
                    }
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch_states(0);
#pragma unroll
    for (int i = 0; i < kAhead; ++i) request_cb(64 * i);
    const float Dh = a.D && !a.D_has_hdim ? a.D[h] : 0.f;
    decays.form(dAc, dtc, a.A[h], kend);
    __syncthreads();
    bool ok = true;
    // the operands of tile i are in place: the first warp issues its MMAs
    auto issue = [&](int i) {
        if (warp != 0) return;
        ok = ok && __all_sync(0xffffffffu, mbar_wait(&full[i & 1], (i >> 1) & 1, status, kStSplitScan));
        if (!ok) return;
        tc_fence_after_sync();
        const uint32_t tm = warp_uniform(tmem), A = tm + kScanA;
        const uint64_t desc = smem_desc_sw128(tiles, 16, 1024);
        const bool steps = i >= nH, on = !((reinterpret_cast<volatile uint32_t *>(skip)[i >> 5] >> (i & 31)) & 1);
        const uint32_t step_b = steps ? 128 : 2, idesc = instr_desc_f16(128, 64, 1, 0, 0) | (steps ? instr_desc_f16(128, 64, 1, 0, 1) : 0);
        if (elect_one()) {
            bool more = false;                               // (as in multiply_tile)
#pragma unroll 1
            for (int s = NP - 1; s >= 0 && on; --s)
#pragma unroll 1
                for (int pa = 0; pa <= s; ++pa) {
                    mma_steps_ts(4, tm, A + 32 * pa, desc + (s - pa) * (kTileB / 16), step_b, idesc, more);
                    more = true;
                }
            mma_commit(&done[i & 1]);
        }
        __syncwarp();
    };
    const uint32_t at = tmem + ((uint32_t)rw << 16) + kScanA + ch / 2;
    const uint32_t plains = *decays.plain;
    const int lm = rw + lane, m = m0 + lm;               // my row of the sums, whose columns ch .. ch + 31 I have
    auto scale = [&](int m) {                            // the entering state belongs to the sequence that ends the previous chunk
        if (m >= len || (a.seq_idx && seq_at(a, b, c * Q + m) != (c > 0 ? seq_at(a, b, c * Q - 1) : 0))) return 0.f;
        return __expf(decays.dA[m]);
    };
    const float sc = scale(m);
    auto skipped = [&](int t) { return (reinterpret_cast<volatile uint32_t *>(skip)[t >> 5] >> (t & 31)) & 1; };
    auto place = [&](int r, int chunk) { return sum_chunk(smem + kScanB, r, chunk); };
    auto wait_done = [&](int i) {
        ok = ok && __all_sync(0xffffffffu, mbar_wait(&done[i & 1], (i >> 1) & 1, status, kStSplitScan));
        if (ok) tc_fence_after_sync();
        return ok;
    };
    auto finish = [&](int i, bool bad) {                 // my part of tile i is in place
        tmem_st_wait();
        fence_proxy_async();
        tc_fence_before_sync();
        if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(&skip[i >> 5], 1u << (i & 31));
        __syncwarp();
        if (lane == 0) mbar_arrive(&full[i & 1]);
    };
    const uint32_t tile_at = tmem + ((uint32_t)rw << 16) + ch, sum_at = tile_at + 64;        // my row's columns: a tile's products, the sum over the tiles
    bool begun = false;                                  // that sum holds something
    auto join = [&](int i, bool scaled) {                // the products of tile i join it; then times exp(dA_m)
        const bool on = !skipped(i);
        if (on || (begun && scaled)) fold(tile_at, sum_at, 32, on, !begun, scaled ? sc : 1.f);
        begun = begun || on;
    };

    // ---- the state entering the chunk: C . H
    int i = 0;
#pragma unroll 1
    for (int n = 0; n < N; n += 64, ++i) {
        if (i > 0) {
            if (!wait_done(i - 1)) break;
            join(i - 1, false);
        }
        bool bad = false;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const float v[8] = {Hr[r][0].x, Hr[r][0].y, Hr[r][1].x, Hr[r][1].y, Hr[r][2].x, Hr[r][2].y, Hr[r][3].x, Hr[r][3].y};
            bad = store_parts<NP, true>(tiles + sw128(r0 + 32 * r, c8), kTileB, v) || bad;
        }
        Finite<__nv_bfloat16> f;
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
            uint32_t w[NP][8];
#pragma unroll
            for (int hr = 0; hr < 2; ++hr) {
                float v[8];
                widen8<T>(Cr[2 * hh + hr], v);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    uint32_t parts[NP];
                    cut2<NP>(lift2(v[2 * q], v[2 * q + 1]), parts);
                    f.feed(parts[0]);
#pragma unroll
                    for (int p = 0; p < NP; ++p) w[p][2 * q + hr] = parts[p];
                }
            }
#pragma unroll
            for (int p = 0; p < NP; ++p) tmem_st_16x128b_x4(at + 32 * p + ((16u * hh) << 16), w[p]);
        }
        if (n + 64 < N) fetch_states(n + 64);
        else fetch_x(0);
        finish(i, bad || f.bad());
        issue(i);
    }

    // ---- steps of the chunk up to the diagonal
#pragma unroll 1
    for (int k = 0; k < kend && ok; k += 64, ++i) {
        if (!wait_done(i - 1)) break;
        join(i - 1, k == 0);
        bool bad = false;
#pragma unroll
        for (int r = 0; r < 2; ++r) bad = store_input<T>(tiles + sw128(place4(r0 + 32 * r), c8), kTileB, xr[r]) || bad;
        if (k + 64 < kend) fetch_x(k + 64);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        if (m0 + rw + 31 < k + ch) {
            const uint32_t none[8] = {};
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                tmem_st_16x128b_x4(at + 32 * p, none);
                tmem_st_16x128b_x4(at + 32 * p + (16u << 16), none);
            }
        } else {
            Finite<__nv_bfloat16> f;
            if (!((plains >> ((k + ch) >> 5)) & 1)) {
                uint64_t fk[4];                          // of my columns 16 q + 4 j .. + 3
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(decays.ck + k + ch + 4 * j4 + 16 * q);
                    fk[2 * q] = v.x;
                    fk[2 * q + 1] = v.y;
                }
                const uint32_t from = ring + ((k >> 6) & 1) * 32768 + (lane >> 2) * 128 + j4 * 16, flip = (lane & 4) << 4;       // (row & 1 = lane / 4 & 1)
                const bool diagonal = k + ch + 31 > m0 + rw;
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    uint32_t w[NP][8];
#pragma unroll
                    for (int hr = 0; hr < 2; ++hr) {
                        const int r = 2 * hh + hr;
                        uint64_t cbv[4];
#pragma unroll
                        for (int q = 0; q < 2; ++q)
                            asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(cbv[2 * q]), "=l"(cbv[2 * q + 1]) : "r"(from + r * 1024 + ((q << 6) ^ flip)));
                        const int past = m0 + ra + 8 * r - (k + ch + 4 * j4);           // columns up to the diagonal
                        const float fm = decays.row(decays.rel[m0 + ra + 8 * r], decays.dA[m0 + rw + 31], (k + ch) >> 5) * kLift;
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            uint64_t v = mul2(cbv[q], mul2(fk[q], pack2(fm, fm)));
                            if (diagonal) {
                                float v0, v1;
                                unpack2(v, v0, v1);
                                const int e = 16 * (q >> 1) + 2 * (q & 1);
                                v = pack2(e <= past ? v0 : 0.f, e + 1 <= past ? v1 : 0.f);
                            }
                            uint32_t parts[NP];
                            cut2<NP>(v, parts);
                            f.feed(parts[0]);
#pragma unroll
                            for (int p = 0; p < NP; ++p) w[p][2 * q + hr] = parts[p];
                        }
                    }
#pragma unroll
                    for (int p = 0; p < NP; ++p) tmem_st_16x128b_x4(at + 32 * p + ((16u * hh) << 16), w[p]);
                }
            } else {
                // rare, and kept short: one word of two rows at a time
#pragma unroll 1
                for (int e = 0; e < 8; ++e) {
                    const int q = e & 3, hh = e >> 2, kk = k + ch + 4 * j4 + 16 * (q >> 1) + 2 * (q & 1);
                    uint32_t w[2][NP];
#pragma unroll
                    for (int hr = 0; hr < 2; ++hr) {
                        const int rr = ra + 8 * (2 * hh + hr), m = m0 + rr;
                        auto one = [&](int kk) { return m < len && kk <= m ? cbm[(int64_t)rr * Q + kk] * (__expf(fminf(dAc[m] - dAc[kk], 0.f)) * dtc[kk] * kLift) : 0.f; };
                        cut2<NP>(pack2(one(kk), one(kk + 1)), w[hr]);
                        f.feed(w[hr][0]);
                    }
                    __syncwarp();
#pragma unroll
                    for (int p = 0; p < NP; ++p) tmem_st_16x128b(at + 32 * p + 4 * q + ((16u * hh) << 16), w[0][p], w[1][p]);
                }
            }
            bad = f.bad() || bad;
        }
        __syncwarp();
        finish(i, bad);
        issue(i);
        request_cb(k + 64 * kAhead);
    }

    // ---- x and z of my rows are on their way while the last products are formed
    const T *z = a.z ? static_cast<const T *>(a.z) + (int64_t)b * a.z_stride[0] + t0 * a.z_stride[1] + (int64_t)h * a.z_stride[2] + p0 : nullptr;
    const bool vz = z && rows16(z, a.z_stride[1]);
    const int left = P - p0 - 8 * c8;
    Raw8<T> xm[4], zm[4];
    if (whole_rows && whole_cols && vx && (!z || vz)) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int64_t m = m0 + r0 + 32 * r;
            if (a.D) xm[r] = load8_whole(x + m * a.x_stride[1] + 8 * c8);
            if (z) zm[r] = load8_whole(z + m * a.z_stride[1] + 8 * c8);
        }
    } else {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int64_t m = m0 + r0 + 32 * r;
            if (a.D) xm[r] = load8(x + m * a.x_stride[1] + 8 * c8, vx, m < len ? left : 0);
            if (z) zm[r] = load8(z + m * a.z_stride[1] + 8 * c8, vz, m < len ? left : 0);
        }
    }
    wait_done(ntiles - 1);
    if (__syncthreads_and(ok)) {                         // (also: everyone's writes to the skip words are there, and C.B^T is not needed any more)
        bool fma = false, fits = true;                   // something is left; the lifted sums of my row did
        for (int t = 0; t < ntiles; ++t) fma = fma || skipped(t);
        const bool on = !skipped(ntiles - 1);
        // from tensor memory, where a thread has a row, to shared memory, so that eight lanes store a row's 64 columns together
        tc_fence_after_sync();
#pragma unroll
        for (int j = ch; j < ch + 32; j += 8) {
            uint32_t u[8], w[8];
            tmem_ld8_issue(tile_at + j - ch, u);
            tmem_ld8_issue(sum_at + j - ch, w);
            tmem_ld_wait(u, w);
            float y[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) y[e] = fmaf(on ? __uint_as_float(u[e]) : 0.f, kDrop, begun ? __uint_as_float(w[e]) : 0.f);
#pragma unroll
            for (int e = 0; e < 8; ++e) fits = fits && finite(y[e]);
            *place(lm, j / 4) = make_float4(y[0], y[1], y[2], y[3]);
            *place(lm, j / 4 + 1) = make_float4(y[4], y[5], y[6], y[7]);
        }
        fma = __syncthreads_or(!fits) || fma;
        T *out = static_cast<T *>(a.out) + (int64_t)b * a.out_stride[0] + t0 * a.out_stride[1] + (int64_t)h * a.out_stride[2] + p0 + 8 * c8;
        const bool vo = rows16(out, a.out_stride[1]);
        if (fma) {
            finish_left_out<T>(a, dtb, dAb, states, cb, nchunks, 64, p0, reinterpret_cast<float *>(smem), smem + kScanB, skip, true);
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int r = r0 + 32 * q;
                if (m0 + r >= len || left <= 0) continue;
                const float4 lo = *place(r, 2 * c8), hi = *place(r, 2 * c8 + 1);
                float y[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w}, f[8];
                if (a.D) {
                    widen8<T>(xm[q], f);
                    if (!a.D_has_hdim) {
#pragma unroll
                        for (int e = 0; e < 8; ++e) y[e] = fmaf(f[e], Dh, y[e]);
                    } else {
#pragma unroll
                        for (int e = 0; e < 8; ++e)
                            if (e < left) y[e] = fmaf(f[e], a.D[(int64_t)h * P + p0 + 8 * c8 + e], y[e]);
                    }
                }
                if (z) {
                    widen8<T>(zm[q], f);
#pragma unroll
                    for (int e = 0; e < 8; ++e) y[e] *= silu(f[e]);
                }
                Raw8<T> o;
                T *oe = reinterpret_cast<T *>(&o);
#pragma unroll
                for (int e = 0; e < 8; ++e) oe[e] = from_float<T>(y[e]);
                T *om = out + (int64_t)(m0 + r) * a.out_stride[1];
                if (vo && left >= 8) {
                    *reinterpret_cast<Raw8<T> *>(om) = o;
                } else {
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        if (e < left) om[e] = oe[e];
                }
            }
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 256);
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
template <class F> int with_type(const mb200_ssd_args &a, F f) { return a.io_dtype == MB200_BF16 ? f(__nv_bfloat16{}) : a.io_dtype == MB200_F16 ? f(__half{}) : f(float{}); }

template <bool PACKED> int run_first(const mb200_ssd_args &a, const SsdScratch &lay, SsdStates form, bool with_states, bool with_cb, cudaStream_t stream)
{
    return with_type(a, [&](auto tag) -> int {
        using T = decltype(tag);
        const Buffers s(a, lay);
        const void *entering = static_cast<const char *>(a.scratch) + (form == SsdStates::pn32 ? lay.off_states : lay.off_prev16);
        const int units = (a.headdim + 63) / 64 * (a.nheads / a.ngroups), tilesN = (a.dstate + 127) / 128;
        const int cb_tiles = (a.chunk_size + 127) / 128 * ((a.chunk_size + 63) / 64);
        const int64_t rows = PACKED ? a.num_seqs : (int64_t)a.batch * lay.nchunks, cb_ctas = with_cb ? rows * cb_tiles * a.ngroups : 0;
        auto go = [&](auto u_c) -> int {
            constexpr int U = decltype(u_c)::value;
            const int state_tiles = (units + U - 1) / U * tilesN;
            const int64_t state_ctas = with_states ? rows * state_tiles * a.ngroups : 0, ctas = state_ctas + cb_ctas;
            if (ctas == 0) return MB200_OK;
            if (ctas > INT32_MAX) return fail(MB200_ERR_BAD_ARG, "ssd: too many chunks and heads");
            const uint32_t both = std::max(kStateSmem<T, U> + state_weight_bytes<U>(a), kCbSmem<T>), smem = state_ctas == 0 ? kCbSmem<T> : both;
            ensure_dynamic_smem(reinterpret_cast<const void *>(&ssd_split_first_kernel<T, PACKED, U>), (int)both, a.device);
            launch_dependent(ssd_split_first_kernel<T, PACKED, U>, dim3((unsigned)ctas), kThreads, smem, stream, a, s.dt, s.dA, entering, form, PACKED ? a.varlen_states : s.states,
                             s.cb, (int)state_ctas, state_tiles, cb_tiles, lay.nchunks, s.status);
            MB200_CHECK_LAUNCH("ssd states and C.B^T (split products)");
            return MB200_OK;
        };
        if constexpr (kInParts<T> > 1 && !PACKED) {
            const bool pairs = with_states && units > 1 && rows * units * tilesN * a.ngroups > (int64_t)(sizeof(T) == 2 ? 3 : 2) * sm_count(a.device);
            if (pairs) return go(std::integral_constant<int, 2>{});
        }
        return go(std::integral_constant<int, 1>{});
    });
}

}  // namespace

int ssd_split_first(const mb200_ssd_args &a, const SsdScratch &lay, bool with_states, bool with_cb, cudaStream_t stream)
{
    return run_first<false>(a, lay, SsdStates::pn32, with_states, with_cb, stream);
}
int ssd_split_varlen(const mb200_ssd_args &a, const SsdScratch &lay, SsdStates entering, cudaStream_t stream) { return run_first<true>(a, lay, entering, true, false, stream); }

int ssd_split_scan(const mb200_ssd_args &a, const SsdScratch &lay, cudaStream_t stream)
{
    return with_type(a, [&](auto tag) -> int {
        using T = decltype(tag);
        const Buffers s(a, lay);
        auto go = [&](auto kernel, int threads, uint32_t smem, int width) {
            smem += scan_decay_bytes(a);
            ensure_dynamic_smem(reinterpret_cast<const void *>(kernel), (int)smem, a.device);
            const unsigned tiles = (unsigned)((a.chunk_size + 127) / 128 * ((a.headdim + width - 1) / width));
            launch_dependent(kernel, dim3(tiles, a.batch * lay.nchunks, a.nheads), threads, smem, stream, a, s.dt, s.dA, s.states, s.cb, lay.nchunks, s.status);
        };
        if constexpr (sizeof(T) == 2) {
            const int64_t singles = (int64_t)((a.chunk_size + 127) / 128) * ((a.headdim + 63) / 64) * a.batch * lay.nchunks * a.nheads;
            if (a.headdim > 64 && singles > 2 * sm_count(a.device)) go(ssd_split_scan16_kernel<T, 2>, kThreads, kScan16A<T> + kScan16B<T, 2> + kTail, 128);
            else go(ssd_split_scan16_kernel<T, 1>, kThreads, kScan16A<T> + kScan16B<T, 1> + kTail, 64);
        } else {
            go(ssd_split_scan_kernel, kThreads, kScanTiles + kScanTail, 64);
        }
        MB200_CHECK_LAUNCH("ssd outputs (split products)");
        return MB200_OK;
    });
}

}  // namespace mb200
