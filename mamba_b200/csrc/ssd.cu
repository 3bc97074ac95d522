// Mamba-2 SSD chunked forward for sm_100a: the stages, and their kernels for fp32 inputs.
//
// Stages (each one launch, all on the caller's stream, handing fp32 intermediates through the
// caller's scratch buffer):
//   1. chunk_cumsum   dt <- clamp(softplus(dt + bias)), dA_cum <- cumsum_Q(dt A)
//   2. chunk_state    S_c[p,n] = sum_k x[k,p] B[k,n] exp(min(dA_last - dA_k, 0)) dt_k
//   3. state_passing  H_{c+1} = exp(dA_last_c) H_c + S_c, slot c rewritten with H_c
//   4. chunk_cb       CB[m,k] = C_m . B_k   (lower block triangle)
//   5. chunk_scan     y_m = exp(dA_m) C_m.H_c + sum_{k<=m} CB[m,k] exp(min(dA_m - dA_k,0)) dt_k x_k + D x_m,
//                     then y_m * silu(z_m)
// The contractions here run on the fp32 FMA pipes through a 64x64 shared-memory tile loop (tile_gemm) and serve fp32 inputs.  For
// bf16/fp16, ssd_tc.cu replaces stages 2 to 5 for the shape that most layers have, and ssd_split.cu stages 2, 4 and 5 for all others.
#include <algorithm>

#include "ssd_common.cuh"

namespace mb200 {
namespace {

constexpr int kT = 128;       // threads per CTA in the tile kernels
constexpr int kKT = 32;       // reduction step
constexpr int kLd = 68;       // padded leading dimension of the staged tiles (keeps float4 alignment)
struct TileSmem { __align__(16) float A[2][kKT * kLd], B[2][kKT * kLd]; };

// Four consecutive elements, in one load where `vec` says that they lie on their own alignment; zeros from `n` on.
__device__ __forceinline__ float4 load4(const float *p, bool vec, int n)
{
    if (vec && n >= 4) return *reinterpret_cast<const float4 *>(p);
    return make_float4(n > 0 ? p[0] : 0.f, n > 1 ? p[1] : 0.f, n > 2 ? p[2] : 0.f, n > 3 ? p[3] : 0.f);
}
__device__ __forceinline__ void store4(float *p, bool vec, int n, const float (&v)[4])
{
    if (vec && n >= 4) {
        *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (i < n) p[i] = v[i];
    }
}
// rows of a (batch, time, group or head, columns) tensor start where load4 can take four at once
__device__ __forceinline__ bool rows_of_4(const float *p, int64_t s0, int64_t s1, int64_t s2)
{
    return (reinterpret_cast<uintptr_t>(p) & 15) == 0 && ((s0 | s1 | s2) & 3) == 0;
}

// acc += A[64 x K] * B[K x 64] for the thread's 8x4 patch: rows ty*8.. in pairs (packed fp32 FMAs), columns tx*4...  fa and fb
// return four bounds-checked operand elements that follow each other in memory: (row, k..k+3) where the source is contiguous
// along k (KFAST), (k, column..column+3) otherwise; wa gives what fa loaded its final value when it is staged, a step later.  Terms
// are added in the order of k.
// What bounds it: with one buffer, a 4x4 patch and single elements staged, a step of 32 was a round trip to memory followed by
// two shared-memory reads per 16 FMAs (73 us for the outputs of 2 x 2048 steps of 8 fp32 heads of 64 x 64; now 54 us).  Here the next
// step's elements are on their way in registers while one is worked on, and three reads serve 32 FMAs.  A lane stages rows that
// are contiguous along k as 2 packets of 16 rows, which fills whole sectors and hits 32 different banks.
template <bool A_KFAST, bool B_KFAST, class FA, class WA, class FB>
__device__ __forceinline__ void tile_gemm(uint64_t (&acc)[4][4], int K, FA fa, WA wa, FB fb, TileSmem &sm)
{
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16, warp = threadIdx.x / 32, lane = threadIdx.x & 31;
    auto place = [&](bool kfast, int e, int &i, int &k) {       // of the e-th four elements of mine
        if (kfast) {
            const int block = warp * 4 + e;                     // 4 blocks of 16 rows x 4 pairs of packets
            i = (block >> 2) * 16 + (lane >> 1);
            k = ((block & 3) * 2 + (lane & 1)) * 4;
        } else {
            k = e * 8 + ty;
            i = tx * 4;
        }
    };
    float4 ra[4], rb[4];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            int i, k;
            place(A_KFAST, e, i, k);
            ra[e] = A_KFAST ? fa(i, k0 + k) : fa(k0 + k, i);
            place(B_KFAST, e, i, k);
            rb[e] = B_KFAST ? fb(i, k0 + k) : fb(k0 + k, i);
        }
    };
    auto stage = [&](float *dst, bool kfast, const float4 (&r)[4], auto final_value) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            int i, k;
            place(kfast, e, i, k);
            const float4 v = final_value(i, k, r[e]);
            if (kfast) {
                dst[k * kLd + i] = v.x;
                dst[(k + 1) * kLd + i] = v.y;
                dst[(k + 2) * kLd + i] = v.z;
                dst[(k + 3) * kLd + i] = v.w;
            } else {
                *reinterpret_cast<float4 *>(dst + k * kLd + i) = v;
            }
        }
    };
    if (K > 0) fetch(0);
    int buf = 0;
    __syncthreads();                // (a tile_gemm before this one may still be read)
    for (int k0 = 0; k0 < K; k0 += kKT, buf ^= 1) {
        stage(sm.A[buf], A_KFAST, ra, [&](int i, int k, float4 v) { return A_KFAST ? wa(i, k0 + k, v) : wa(k0 + k, i, v); });
        stage(sm.B[buf], B_KFAST, rb, [](int, int, float4 v) { return v; });
        __syncthreads();            // also: every warp is done with the other buffer
        if (k0 + kKT < K) fetch(k0 + kKT);
        const float *As = sm.A[buf] + ty * 8, *Bs = sm.B[buf] + tx * 4;
#pragma unroll 8
        for (int kk = 0; kk < kKT; ++kk) {
            const ulonglong2 a0 = *reinterpret_cast<const ulonglong2 *>(As + kk * kLd), a1 = *reinterpret_cast<const ulonglong2 *>(As + kk * kLd + 4);
            const float4 bv = *reinterpret_cast<const float4 *>(Bs + kk * kLd);
            const uint64_t ar[4] = {a0.x, a0.y, a1.x, a1.y}, br[4] = {pack2(bv.x, bv.x), pack2(bv.y, bv.y), pack2(bv.z, bv.z), pack2(bv.w, bv.w)};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fma2(ar[i], br[j], acc[i][j]);
        }
    }
}
__device__ __forceinline__ float4 as_loaded(int, int, float4 v) { return v; }
// the thread's patch row by row
__device__ __forceinline__ void patch_row(const uint64_t (&acc)[4][4], int i, float (&v)[4])
{
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        float lo, hi;
        unpack2(acc[i >> 1][j], lo, hi);
        v[j] = i & 1 ? hi : lo;
    }
}

// Sequence id of position t of batch row b (packed sequences), or 0 when no ids were given.
__device__ __forceinline__ int seq_at(const mb200_ssd_args &a, int b, int t)
{
    return a.seq_idx ? a.seq_idx[(int64_t)b * a.seqlen + t] : 0;
}

// ---- stage 1 ------------------------------------------------------------------------------------
// One CTA per (chunk, batch, 32 heads): coalesced read of dt over heads, transposed in shared memory, then a warp scan along
// the chunk per head.  Little is moved (5 MB in, 21 MB out for 8 x 4096 steps of 80 heads); the time is the chain load ->
// softplus -> barrier -> scan, so the eight 32-step scans of a head run side by side and only their totals are chained
// (18.9 -> 13.0 us for that size).  The first CTA clears the call's status word: no kernel that could set it is launched before.
// NW warps: 32, one per head, while all CTAs fit the GPU at once -- with eight the chain, and the code, which a small call fetches
// cold, are four times as long (1 x 777 steps of 80 heads: 9.2 -> 6.1 us).  Larger grids keep eight, which overlap their phases
// better (1 x 262144 steps of 128 heads: 113 us, 162 with 32).
template <typename TD, int NW>
__global__ void __launch_bounds__(NW * 32) ssd_cumsum_kernel(const mb200_ssd_args a, float *dt_out, float *dA_out, int nchunks, uint8_t *seq_start,
                                                         uint8_t *seq_carry, int *status)
{
    extern __shared__ float sm[];   // Q x 33
    const int Q = a.chunk_size;
    const int c = blockIdx.x, b = blockIdx.y, h0 = blockIdx.z * 32;
    const int t0 = c * Q;
    pdl_wait();
    pdl_trigger();        // the tensor-core stage that follows may set itself up, and load what was there before this launch
    if (threadIdx.x == 0 && (blockIdx.x | blockIdx.y | blockIdx.z) == 0) *status = 0;
    // a thread keeps one head (lane) and takes every NW-th step: the loads are issued back to back so
    // that their latencies overlap instead of adding up
    const int hh = threadIdx.x & 31, h = h0 + hh;
    const bool h_ok = h < a.nheads;
    const float bias = (h_ok && a.dt_bias) ? a.dt_bias[h] : 0.f;
    const TD *src = static_cast<const TD *>(a.dt) + (int64_t)b * a.dt_stride[0] + (int64_t)h * a.dt_stride[2];
    constexpr int NB = 256 / NW;    // loads in flight per thread: a whole chunk of 256 steps in one round trip
    for (int k0 = threadIdx.x >> 5; k0 < Q; k0 += NW * NB) {
        TD raw[NB];
#pragma unroll
        for (int u = 0; u < NB; ++u) {
            const int k = k0 + NW * u;
            raw[u] = (h_ok && k < Q && t0 + k < a.seqlen) ? src[(int64_t)(t0 + k) * a.dt_stride[1]] : from_float<TD>(0.f);
        }
#pragma unroll
        for (int u = 0; u < NB; ++u) {
            const int k = k0 + NW * u;
            if (k < Q) {
                float v = 0.f;
                if (h_ok && t0 + k < a.seqlen) {
                    v = to_float(raw[u]) + bias;
                    if (a.dt_softplus) v = fast_softplus20(v);
                    v = fminf(fmaxf(v, a.dt_min), a.dt_max);
                }
                sm[k * 33 + hh] = v;
            }
        }
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int hh = warp; hh < 32; hh += NW) {
        const int h = h0 + hh;
        if (h >= a.nheads) break;
        const float A = a.A[h];
        float carry = 0.f;
        const int64_t o = (((int64_t)b * a.nheads + h) * nchunks + c) * Q;
        for (int k0 = 0; k0 < Q; k0 += 256) {
            float dtv[8], v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int k = k0 + 32 * j + lane;
                dtv[j] = k < Q ? sm[k * 33 + hh] : 0.f;
                v[j] = dtv[j] * A;
            }
#pragma unroll
            for (int o2 = 1; o2 < 32; o2 <<= 1) {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float up = __shfl_up_sync(0xffffffffu, v[j], o2);
                    if (lane >= o2) v[j] += up;
                }
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int k = k0 + 32 * j + lane;
                const float tot = __shfl_sync(0xffffffffu, v[j], 31);
                if (k < Q) {
                    dt_out[o + k] = dtv[j];
                    dA_out[o + k] = v[j] + carry;
                }
                carry += tot;
            }
        }
    }
    // Packed sequences on the tensor-core path (chunk of 256 = one position per thread): where, inside the chunk, the
    // sequence of every position starts, and whether the chunk's first position continues the previous chunk's last
    // sequence.  The output kernel masks with these two instead of comparing ids.
    if (seq_start && blockIdx.z == 0) {
        __syncthreads();            // the transposing buffer is free
        int *wmax = reinterpret_cast<int *>(sm);
        const int32_t *sid = a.seq_idx + (int64_t)b * a.seqlen;
        const int k = threadIdx.x;
        const bool in = k < kTcChunk;
        const int me = in ? sid[min(t0 + k, a.seqlen - 1)] : 0;
        const int before = in && k > 0 ? sid[min(t0 + k - 1, a.seqlen - 1)] : me;
        int start = (k > 0 && me != before) ? k : 0;            // a sequence starts here
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) start = max(start, __shfl_up_sync(0xffffffffu, start, o) * (lane >= o ? 1 : 0));
        if (lane == 31) wmax[warp] = start;
        __syncthreads();
        if (in) {
            for (int w2 = 0; w2 < warp; ++w2) start = max(start, wmax[w2]);
            seq_start[((int64_t)b * nchunks + c) * Q + k] = (uint8_t)start;
            if (k == 0) seq_carry[(int64_t)b * nchunks + c] = me == (c > 0 ? sid[t0 - 1] : 0) ? 1 : 0;
        }
    }
}

// ---- stage 2 ------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kT, 4) ssd_chunk_state_kernel(const mb200_ssd_args a, const float *dtb, const float *dAb,
                                                             float *states, int nchunks)
{
    __shared__ TileSmem sm;
    const int Q = a.chunk_size, P = a.headdim, N = a.dstate;
    const int tilesN = (N + 63) / 64;
    const int p0 = (blockIdx.x / tilesN) * 64, n0 = (blockIdx.x % tilesN) * 64;
    const int b = blockIdx.y / nchunks, c = blockIdx.y % nchunks, h = blockIdx.z;
    const int g = h / (a.nheads / a.ngroups);
    const int t0 = c * Q;
    const int len = min(Q, a.seqlen - t0);
    const float *dtc = dtb + (((int64_t)b * a.nheads + h) * nchunks + c) * Q;
    const float *dAc = dAb + (((int64_t)b * a.nheads + h) * nchunks + c) * Q;
    const float dA_last = dAc[Q - 1];
    const float *x = static_cast<const float *>(a.x) + (int64_t)b * a.x_stride[0] + (int64_t)t0 * a.x_stride[1] + (int64_t)h * a.x_stride[2];
    const float *B = static_cast<const float *>(a.B) + (int64_t)b * a.B_stride[0] + (int64_t)t0 * a.B_stride[1] + (int64_t)g * a.B_stride[2];
    const bool vx = rows_of_4(x, 0, a.x_stride[1], 0), vB = rows_of_4(B, 0, a.B_stride[1], 0);
    uint64_t acc[4][4] = {};
    const int seq_last = seq_at(a, b, t0 + len - 1);    // only steps of the chunk's last sequence reach its end state
    tile_gemm<false, false>(
        acc, len,
        [&](int k, int i) {
            const bool in = k < len && (!a.seq_idx || seq_at(a, b, t0 + k) == seq_last);
            return load4(x + (int64_t)k * a.x_stride[1] + p0 + i, vx, in ? P - p0 - i : 0);
        },
        [&](int k, int, float4 v) {
            const float w = k < len ? __expf(fminf(dA_last - dAc[k], 0.f)) * dtc[k] : 0.f;
            return make_float4(v.x * w, v.y * w, v.z * w, v.w * w);
        },
        [&](int k, int j) { return load4(B + (int64_t)k * a.B_stride[1] + n0 + j, vB, k < len ? N - n0 - j : 0); }, sm);
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16, n = n0 + tx * 4;
    float *S = states + (((int64_t)b * nchunks + c) * a.nheads + h) * (int64_t)P * N;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int p = p0 + ty * 8 + i;
        float v[4];
        patch_row(acc, i, v);
        if (p < P && n < N) store4(S + (int64_t)p * N + n, (N & 3) == 0, N - n, v);
    }
}

// ---- stage 3 ------------------------------------------------------------------------------------
// Elementwise over P*N, serial over chunks.  Slot c of `states` receives the state entering chunk c;
// with `prev16` the entering states go there as 16-bit values (the tensor-core chunk_scan reads them
// by TMA) and the fp32 slots are left alone.  VEC elements per thread and kAhead chunks of loads in
// flight keep enough bytes in the air to stream at HBM speed.
template <int VEC>
__global__ void __launch_bounds__(256) ssd_state_passing_kernel(const mb200_ssd_args a, const float *dAb, float *states,
                                                                int nchunks, bool write_prev, void *prev16)
{
    constexpr int kAhead = 4;
    const int64_t PN = (int64_t)a.headdim * a.dstate;
    const int64_t e = ((int64_t)blockIdx.x * 256 + threadIdx.x) * VEC;
    const int h = blockIdx.y, b = blockIdx.z;
    const int Q = a.chunk_size;
    const float *dA_last = dAb + ((int64_t)b * a.nheads + h) * nchunks * Q + (Q - 1);
    if (e < PN) {
        float run[VEC];
#pragma unroll
        for (int i = 0; i < VEC; ++i) run[i] = a.initial_states ? a.initial_states[((int64_t)b * a.nheads + h) * PN + e + i] : 0.f;
        for (int c0 = 0; c0 < nchunks; c0 += kAhead) {
            float s[kAhead][VEC], dec[kAhead];
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                const int c = c0 + u;
                if (c < nchunks) {
                    const float *slot = states + (((int64_t)b * nchunks + c) * a.nheads + h) * PN + e;
                    if (VEC == 4) {
                        const float4 v = *reinterpret_cast<const float4 *>(slot);
                        s[u][0] = v.x; s[u][1 % VEC] = v.y; s[u][2 % VEC] = v.z; s[u][3 % VEC] = v.w;
                    } else {
                        s[u][0] = slot[0];
                    }
                    dec[u] = __expf(dA_last[(int64_t)c * Q]);
                    if (a.seq_idx) {   // a new sequence at the end of this chunk: nothing carries over from the previous one
                        const int s_new = seq_at(a, b, min((c + 1) * Q, a.seqlen) - 1);
                        const int s_old = c > 0 ? seq_at(a, b, c * Q - 1) : 0;
                        if (s_new != s_old) dec[u] = 0.f;
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                const int c = c0 + u;
                if (c < nchunks) {
                    const int64_t o = (((int64_t)b * nchunks + c) * a.nheads + h) * PN + e;
                    if (write_prev) {
#pragma unroll
                        for (int i = 0; i < VEC; ++i) {
                            if (prev16) store_any(prev16, a.io_dtype, o + i, run[i]);
                            else states[o + i] = run[i];
                        }
                    }
#pragma unroll
                    for (int i = 0; i < VEC; ++i) run[i] = fmaf(dec[u], run[i], s[u][i]);
                }
            }
        }
        if (a.final_states) {
#pragma unroll
            for (int i = 0; i < VEC; ++i) a.final_states[((int64_t)b * a.nheads + h) * PN + e + i] = run[i];
        }
    }
    if (a.range_decay && blockIdx.x == 0 && threadIdx.x == 0) {
        float tot = 0.f;
        for (int c = 0; c < nchunks; ++c) tot += dA_last[(int64_t)c * Q];
        a.range_decay[(int64_t)b * a.nheads + h] = __expf(tot);
    }
}

// ---- stage 4 ------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kT, 4) ssd_cb_kernel(const mb200_ssd_args a, float *cb, int nchunks)
{
    __shared__ TileSmem sm;
    const int Q = a.chunk_size, N = a.dstate;
    const int tiles = (Q + 63) / 64;
    const int m0 = (blockIdx.x / tiles) * 64, k0 = (blockIdx.x % tiles) * 64;
    if (k0 > m0) return;   // strictly upper blocks are never read
    const int b = blockIdx.y / nchunks, c = blockIdx.y % nchunks, g = blockIdx.z;
    const int t0 = c * Q;
    const int len = min(Q, a.seqlen - t0);
    const float *C = static_cast<const float *>(a.C) + (int64_t)b * a.C_stride[0] + (int64_t)t0 * a.C_stride[1] + (int64_t)g * a.C_stride[2];
    const float *B = static_cast<const float *>(a.B) + (int64_t)b * a.B_stride[0] + (int64_t)t0 * a.B_stride[1] + (int64_t)g * a.B_stride[2];
    const bool vC = rows_of_4(C, 0, a.C_stride[1], 0), vB = rows_of_4(B, 0, a.B_stride[1], 0);
    uint64_t acc[4][4] = {};
    tile_gemm<true, true>(
        acc, N, [&](int i, int n) { return load4(C + (int64_t)(m0 + i) * a.C_stride[1] + n, vC, m0 + i < len ? N - n : 0); }, as_loaded,
        [&](int j, int n) { return load4(B + (int64_t)(k0 + j) * a.B_stride[1] + n, vB, k0 + j < len ? N - n : 0); }, sm);
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16, k = k0 + tx * 4;
    float *out = cb + (((int64_t)b * nchunks + c) * a.ngroups + g) * (int64_t)Q * Q;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int m = m0 + ty * 8 + i;
        float v[4];
        patch_row(acc, i, v);
        if (a.seq_idx) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (!(m < len && k + j < len && seq_at(a, b, t0 + m) == seq_at(a, b, t0 + k + j))) v[j] = 0.f;
        }
        if (m < Q && k < Q) store4(out + (int64_t)m * Q + k, (Q & 3) == 0, Q - k, v);
    }
}

// ---- stage 5 ------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kT, 4) ssd_chunk_scan_kernel(const mb200_ssd_args a, const float *dtb, const float *dAb,
                                                            const float *states, const float *cb, int nchunks)
{
    __shared__ TileSmem sm;
    const int Q = a.chunk_size, P = a.headdim, N = a.dstate;
    const int tilesP = (P + 63) / 64;
    const int m0 = (blockIdx.x / tilesP) * 64, p0 = (blockIdx.x % tilesP) * 64;
    const int b = blockIdx.y / nchunks, c = blockIdx.y % nchunks, h = blockIdx.z;
    const int g = h / (a.nheads / a.ngroups);
    const int t0 = c * Q;
    const int len = min(Q, a.seqlen - t0);
    if (m0 >= len) return;
    const float *dtc = dtb + (((int64_t)b * a.nheads + h) * nchunks + c) * Q;
    const float *dAc = dAb + (((int64_t)b * a.nheads + h) * nchunks + c) * Q;
    const float *x = static_cast<const float *>(a.x) + (int64_t)b * a.x_stride[0] + (int64_t)t0 * a.x_stride[1] + (int64_t)h * a.x_stride[2];
    const float *C = static_cast<const float *>(a.C) + (int64_t)b * a.C_stride[0] + (int64_t)t0 * a.C_stride[1] + (int64_t)g * a.C_stride[2];
    const float *prev = states + (((int64_t)b * nchunks + c) * a.nheads + h) * (int64_t)P * N;
    const float *cbc = cb + (((int64_t)b * nchunks + c) * a.ngroups + g) * (int64_t)Q * Q;
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    const bool vx = rows_of_4(x, 0, a.x_stride[1], 0), vC = rows_of_4(C, 0, a.C_stride[1], 0), vN = (N & 3) == 0, vQ = (Q & 3) == 0;

    uint64_t acc[4][4] = {};
    // contribution of the state entering the chunk: exp(dA_m) * C_m . H[p,:]
    tile_gemm<true, true>(
        acc, N, [&](int i, int n) { return load4(C + (int64_t)(m0 + i) * a.C_stride[1] + n, vC, m0 + i < len ? N - n : 0); }, as_loaded,
        [&](int j, int n) { return load4(prev + (int64_t)(p0 + j) * N + n, vN, p0 + j < P ? N - n : 0); }, sm);
    float sc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int m = m0 + ty * 8 + i;
        sc[i] = m < len ? __expf(dAc[m]) : 0.f;
        // the entering state belongs to the sequence that ends the previous chunk
        if (a.seq_idx && m < len && seq_at(a, b, t0 + m) != (c > 0 ? seq_at(a, b, t0 - 1) : 0)) sc[i] = 0.f;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = mul2(acc[i][j], pack2(sc[2 * i], sc[2 * i + 1]));
    // causal intra-chunk part
    const int kend = min(m0 + 64, len);
    tile_gemm<true, false>(
        acc, kend,
        [&](int i, int k) {
            const int m = m0 + i;                       // columns up to the diagonal
            return load4(cbc + (int64_t)m * Q + k, vQ, m < len ? min(m + 1, kend) - k : 0);
        },
        [&](int i, int k, float4 v) {
            const int n = min(m0 + i + 1, kend) - k;
            const float4 d = load4(dAc + k, vQ, n), t = load4(dtc + k, vQ, n);
            const float dm = dAc[min(m0 + i, len - 1)];
            return make_float4(v.x * __expf(fminf(dm - d.x, 0.f)) * t.x, v.y * __expf(fminf(dm - d.y, 0.f)) * t.y,
                               v.z * __expf(fminf(dm - d.z, 0.f)) * t.z, v.w * __expf(fminf(dm - d.w, 0.f)) * t.w);
        },
        [&](int k, int j) { return load4(x + (int64_t)k * a.x_stride[1] + p0 + j, vx, k < kend ? P - p0 - j : 0); }, sm);

    const float *z = a.z ? static_cast<const float *>(a.z) + (int64_t)b * a.z_stride[0] + (int64_t)t0 * a.z_stride[1] + (int64_t)h * a.z_stride[2] : nullptr;
    float *out = static_cast<float *>(a.out) + (int64_t)b * a.out_stride[0] + (int64_t)t0 * a.out_stride[1] + (int64_t)h * a.out_stride[2];
    const bool vz = z && rows_of_4(z, 0, a.z_stride[1], 0), vo = rows_of_4(out, 0, a.out_stride[1], 0);
    const int p = p0 + tx * 4, np = P - p;
    if (np <= 0) return;
    float Dv[4] = {};
    if (a.D) {
#pragma unroll
        for (int j = 0; j < 4; ++j) Dv[j] = a.D_has_hdim ? (j < np ? a.D[(int64_t)h * P + p + j] : 0.f) : a.D[h];
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int m = m0 + ty * 8 + i;
        if (m >= len) continue;
        float y[4];
        patch_row(acc, i, y);
        if (a.D) {
            const float4 v = load4(x + (int64_t)m * a.x_stride[1] + p, vx, np);
            y[0] = fmaf(v.x, Dv[0], y[0]); y[1] = fmaf(v.y, Dv[1], y[1]); y[2] = fmaf(v.z, Dv[2], y[2]); y[3] = fmaf(v.w, Dv[3], y[3]);
        }
        if (z) {
            const float4 v = load4(z + (int64_t)m * a.z_stride[1] + p, vz, np);
            y[0] *= silu(v.x); y[1] *= silu(v.y); y[2] *= silu(v.z); y[3] *= silu(v.w);
        }
        store4(out + (int64_t)m * a.out_stride[1] + p, vo, np, y);
    }
}

// ---- packed sequences: state after the last token of each one ------------------------------------
// A 64 x 64 tile of one (sequence, head): the contribution of the sequence's steps inside the chunk that holds its last
// token, plus the state entering that chunk if the sequence began earlier.
__global__ void __launch_bounds__(kT, 4) ssd_varlen_state_kernel(const mb200_ssd_args a, const float *dtb, const float *dAb, const float *states, int nchunks)
{
    __shared__ TileSmem sm;
    const int P = a.headdim, N = a.dstate, Q = a.chunk_size;
    const int tilesN = (N + 63) / 64;
    const int p0 = (blockIdx.x / tilesN) * 64, n0 = (blockIdx.x % tilesN) * 64;
    const int s = blockIdx.y, h = blockIdx.z;
    const int g = h / (a.nheads / a.ngroups);
    const int start = a.cu_seqlens[s], end = a.cu_seqlens[s + 1];
    const bool empty = end <= start || end > a.seqlen || start < 0;
    const int c = empty ? 0 : (end - 1) / Q, t0 = c * Q;
    const int first = empty ? 0 : max(start, t0);
    const float *dtc = dtb + ((int64_t)h * nchunks + c) * Q + (first - t0);
    const float *dAc = dAb + ((int64_t)h * nchunks + c) * Q + (first - t0);
    const float dA_end = empty ? 0.f : dAc[end - 1 - first];
    const float *x = static_cast<const float *>(a.x) + (int64_t)first * a.x_stride[1] + (int64_t)h * a.x_stride[2];
    const float *B = static_cast<const float *>(a.B) + (int64_t)first * a.B_stride[1] + (int64_t)g * a.B_stride[2];
    const bool vx = rows_of_4(x, 0, a.x_stride[1], 0), vB = rows_of_4(B, 0, a.B_stride[1], 0);
    const int steps = empty ? 0 : end - first;
    uint64_t acc[4][4] = {};
    tile_gemm<false, false>(
        acc, steps,
        [&](int k, int i) {
            return load4(x + (int64_t)k * a.x_stride[1] + p0 + i, vx, k < steps ? P - p0 - i : 0);
        },
        [&](int k, int, float4 v) {
            const float w = k < steps ? __expf(fminf(dA_end - dAc[k], 0.f)) * dtc[k] : 0.f;
            return make_float4(v.x * w, v.y * w, v.z * w, v.w * w);
        },
        [&](int k, int j) { return load4(B + (int64_t)k * a.B_stride[1] + n0 + j, vB, k < steps ? N - n0 - j : 0); }, sm);
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16, n = n0 + tx * 4;
    const float *entering = !empty && start < t0 ? states + (((int64_t)c) * a.nheads + h) * (int64_t)P * N : nullptr;
    const float decay = __expf(dA_end);
    float *dst = a.varlen_states + ((int64_t)s * a.nheads + h) * P * N;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int p = p0 + ty * 8 + i;
        if (p >= P || n >= N) continue;
        const int64_t e = (int64_t)p * N + n;
        float v[4];
        patch_row(acc, i, v);
        if (entering) {
            const float4 in = load4(entering + e, (N & 3) == 0, N - n);
            v[0] = fmaf(in.x, decay, v[0]); v[1] = fmaf(in.y, decay, v[1]); v[2] = fmaf(in.z, decay, v[2]); v[3] = fmaf(in.w, decay, v[3]);
        }
        store4(dst + e, (N & 3) == 0, N - n, v);
    }
}

__global__ void ssd_fill_kernel(float *dst, float v, int64_t n)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = v;
}

__global__ void ssd_fold_kernel(const float *s_in, const float *decay, const float *s_local, float *s_out, int64_t rows,
                                int64_t row)
{
    const int64_t total = rows * row;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const float in = s_in ? s_in[i] : 0.f;
        s_out[i] = fmaf(decay[i / row], in, s_local[i]);
    }
}

__global__ void ssd_fold_ranges_kernel(const float *summaries, int64_t record_stride, int first, int last, float *s_out, int64_t rows,
                                       int64_t row)
{
    const int64_t total = rows * row;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        float s = summaries[(int64_t)first * record_stride + i];
        for (int r = first + 1; r <= last; ++r) {
            const float *rec = summaries + (int64_t)r * record_stride;
            s = fmaf(rec[total + i / row], s, rec[i]);
        }
        s_out[i] = s;
    }
}

int run_ssd(const mb200_ssd_args &a, const SsdScratch &lay, cudaStream_t stream)
{
    char *base = static_cast<char *>(a.scratch);
    float *dtb = reinterpret_cast<float *>(base + lay.off_dt);
    float *dAb = reinterpret_cast<float *>(base + lay.off_dA);
    float *states = reinterpret_cast<float *>(base + lay.off_states);
    float *cb = reinterpret_cast<float *>(base + lay.off_cb);
    int *status = ssd_status_word(a, lay);
    const int nc = lay.nchunks, Q = a.chunk_size;
    const int64_t PN = (int64_t)a.headdim * a.dstate;
    // Path choice.  The LOCAL stages (cumsum, chunk states, recurrence) read x, B and dt; the OUTPUT stages add C,
    // z and out.  A whole-operator call takes the tensor-core path only when both halves can; in a sequence split
    // each half decides from what IT reads, so an OUTPUT call can tell how the earlier LOCAL call ran even though
    // that call never saw C, z or out.
    const bool has_local = (a.phases & MB200_SSD_PHASE_LOCAL) != 0, has_out = (a.phases & MB200_SSD_PHASE_OUTPUT) != 0;
    const bool tc_out = ssd_tc_local_eligible(a) && ssd_tc_output_eligible(a);     // OUTPUT stages on tensor cores
    const bool tc_loc = (has_local && has_out) ? tc_out : ssd_tc_local_eligible(a);  // LOCAL stages on tensor cores
    // C.B^T ahead of the exchange of a sequence split: the tensor-core output kernel forms its own, so only a call whose C
    // rules that kernel out (which both halves can tell: they are handed the same C) does it.
    const bool tc_cb = ssd_tc_local_eligible(a) && ssd_tc_cb_eligible(a);
    const bool cb_early = has_local && !has_out && (a.phases & MB200_SSD_PHASE_CB) && a.C && !tc_cb;
    const bool cb_ready = !has_local && has_out && (a.phases & MB200_SSD_PHASE_CB_READY) && !tc_cb;
    void *prev16 = tc_out ? static_cast<void *>(base + lay.off_prev16) : nullptr;
    if (!has_local) {      // the cumsum kernel of the LOCAL stages clears the word otherwise
        cudaError_t e = cudaMemsetAsync(status, 0, sizeof(int), stream);
        if (e != cudaSuccess) return fail(MB200_ERR_LAUNCH, "ssd: status reset: %s", cudaGetErrorString(e));
    }
    // Chunk states + inter-chunk recurrence in one streaming launch.  In a sequence split the LOCAL phase runs it
    // from a zero state (entering states of the range as if nothing came in, range summary), and the OUTPUT phase
    // adds the incoming state's share to those entering states: H_c += prefix_decay_c * S_in.
    const bool fused_states = tc_loc && ssd_tc_stream_eligible(a);
    // The LOCAL half took the streaming launch but this OUTPUT half cannot use its 16-bit entering states: the
    // scratch holds no fp32 chunk states, so they are formed here before the recurrence.
    const bool local_streamed = !has_local && fused_states && !tc_out;
    const bool split = a.io_dtype != MB200_F32;       // the general stages for 16-bit inputs
    const int tq = (Q + 63) / 64, tp = (a.headdim + 63) / 64, tn = (a.dstate + 63) / 64;
    auto form_cb = [&]() -> int {
        if (split) return ssd_split_cb(a, lay, stream);
        ssd_cb_kernel<<<dim3(tq * tq, a.batch * nc, a.ngroups), kT, 0, stream>>>(a, cb, nc);
        MB200_CHECK_LAUNCH("ssd chunk_cb");
        return MB200_OK;
    };
    auto state_passing = [&](const mb200_ssd_args &p, bool write_prev, void *to16) {
        if (PN % 4 == 0)
            ssd_state_passing_kernel<4><<<dim3((unsigned)((PN / 4 + 255) / 256), a.nheads, a.batch), 256, 0, stream>>>(p, dAb, states, nc, write_prev, to16);
        else
            ssd_state_passing_kernel<1><<<dim3((unsigned)((PN + 255) / 256), a.nheads, a.batch), 256, 0, stream>>>(p, dAb, states, nc, write_prev, to16);
    };
    if (has_local) {
        const size_t cs_smem = sizeof(float) * Q * 33;
        // the sequence-start table is only read by the tensor-core output kernel (chunk of 256 positions = one per thread)
        uint8_t *seq_start = (a.seq_idx && tc_out) ? reinterpret_cast<uint8_t *>(base + lay.off_seq_start) : nullptr;
        uint8_t *seq_carry = reinterpret_cast<uint8_t *>(base + lay.off_seq_carry);
        auto cumsum = [&](auto tag) -> cudaError_t {
            using TD = decltype(tag);
            const dim3 grid(nc, a.batch, (a.nheads + 31) / 32);
            auto go = [&](auto nw_c) {
                constexpr int NW = decltype(nw_c)::value;
                if (cs_smem > 48 * 1024)
                    if (cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void *>(&ssd_cumsum_kernel<TD, NW>), (int)cs_smem, a.device)) return e;
                launch_dependent(ssd_cumsum_kernel<TD, NW>, grid, NW * 32, cs_smem, stream, a, dtb, dAb, nc, seq_start, seq_carry, status);
                return cudaSuccess;
            };
            return (int64_t)grid.x * grid.y * grid.z <= 2 * 148 ? go(std::integral_constant<int, 32>{}) : go(std::integral_constant<int, 8>{});
        };
        const cudaError_t ce = a.dt_dtype == MB200_F32 ? cumsum(float{}) : a.dt_dtype == MB200_BF16 ? cumsum(__nv_bfloat16{}) : cumsum(__half{});
        if (ce != cudaSuccess) return fail(MB200_ERR_LAUNCH, "ssd chunk_cumsum: shared memory opt-in: %s", cudaGetErrorString(ce));
        MB200_CHECK_LAUNCH("ssd chunk_cumsum");
        if (cb_early)
            if (int rc = form_cb()) return rc;
        if (fused_states) {
            if (int rc = ssd_tc_state_stream(a, lay, stream)) return rc;
        } else if (tc_loc) {
            if (int rc = ssd_tc_chunk_state(a, lay, stream)) return rc;
        } else if (split) {
            if (int rc = ssd_split_states(a, lay, stream)) return rc;
        } else {
            ssd_chunk_state_kernel<<<dim3(tp * tn, a.batch * nc, a.nheads), kT, 0, stream>>>(a, dtb, dAb, states, nc);
            MB200_CHECK_LAUNCH("ssd chunk_state");
        }
        if (!fused_states && !has_out && (a.final_states || a.range_decay)) {
            // range summary only: fold the local chunk states from a zero state, leave the slots as they are
            mb200_ssd_args z = a;
            z.initial_states = nullptr;
            state_passing(z, false, nullptr);
            MB200_CHECK_LAUNCH("ssd range summary");
        }
    }
    if (has_out) {
        mb200_ssd_args p = a;
        if (!has_local) p.range_decay = nullptr;
        if (local_streamed)      // x and B qualified for the tensor-core chunk-state kernel (that is why LOCAL streamed)
            if (int rc = ssd_tc_chunk_state(a, lay, stream)) return rc;
        if (fused_states && tc_out) {
            // the entering states and the final state come from the state-stream kernel; in the OUTPUT half of a
            // sequence split the incoming state is added to what the LOCAL half left
            if (!has_local)
                if (int rc = ssd_tc_apply_incoming(a, lay, stream)) return rc;
        } else {
            state_passing(p, true, prev16);
        }
        MB200_CHECK_LAUNCH("ssd state_passing");
        const bool varlen = a.cu_seqlens && a.varlen_states && a.num_seqs > 0;
        if (tc_out) {
            if (int rc = ssd_tc_output(a, lay, fused_states, stream)) return rc;
            if (varlen)
                if (int rc = a.io_dtype == MB200_BF16 ? ssd_tc_varlen(a, lay, fused_states, stream)
                                                      : ssd_split_varlen(a, lay, fused_states ? SsdStates::np16 : SsdStates::pn16, stream))
                    return rc;
        } else {
            if (!cb_ready)
                if (int rc = form_cb()) return rc;
            if (split) {
                if (int rc = ssd_split_scan(a, lay, stream)) return rc;
                if (varlen)
                    if (int rc = ssd_split_varlen(a, lay, SsdStates::pn32, stream)) return rc;
            } else {
                ssd_chunk_scan_kernel<<<dim3(tq * tp, a.batch * nc, a.nheads), kT, 0, stream>>>(a, dtb, dAb, states, cb, nc);
                MB200_CHECK_LAUNCH("ssd chunk_scan");
                if (varlen) {
                    ssd_varlen_state_kernel<<<dim3(tp * tn, a.num_seqs, a.nheads), kT, 0, stream>>>(a, dtb, dAb, states, nc);
                    MB200_CHECK_LAUNCH("ssd varlen states");
                }
            }
        }
    }
    return MB200_OK;
}

int check_ssd(const mb200_ssd_args &a)
{
    MB200_CHECK_ARG(a.batch >= 0 && a.seqlen >= 0 && a.nheads > 0 && a.headdim > 0 && a.ngroups > 0 && a.dstate > 0 && a.chunk_size > 0,
                    "ssd: bad sizes (batch %d seqlen %d nheads %d headdim %d ngroups %d dstate %d chunk %d)", a.batch, a.seqlen,
                    a.nheads, a.headdim, a.ngroups, a.dstate, a.chunk_size);
    MB200_CHECK_ARG(a.nheads % a.ngroups == 0, "nheads must be divisible by ngroups");
    MB200_CHECK_ARG(a.io_dtype == MB200_F32 || a.io_dtype == MB200_F16 || a.io_dtype == MB200_BF16, "ssd: unknown io_dtype %d", a.io_dtype);
    MB200_CHECK_ARG(a.dt_dtype == MB200_F32 || a.dt_dtype == MB200_F16 || a.dt_dtype == MB200_BF16, "ssd: unknown dt_dtype %d", a.dt_dtype);
    MB200_CHECK_ARG(a.chunk_size <= 1024, "ssd: chunk_size must be <= 1024");
    MB200_CHECK_ARG((a.phases & MB200_SSD_PHASE_ALL) != 0 && (a.phases & ~(MB200_SSD_PHASE_ALL | MB200_SSD_PHASE_CB | MB200_SSD_PHASE_CB_READY)) == 0,
                    "ssd: phases must be a combination of LOCAL and OUTPUT");
    MB200_CHECK_ARG(!(a.phases & MB200_SSD_PHASE_CB) || (a.phases & MB200_SSD_PHASE_ALL) == MB200_SSD_PHASE_LOCAL, "ssd: PHASE_CB goes with a LOCAL-only call");
    MB200_CHECK_ARG(!(a.phases & MB200_SSD_PHASE_CB_READY) || (a.phases & MB200_SSD_PHASE_ALL) == MB200_SSD_PHASE_OUTPUT,
                    "ssd: PHASE_CB_READY goes with an OUTPUT-only call");
    return MB200_OK;
}

}  // namespace
}  // namespace mb200

extern "C" int mb200_ssd_scratch_bytes(const mb200_ssd_args *args, size_t *bytes)
{
    using namespace mb200;
    if (!args || !bytes) return fail(MB200_ERR_BAD_ARG, "ssd_scratch_bytes: NULL argument");
    if (int rc = check_ssd(*args)) return rc;
    *bytes = ssd_scratch_layout(*args).total;
    return MB200_OK;
}

extern "C" int mb200_ssd_chunk_scan_fwd(const mb200_ssd_args *args, void *stream_)
{
    using namespace mb200;
    if (!args) return fail(MB200_ERR_BAD_ARG, "ssd_chunk_scan_fwd: args is NULL");
    const mb200_ssd_args &a = *args;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (int rc = check_ssd(a)) return rc;
    MB200_CHECK_ARG(!(a.phases & MB200_SSD_PHASE_OUTPUT) || a.out || a.seqlen == 0 || a.batch == 0, "ssd: out is NULL");
    MB200_CHECK_ARG(!a.cu_seqlens || a.batch == 1, "passing cu_seqlens to get the varlen states is only supported if batch dimension is 1");
    MB200_CHECK_ARG(!a.cu_seqlens || (a.num_seqs >= 0 && a.num_seqs <= 65535), "ssd: num_seqs must be in [0, 65535]");
    MB200_CHECK_ARG(!(a.seq_idx || a.cu_seqlens) || (a.phases & MB200_SSD_PHASE_ALL) == MB200_SSD_PHASE_ALL, "ssd: packed sequences cannot be combined with a sequence split");
    if (a.batch == 0) return MB200_OK;   // nothing to do; empty tensors carry NULL pointers
    MB200_CHECK_ARG(a.seqlen == 0 || (a.x && a.dt && a.A && a.B && a.C), "ssd: a required tensor is NULL");
    if (int rc = enter_device(a.device)) return rc;
    MB200_CHECK_ARG(a.batch * (int64_t)((a.seqlen + a.chunk_size - 1) / a.chunk_size) <= 65535 && a.nheads <= 65535 && a.batch <= 65535,
                    "ssd: batch*nchunks and nheads must be <= 65535");
    if (a.seqlen == 0) {
        const size_t n = sizeof(float) * (size_t)a.batch * a.nheads * a.headdim * a.dstate;
        if (a.final_states && (a.phases & MB200_SSD_PHASE_OUTPUT)) {
            cudaError_t e = a.initial_states ? cudaMemcpyAsync(a.final_states, a.initial_states, n, cudaMemcpyDeviceToDevice, stream)
                                             : cudaMemsetAsync(a.final_states, 0, n, stream);
            if (e != cudaSuccess) return fail(MB200_ERR_LAUNCH, "ssd: final state copy: %s", cudaGetErrorString(e));
        } else if ((a.phases & MB200_SSD_PHASE_ALL) == MB200_SSD_PHASE_LOCAL) {
            // an empty range of a sequence split is summarised by the identity: state 0, decay 1
            if (a.final_states) {
                const cudaError_t e = cudaMemsetAsync(a.final_states, 0, n, stream);
                if (e != cudaSuccess) return fail(MB200_ERR_LAUNCH, "ssd: empty range state: %s", cudaGetErrorString(e));
            }
            if (a.range_decay) {
                const int64_t rows = (int64_t)a.batch * a.nheads;
                ssd_fill_kernel<<<(unsigned)((rows + 255) / 256), 256, 0, stream>>>(a.range_decay, 1.f, rows);
                MB200_CHECK_LAUNCH("ssd: empty range decay");
            }
        }
        return MB200_OK;
    }
    const SsdScratch lay = ssd_scratch_layout(a);
    MB200_CHECK_ARG(a.scratch && a.scratch_bytes >= lay.total, "ssd: scratch too small (%zu < %zu bytes)", a.scratch_bytes, lay.total);
    MB200_CHECK_ARG((reinterpret_cast<uintptr_t>(a.scratch) & 255) == 0, "ssd: scratch must be 256-byte aligned");
    return run_ssd(a, lay, stream);
}

// ---- the variant that allocates nothing ---------------------------------------------------------------
// The intermediates of the SSD stages for callers that cannot allocate: a fixed buffer inside the
// library image.  In host code this name is only a handle for the runtime, not a device address; the
// address each device gave it is fetched once per device with cudaGetSymbolAddress below.
static __device__ __align__(256) unsigned char g_ssd_static_scratch[MB200_SSD_STATIC_SCRATCH_BYTES];

extern "C" int mb200_ssd_chunk_scan_fwd_static(const mb200_ssd_args *args, void *stream)
{
    using namespace mb200;
    if (!args) return fail(MB200_ERR_BAD_ARG, "ssd_chunk_scan_fwd_static: args is NULL");
    if (int rc = check_ssd(*args)) return rc;
    const size_t need = ssd_scratch_layout(*args).total;
    if (need > MB200_SSD_STATIC_SCRATCH_BYTES)
        return fail(MB200_ERR_BAD_ARG,
                    "ssd_chunk_scan_fwd_static: this problem needs %zu bytes of intermediates, the built-in buffer holds %u; "
                    "use mb200_ssd_chunk_scan_fwd with caller-owned scratch",
                    need, (unsigned)MB200_SSD_STATIC_SCRATCH_BYTES);
    if (args->batch == 0) return MB200_OK;
    if (int rc = enter_device(args->device)) return rc;
    // one look-up per device, made with that device current (enter_device did that)
    static void *device_address[64] = {nullptr};
    void *ptr = device_address[args->device];
    if (!ptr) {
        const cudaError_t e = cudaGetSymbolAddress(&ptr, g_ssd_static_scratch);
        if (e != cudaSuccess || !ptr)
            return fail(MB200_ERR_LAUNCH, "ssd_chunk_scan_fwd_static: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
        device_address[args->device] = ptr;
    }
    mb200_ssd_args a = *args;
    a.scratch = ptr;
    a.status = nullptr;      // mb200_ssd_static_status reads the word in the built-in buffer
    a.scratch_bytes = MB200_SSD_STATIC_SCRATCH_BYTES;
    return mb200_ssd_chunk_scan_fwd(&a, stream);
}

extern "C" int mb200_ssd_static_status(const mb200_ssd_args *args, int *status)
{
    using namespace mb200;
    if (!args || !status) return fail(MB200_ERR_BAD_ARG, "ssd_static_status: NULL argument");
    if (int rc = check_ssd(*args)) return rc;
    const SsdScratch lay = ssd_scratch_layout(*args);
    if (lay.total > MB200_SSD_STATIC_SCRATCH_BYTES) return fail(MB200_ERR_BAD_ARG, "ssd_static_status: this problem does not fit the built-in buffer");
    if (int rc = enter_device(args->device)) return rc;
    // synchronises with the device: a diagnostic, not part of the hot path
    const cudaError_t e = cudaMemcpyFromSymbol(status, g_ssd_static_scratch, sizeof(int), lay.off_status);
    if (e != cudaSuccess) return fail(MB200_ERR_LAUNCH, "ssd_static_status: %s", cudaGetErrorString(e));
    return MB200_OK;
}

extern "C" int mb200_ssd_fold_state(const float *s_in, const float *range_decay, const float *s_local, float *s_out,
                                    int64_t rows, int64_t row, int32_t device, void *stream)
{
    using namespace mb200;
    MB200_CHECK_ARG(range_decay && s_local && s_out && rows >= 0 && row > 0, "ssd_fold_state: bad argument");
    if (rows == 0) return MB200_OK;
    if (int rc = enter_device(device)) return rc;
    const int64_t total = rows * row;
    const int blocks = (int)((total + 255) / 256 < 148 * 8 ? (total + 255) / 256 : 148 * 8);
    ssd_fold_kernel<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(s_in, range_decay, s_local, s_out, rows, row);
    MB200_CHECK_LAUNCH("ssd_fold_state");
    return MB200_OK;
}

extern "C" int mb200_ssd_fold_ranges(const float *summaries, int64_t record_stride, int32_t first, int32_t last, float *s_out,
                                     int64_t rows, int64_t row, int32_t device, void *stream)
{
    using namespace mb200;
    MB200_CHECK_ARG(summaries && s_out && rows >= 0 && row > 0 && first >= 0 && last >= first && record_stride >= rows * row + rows,
                    "ssd_fold_ranges: bad argument");
    if (rows == 0) return MB200_OK;
    if (int rc = enter_device(device)) return rc;
    const int64_t total = rows * row;
    const int blocks = (int)std::min<int64_t>((total + 255) / 256, 148 * 8);
    ssd_fold_ranges_kernel<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(summaries, record_stride, first, last, s_out, rows, row);
    MB200_CHECK_LAUNCH("ssd_fold_ranges");
    return MB200_OK;
}
