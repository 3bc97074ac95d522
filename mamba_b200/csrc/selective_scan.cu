// Mamba-1 selective scan forward for sm_100a.
//
// Work split: a CTA owns kWarps*cpw consecutive channels of one (batch, group) and walks the
// sequence in tiles of kTile = 32 lanes x kItems steps.  For every tile the B and C rows of the
// group (dstate x kTile, shared by all channels of the CTA) are staged once in shared memory as
// fp32 in a packet-swizzled layout; a warp then takes one channel at a time: each lane loads its
// kItems consecutive steps of u, delta (16-byte packets), and for each state n
//   1. forms a_i = 2^(dt_i A_n log2e), b_i = dt_i u_i B_{n,i}                (registers)
//   2. folds them sequentially into the lane aggregate (prod a, h_local)      (prod a = 2^(A sum dt))
//   3. runs a 5-step shuffle scan over the lanes with (a1,b1)o(a0,b0) = (a1 a0, a1 b0 + b1)
//   4. re-runs the recurrence from the true incoming state and accumulates y_i += C_{n,i} h_i
// The state carried between tiles lives in shared memory (one float per channel and state), so any
// dstate <= 256 works; states are processed in blocks of kStateBlock with B/C re-staged per block.
// Steps past seqlen get dt = 0, u = 0, i.e. the identity (1, 0), so the final state is exact.
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "tc_sm100.cuh"
#include "tensor_map.cuh"

namespace mb200 {
namespace {

constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;
constexpr int kItems = 16;
constexpr int kTile = 32 * kItems;        // 512 steps
constexpr int kStateBlock = 16;
constexpr int kPackets = kTile / 4;       // float4 packets per staged row

// Packet q of a staged row is stored at q ^ ((q >> 2) & 7): the four packets a lane reads back to
// back (4*lane + j) then fall in distinct bank groups across each quarter warp.
__device__ __forceinline__ int swz(int q) { return q ^ ((q >> 2) & 7); }

template <typename T>
__device__ __forceinline__ void load_items(const T *row, int t0, int L, bool vec_ok, float (&v)[kItems])
{
    constexpr int VEC = 16 / sizeof(T);
    if (vec_ok && t0 + kItems <= L) {
#pragma unroll
        for (int k = 0; k < kItems / VEC; ++k) {
            Vec16<T> p;
            p.load(row + t0 + k * VEC);
            float f[VEC];
            p.unpack(f);
#pragma unroll
            for (int i = 0; i < VEC; ++i) v[k * VEC + i] = f[i];
        }
    } else {
#pragma unroll
        for (int i = 0; i < kItems; ++i) v[i] = (t0 + i < L) ? to_float(row[t0 + i]) : 0.f;
    }
}

template <typename T>
__device__ __forceinline__ void store_items(T *row, int t0, int L, bool vec_ok, const float (&v)[kItems])
{
    constexpr int VEC = 16 / sizeof(T);
    if (vec_ok && t0 + kItems <= L) {
#pragma unroll
        for (int k = 0; k < kItems / VEC; ++k) {
            float f[VEC];
#pragma unroll
            for (int i = 0; i < VEC; ++i) f[i] = v[k * VEC + i];
            Vec16<T> p;
            p.pack(f);
            p.store(row + t0 + k * VEC);
        }
    } else {
#pragma unroll
        for (int i = 0; i < kItems; ++i)
            if (t0 + i < L) row[t0 + i] = from_float<T>(v[i]);
    }
}

// Four steps of a row, zeros past the end; off their alignment, or at the end, out of the aligned granules that hold them.
template <typename T>
__device__ __forceinline__ float4 load_quarter(const T *row, int t, int L, bool vec_ok)
{
    constexpr int GW = sizeof(T);                        // words of a granule: as large as four elements
    if (t >= L) return make_float4(0.f, 0.f, 0.f, 0.f);
    uint32_t g[2 * GW], w[GW];
    const uint8_t *first = reinterpret_cast<const uint8_t *>(row + t), *end = reinterpret_cast<const uint8_t *>(row + L);
    const int shift = vec_ok ? 0 : (int)(reinterpret_cast<uintptr_t>(first) & (GW * 4 - 1));
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const uint8_t *p = first - shift + c * GW * 4;
        const bool in = c == 0 || (shift != 0 && p < end);
        if constexpr (GW == 2) {
            const uint2 v = in ? *reinterpret_cast<const uint2 *>(p) : make_uint2(0, 0);
            g[2 * c] = v.x; g[2 * c + 1] = v.y;
        } else {
            const uint4 v = in ? *reinterpret_cast<const uint4 *>(p) : make_uint4(0, 0, 0, 0);
            g[4 * c] = v.x; g[4 * c + 1] = v.y; g[4 * c + 2] = v.z; g[4 * c + 3] = v.w;
        }
    }
    shift_words<T, GW, GW>(g, shift, w);
    const T *e = reinterpret_cast<const T *>(w);
    return make_float4(to_float(e[0]), t + 1 < L ? to_float(e[1]) : 0.f, t + 2 < L ? to_float(e[2]) : 0.f, t + 3 < L ? to_float(e[3]) : 0.f);
}

// Stage rows [n0, n0+kStateBlock) x steps [tile0, tile0+kTile) of a variable B or C as fp32.
template <typename T>
__device__ __forceinline__ void stage_rows(float *dst, const T *src, int64_t n_stride, int n0, int N, int tile0, int L,
                                           bool vec_ok, int threads = kThreads)
{
#pragma unroll 4
    for (int idx = threadIdx.x; idx < kStateBlock * kPackets; idx += threads) {
        const int n = idx / kPackets, q = idx % kPackets;
        const float4 v = n0 + n < N ? load_quarter(src + (int64_t)(n0 + n) * n_stride, tile0 + q * 4, L, vec_ok) : make_float4(0.f, 0.f, 0.f, 0.f);
        reinterpret_cast<float4 *>(dst)[n * kPackets + swz(q)] = v;
    }
}

// Pulls the 16-byte packets a lane will need for steps [t0, t0+kItems) of `row` into L1 ahead of use.
template <typename T>
__device__ __forceinline__ void prefetch_items(const T *row, int t0, int L)
{
    if (t0 < L) {
        const char *p = reinterpret_cast<const char *>(row + t0);
#pragma unroll
        for (int o = 0; o < (int)(kItems * sizeof(T)); o += 32) asm volatile("prefetch.global.L1 [%0];" ::"l"(p + o));
    }
}

__device__ __forceinline__ void read_items(const float *rowbase, int lane, float (&v)[kItems])
{
    const float4 *r = reinterpret_cast<const float4 *>(rowbase);
#pragma unroll
    for (int j = 0; j < kItems / 4; ++j) {
        const float4 p = r[swz(lane * (kItems / 4) + j)];
        v[4 * j + 0] = p.x; v[4 * j + 1] = p.y; v[4 * j + 2] = p.z; v[4 * j + 3] = p.w;
    }
}

template <typename T>
__global__ void __launch_bounds__(kThreads)
scan_fwd_kernel(const mb200_scan_args a, const int cpw, const int nblocks, const int npad, const int vec_flags)
{
    extern __shared__ __align__(16) float smem[];
    float *Bs = smem;                                // kStateBlock x kTile
    float *Cs = Bs + kStateBlock * kTile;            // kStateBlock x kTile
    float *A2s = Cs + kStateBlock * kTile;           // channels x npad : A log2e
    float *run = A2s + kWarps * cpw * npad;          // channels x npad : state entering the tile

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int b = blockIdx.y;
    const int N = a.dstate, L = a.seqlen;
    const int per_group = a.dim / a.ngroups;
    const int chans = kWarps * cpw;
    const int tiles_per_group = (per_group + chans - 1) / chans;
    const int g = blockIdx.x / tiles_per_group;
    const int d_first = g * per_group + (blockIdx.x % tiles_per_group) * chans;
    const int d_end = (g + 1) * per_group;
    const bool io_vec = vec_flags & 1, bc_vec = vec_flags & 2;

    for (int i = threadIdx.x; i < chans * npad; i += kThreads) {
        const int cl = i / npad, n = i % npad;
        const int d = d_first + cl;
        A2s[i] = (d < d_end && n < N) ? a.A[(int64_t)d * a.A_stride[0] + (int64_t)n * a.A_stride[1]] * kLog2e : 0.f;
        run[i] = 0.f;
    }

    const T *Bg = a.B_variable ? static_cast<const T *>(a.B) + (int64_t)b * a.B_stride[0] + (int64_t)g * a.B_stride[1] : nullptr;
    const T *Cg = a.C_variable ? static_cast<const T *>(a.C) + (int64_t)b * a.C_stride[0] + (int64_t)g * a.C_stride[1] : nullptr;

    const int ntiles = (L + kTile - 1) / kTile;
    for (int tile = 0; tile < ntiles; ++tile) {
        const int tile0 = tile * kTile;
        const int t0 = tile0 + lane * kItems;
        for (int c = 0; c < cpw; ++c) {
            const int cl = warp * cpw + c;
            const int d = d_first + cl;
            const bool live = d < d_end;
            float dl[kItems], du[kItems], y[kItems];
            float sum_dt = 0.f;
            if (live) {
                const T *urow = static_cast<const T *>(a.u) + (int64_t)b * a.u_stride[0] + (int64_t)d * a.u_stride[1];
                const T *drow = static_cast<const T *>(a.delta) + (int64_t)b * a.delta_stride[0] + (int64_t)d * a.delta_stride[1];
                float uu[kItems];
                load_items(urow, t0, L, io_vec, uu);
                load_items(drow, t0, L, io_vec, dl);
                const float bias = a.delta_bias ? a.delta_bias[d] : 0.f;
                const float Dd = a.D ? a.D[d] : 0.f;
#pragma unroll
                for (int i = 0; i < kItems; ++i) {
                    float v = dl[i] + bias;
                    if (a.delta_softplus) v = fast_softplus20(v);
                    if (t0 + i >= L) v = 0.f;
                    dl[i] = v;
                    sum_dt += v;
                    du[i] = v * uu[i];
                    y[i] = Dd * uu[i];
                }
                // while this channel's states are scanned, fetch what comes next: its own z row and
                // the u / delta rows of the warp's next (channel, tile)
                if (a.z) prefetch_items(static_cast<const T *>(a.z) + (int64_t)b * a.z_stride[0] + (int64_t)d * a.z_stride[1], t0, L);
                const int dn = (c + 1 < cpw) ? d + 1 : d_first + warp * cpw;
                const int tn = (c + 1 < cpw) ? t0 : t0 + kTile;
                if (dn < d_end) {
                    prefetch_items(static_cast<const T *>(a.u) + (int64_t)b * a.u_stride[0] + (int64_t)dn * a.u_stride[1], tn, L);
                    prefetch_items(static_cast<const T *>(a.delta) + (int64_t)b * a.delta_stride[0] + (int64_t)dn * a.delta_stride[1], tn, L);
                }
            }
            for (int nb = 0; nb < nblocks; ++nb) {
                const int n0 = nb * kStateBlock;
                if (c == 0 || nblocks > 1) {
                    __syncthreads();   // the previous contents of Bs/Cs are no longer being read
                    if (a.B_variable) stage_rows(Bs, Bg, a.B_stride[2], n0, N, tile0, L, bc_vec);
                    if (a.C_variable) stage_rows(Cs, Cg, a.C_stride[2], n0, N, tile0, L, bc_vec);
                    __syncthreads();
                }
                if (!live) continue;
                const int ns = min(kStateBlock, N - n0);
                for (int s = 0; s < ns; ++s) {
                    const int n = n0 + s;
                    const float A2 = A2s[cl * npad + n];
                    float av[kItems], bv[kItems], tmp[kItems];
                    if (a.B_variable) {
                        read_items(Bs + s * kTile, lane, tmp);
                    } else {
                        const float Bc = static_cast<const float *>(a.B)[(int64_t)d * a.B_stride[0] + (int64_t)n * a.B_stride[1]];
#pragma unroll
                        for (int i = 0; i < kItems; ++i) tmp[i] = Bc;
                    }
                    float h = 0.f;
#pragma unroll
                    for (int i = 0; i < kItems; ++i) {
                        av[i] = ex2(dl[i] * A2);
                        bv[i] = du[i] * tmp[i];
                        h = fmaf(av[i], h, bv[i]);
                    }
                    // lane aggregate, then inclusive scan over lanes
                    float P = ex2(sum_dt * A2), H = h;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const float Pp = __shfl_up_sync(0xffffffffu, P, o);
                        const float Hp = __shfl_up_sync(0xffffffffu, H, o);
                        if (lane >= o) {
                            H = fmaf(P, Hp, H);
                            P *= Pp;
                        }
                    }
                    float Pe = __shfl_up_sync(0xffffffffu, P, 1);
                    float He = __shfl_up_sync(0xffffffffu, H, 1);
                    if (lane == 0) { Pe = 1.f; He = 0.f; }
                    const float h_run = run[cl * npad + n];
                    h = fmaf(Pe, h_run, He);                   // state entering this lane's steps
                    if (a.C_variable) {
                        read_items(Cs + s * kTile, lane, tmp);
                    } else {
                        const float Cc = static_cast<const float *>(a.C)[(int64_t)d * a.C_stride[0] + (int64_t)n * a.C_stride[1]];
#pragma unroll
                        for (int i = 0; i < kItems; ++i) tmp[i] = Cc;
                    }
#pragma unroll
                    for (int i = 0; i < kItems; ++i) {
                        h = fmaf(av[i], h, bv[i]);
                        y[i] = fmaf(h, tmp[i], y[i]);
                    }
                    if (lane == 31) run[cl * npad + n] = h;    // read back only by this warp, next tile
                }
                __syncwarp();
            }
            if (live) {
                T *orow = static_cast<T *>(a.out) + (int64_t)b * a.out_stride[0] + (int64_t)d * a.out_stride[1];
                if (a.z) {
                    if (a.out_pregate) {
                        T *prow = static_cast<T *>(a.out_pregate) + (int64_t)b * a.pregate_stride[0] + (int64_t)d * a.pregate_stride[1];
                        store_items(prow, t0, L, io_vec, y);
                    }
                    const T *zrow = static_cast<const T *>(a.z) + (int64_t)b * a.z_stride[0] + (int64_t)d * a.z_stride[1];
                    float zz[kItems];
                    load_items(zrow, t0, L, io_vec, zz);
#pragma unroll
                    for (int i = 0; i < kItems; ++i) y[i] *= fast_silu(zz[i]);
                }
                store_items(orow, t0, L, io_vec, y);
            }
        }
    }
    if (a.last_state) {
        __syncwarp();
        for (int c = 0; c < cpw; ++c) {
            const int cl = warp * cpw + c;
            const int d = d_first + cl;
            if (d >= d_end) continue;
            for (int n = lane; n < N; n += 32)
                a.last_state[((int64_t)b * a.dim + d) * N + n] = run[cl * npad + n];
        }
    }
}

// ------------------------------------------------------------------------------------------------
// The same for few channels with at most 16 states and input-dependent B and C: FOUR warps share a channel, four states each, so
// that 512 channels are 2048 warps and not 512 -- what such a call takes is one warp's chain of loads, exponentials and lane scans,
// not throughput.  A warp prepares a quarter of the steps (softplus) and finishes a quarter of the outputs, with shared memory in
// between; its four states go two at a time, so that one's shuffles hide behind the other's.
// 2 x 256 fp32 channels of 512 steps: 10.2 us, against 14.5 with one warp per channel.
// CH channels per CTA: four, which share the staged B and C, unless that would leave SMs without a CTA.
template <int CH> struct FewSmem {
    float B[kStateBlock * kTile], C[kStateBlock * kTile];
    float dl[CH][kTile], du[CH][kTile];
    float y[CH][4][kTile];
};

template <typename T, int CH>
__global__ void __launch_bounds__(CH * 128) scan_few_kernel(const mb200_scan_args a, const int vec_flags)
{
    pdl_wait();
    pdl_trigger();
    extern __shared__ __align__(16) uint8_t few_raw[];
    FewSmem<CH> &sm = *reinterpret_cast<FewSmem<CH> *>(few_raw);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, cl = warp >> 2, q = warp & 3;
    const int b = blockIdx.y, N = a.dstate, L = a.seqlen, per_group = a.dim / a.ngroups;
    const int tiles_per_group = (per_group + CH - 1) / CH;
    const int g = blockIdx.x / tiles_per_group, d_first = g * per_group + (blockIdx.x % tiles_per_group) * CH;
    const bool live = d_first + cl < (g + 1) * per_group;
    const int d = live ? d_first + cl : d_first;        // warps without a channel shadow one and store nothing
    const bool io_vec = vec_flags & 1, bc_vec = vec_flags & 2;
    auto row_of = [&](const void *p, const int64_t *s) { return const_cast<T *>(static_cast<const T *>(p)) + (int64_t)b * s[0] + (int64_t)d * s[1]; };
    const T *urow = row_of(a.u, a.u_stride), *drow = row_of(a.delta, a.delta_stride), *zrow = a.z ? row_of(a.z, a.z_stride) : nullptr;
    T *orow = row_of(a.out, a.out_stride), *prow = a.z && a.out_pregate ? row_of(a.out_pregate, a.pregate_stride) : nullptr;
    const T *Bg = static_cast<const T *>(a.B) + (int64_t)b * a.B_stride[0] + (int64_t)g * a.B_stride[1];
    const T *Cg = static_cast<const T *>(a.C) + (int64_t)b * a.C_stride[0] + (int64_t)g * a.C_stride[1];
    const float bias = a.delta_bias ? a.delta_bias[d] : 0.f, Dd = a.D ? a.D[d] : 0.f;
    float A2[4], run[4] = {0.f, 0.f, 0.f, 0.f};          // my states: A log2e, value entering the tile
#pragma unroll
    for (int s = 0; s < 4; ++s) A2[s] = 4 * q + s < N ? a.A[(int64_t)d * a.A_stride[0] + (int64_t)(4 * q + s) * a.A_stride[1]] * kLog2e : 0.f;

    for (int tile0 = 0; tile0 < L; tile0 += kTile) {
        const int t = tile0 + lane * kItems + 4 * q, slot = swz(lane * 4 + q);
        const float4 u4 = load_quarter(urow, t, L, io_vec), d4 = load_quarter(drow, t, L, io_vec);
        const float4 z4 = zrow ? load_quarter(zrow, t, L, io_vec) : make_float4(0.f, 0.f, 0.f, 0.f);
        stage_rows(sm.B, Bg, a.B_stride[2], 0, N, tile0, L, bc_vec, CH * 128);
        stage_rows(sm.C, Cg, a.C_stride[2], 0, N, tile0, L, bc_vec, CH * 128);
        const float uu[4] = {u4.x, u4.y, u4.z, u4.w};
        float dl4[4] = {d4.x, d4.y, d4.z, d4.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float v = dl4[i] + bias;
            if (a.delta_softplus) v = fast_softplus20(v);
            dl4[i] = t + i < L ? v : 0.f;
        }
        reinterpret_cast<float4 *>(sm.dl[cl])[slot] = make_float4(dl4[0], dl4[1], dl4[2], dl4[3]);
        reinterpret_cast<float4 *>(sm.du[cl])[slot] = make_float4(dl4[0] * uu[0], dl4[1] * uu[1], dl4[2] * uu[2], dl4[3] * uu[3]);
        __syncthreads();
        float dl[kItems], du[kItems], y[kItems], sum_dt = 0.f;
        read_items(sm.dl[cl], lane, dl);
        read_items(sm.du[cl], lane, du);
#pragma unroll
        for (int i = 0; i < kItems; ++i) {
            y[i] = 0.f;
            sum_dt += dl[i];
        }
#pragma unroll
        for (int s0 = 0; s0 < 4; s0 += 2) {
            if (4 * q + s0 >= N) break;
            float av[2][kItems], bv[2][kItems], P[2], H[2], h[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                read_items(sm.B + (4 * q + s0 + e) * kTile, lane, bv[e]);
                h[e] = 0.f;
#pragma unroll
                for (int i = 0; i < kItems; ++i) {
                    av[e][i] = ex2(dl[i] * A2[s0 + e]);
                    bv[e][i] *= du[i];
                    h[e] = fmaf(av[e][i], h[e], bv[e][i]);
                }
                P[e] = ex2(sum_dt * A2[s0 + e]);         // aggregate of my steps, then an inclusive scan over the lanes
                H[e] = h[e];
            }
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const float Pp = __shfl_up_sync(0xffffffffu, P[e], o), Hp = __shfl_up_sync(0xffffffffu, H[e], o);
                    if (lane >= o) {
                        H[e] = fmaf(P[e], Hp, H[e]);
                        P[e] *= Pp;
                    }
                }
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                float Pe = __shfl_up_sync(0xffffffffu, P[e], 1), He = __shfl_up_sync(0xffffffffu, H[e], 1);
                if (lane == 0) { Pe = 1.f; He = 0.f; }
                h[e] = fmaf(Pe, run[s0 + e], He);        // state entering my steps
                float cv[kItems];
                read_items(sm.C + (4 * q + s0 + e) * kTile, lane, cv);
#pragma unroll
                for (int i = 0; i < kItems; ++i) {
                    h[e] = fmaf(av[e][i], h[e], bv[e][i]);
                    y[i] = fmaf(h[e], cv[i], y[i]);
                }
                run[s0 + e] = __shfl_sync(0xffffffffu, h[e], 31);
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) reinterpret_cast<float4 *>(sm.y[cl][q])[swz(lane * 4 + j)] = make_float4(y[4 * j], y[4 * j + 1], y[4 * j + 2], y[4 * j + 3]);
        __syncthreads();
        float o[4] = {Dd * uu[0], Dd * uu[1], Dd * uu[2], Dd * uu[3]};
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            const float4 v = reinterpret_cast<const float4 *>(sm.y[cl][w])[slot];
            o[0] += v.x; o[1] += v.y; o[2] += v.z; o[3] += v.w;
        }
        auto put = [&](T *row) {
            if (io_vec && t + 4 <= L) {
                if constexpr (sizeof(T) == 4) {
                    *reinterpret_cast<float4 *>(row + t) = make_float4(o[0], o[1], o[2], o[3]);
                } else {
                    uint2 w;
                    T *e = reinterpret_cast<T *>(&w);
#pragma unroll
                    for (int i = 0; i < 4; ++i) e[i] = from_float<T>(o[i]);
                    *reinterpret_cast<uint2 *>(row + t) = w;
                }
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (t + i < L) row[t + i] = from_float<T>(o[i]);
            }
        };
        if (live && prow) put(prow);
        if (zrow) {
            o[0] *= fast_silu(z4.x); o[1] *= fast_silu(z4.y); o[2] *= fast_silu(z4.z); o[3] *= fast_silu(z4.w);
        }
        if (live) put(orow);
    }
    if (a.last_state && live && lane == 0) {
#pragma unroll
        for (int s = 0; s < 4; ++s)
            if (4 * q + s < N) a.last_state[((int64_t)b * a.dim + d) * N + 4 * q + s] = run[s];
    }
}

template <typename T>
__device__ __forceinline__ float words_get(const uint32_t *w, int i)
{
    if constexpr (sizeof(T) == 4) {
        return __uint_as_float(w[i]);
    } else if constexpr (std::is_same<T, __nv_bfloat16>::value) {
        const uint32_t x = w[i >> 1];
        return __uint_as_float((i & 1) ? (x & 0xffff0000u) : (x << 16));
    } else {
        const uint32_t x = w[i >> 1];
        return __half2float(__ushort_as_half((unsigned short)((i & 1) ? (x >> 16) : (x & 0xffffu))));
    }
}

template <int HS>
__device__ __forceinline__ void lds_pairs(const float *p, uint64_t (&v)[HS / 2])
{
    if constexpr (HS % 4 == 0) {
#pragma unroll
        for (int q = 0; q < HS / 4; ++q) {
            const ulonglong2 r = reinterpret_cast<const ulonglong2 *>(p)[q];
            v[2 * q] = r.x;
            v[2 * q + 1] = r.y;
        }
    } else {
#pragma unroll
        for (int j = 0; j < HS / 2; ++j) v[j] = reinterpret_cast<const uint64_t *>(p)[j];
    }
}

// ------------------------------------------------------------------------------------------------
// Channel-parallel scan, warp-specialised (dstate <= 16, input-dependent B and C): time is sequential.
// The lanes of a warp are 32 different CHANNELS, so B_t and C_t are read
// from shared memory at one address per warp (a single wavefront per 128-bit load), and nothing in
// the recurrence loop crosses lanes.  A CTA of three warps owns 32 channels of one batch row:
//   warp 0   ("scalar" warp) streams the u, dt, z rows and the group's B/C rows as TMA tiles
//            (32 bytes of every row per tile, SWIZZLE_32B so that each lane reads its own row without
//            bank conflicts), evaluates softplus(dt) and hands (dt, u) for 8 steps at a time to the
//            state warps through shared memory (dt and dt*u) together with the B/C values converted to
//            fp32; later it adds the two partial outputs and D*u, applies silu(z) and sends the output
//            tile back with a TMA store;
//   warps 1,2 ("state" warps) each keep half of the states of the 32 channels in registers and run
//            the recurrence: per (step, state) one MUFU ex2 and four FMA-pipe operations, no shuffles.
// Hand-offs are mbarriers: ready[2] (scalar -> state, 8 steps of dt/u/B/C in place) and ydone[2]
// (state -> scalar, 8 steps of partial outputs in place), all buffers double.  The scalar warp runs
// one hand-off ahead, and the TMA tiles two tiles ahead, of the recurrence.  Every wait is bounded;
// on expiry the kernel records a code in g_scan_status, stops, and drains its outstanding copies.
//
// Rows that TMA cannot describe (an odd number of steps, a slice at an odd offset, a group that is no multiple of 32
// channels, two outputs) are read and written by the scalar warps' lanes themselves (TMA = false): a lane streams its
// channel's rows as ALIGNED 16-byte granules, copied a few hand-offs ahead with cp.async into a ring of its own, takes the
// 8 steps of a hand-off out of two neighbouring granules with a shift that is fixed for the row, and on the way out carries
// the end of one hand-off into the granule that the next completes.  Nothing is read element by element, only the two ends
// of an output row are written so.  8 x 5120 rows of 2047 bf16 steps: 675 us (aligned rows of 2048: 530); 5120 rows of
// 1999: 160 us, against 275 in the time-parallel kernel with element loads.
__device__ int g_scan_status;
enum { kStScanFull = 31, kStScanZ, kStScanReady, kStScanYdone, kStScanAlign };

constexpr int kStreamCh = 32;      // channels per CTA (lanes of a warp)
constexpr int64_t kStreamMinChannels = 1024;   // fewer (batch x dim) channels than this go to the time-parallel kernel
constexpr int kHB = 8;             // steps per hand-off

struct ScanMaps { CUtensorMap u, dt, z, out, B, C; };

// Sequence split inside one launch: CTA (group of channels, batch row, segment) walks steps [s * seg_len, (s+1) * seg_len)
// from the state h0[b][s] (zero when h0 is NULL).  A SUMMARY launch computes, for every segment but the last, the state
// at its end from a zero start (hend) and the product of its decays (pdec); after a fold over the segments a second,
// full launch runs every segment from its true entering state.  nseg = 1 is the plain one-pass scan.
struct ScanSplit {
    int nseg, seg_len;
    const float *h0;        // (batch, nseg, dim, dstate) or NULL
    float *hend, *pdec;     // (batch, nseg, dim, dstate), SUMMARY launches only
};

// What the inputs land in: two TMA tiles of each tensor, or R hand-offs of every lane's granules ([hand-off][granule][lane]).
// R: as many hand-offs as leave room for the CTAs per SM that each layout is made for.
template <typename T, int NS, int SW, bool SPLIT, bool TMA> struct StreamTiles {
    uint8_t u[2][kStreamCh * 32];
    uint8_t dt[2][kStreamCh * 32];
    uint8_t z[2][kStreamCh * 32];
    uint8_t out[2][kStreamCh * 32];
    uint8_t B[2][(NS * 32 + 255) / 256 * 256];
    uint8_t C[2][(NS * 32 + 255) / 256 * 256];
};
template <typename T, int NS, int SW, bool SPLIT> struct StreamTiles<T, NS, SW, SPLIT, false> {
    static constexpr int R = sizeof(T) == 4 ? 3 : !SPLIT ? 4 : SW == 2 ? 6 : 7;
    static constexpr int kUnit = kStreamCh * kHB * sizeof(T);
    uint8_t u[R * kUnit], dt[R * kUnit], bc[R * kUnit], z[R * kUnit];
};

template <typename T, int NS, int SW, bool SPLIT, bool TMA>
struct __align__(256) StreamSmem {
    // hand-off buffers: with one scalar warp two are all it can use (it prepares hand-off hb+1, then finishes hb); with
    // the work on two warps, four let the three stages of the chain run at the pace of the slowest, not of their sum
    static constexpr int NB = SPLIT ? 4 : 2;
    StreamTiles<T, NS, SW, SPLIT, TMA> t;
    // per-channel rows of 8 steps (32 bytes) in the same chunk-swizzled layout as the tiles: a lane moves four
    // steps with one conflict-free 128-bit access
    float xd[NB][2][kStreamCh * kHB];        // [buffer][dt | dt*u][channel][step]
    float du[NB][kStreamCh * kHB];           // [buffer][channel][step]: D*u, kept by the scalar warp for its epilogue
    float bc[NB][2][kHB * NS + 16];          // [buffer][B | C][step][state]; the pad puts B and C on different banks
    float yp[NB][SW][kStreamCh * kHB];       // [buffer][state warp][channel][step]
    uint64_t full[2], zfull[2], ready[NB], ydone[NB], edone[NB];
};

__device__ __forceinline__ void cp_async16(void *dst, const void *src, bool on)      // zeros when off
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(tc::smem_u32(dst)), "l"(src), "r"(on ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory"); }

// A row as its aligned granules: `bytes` is where the valid part ends, counted from the first granule.
struct GranuleRow {
    const uint8_t *p;
    int shift, bytes;
};
template <typename T> __device__ __forceinline__ GranuleRow granule_row(const T *first, int L)
{
    const int shift = (int)(reinterpret_cast<uintptr_t>(first) & 15);
    return {reinterpret_cast<const uint8_t *>(first) - shift, shift, shift + L * (int)sizeof(T)};
}

// Output side of the same: every hand-off completes granules with what the one before left over.
template <typename T, int NW> struct GranuleOut {
    uint8_t *row;
    int lag, bytes;             // bytes of a hand-off that wait for the next one (1..16); bytes of the row
    uint32_t prev[4];
    __device__ __forceinline__ void init(T *first, int L)
    {
        const int s = (int)(reinterpret_cast<uintptr_t>(first) & 15);
        row = reinterpret_cast<uint8_t *>(first);
        lag = s ? s : 16;       // a granule ends `lag` bytes before the hand-off does
        bytes = L * (int)sizeof(T);
#pragma unroll
        for (int i = 0; i < 4; ++i) prev[i] = 0u;
    }
    __device__ __forceinline__ void put(int pos, uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3)
    {
        if (pos >= 0 && pos + 16 <= bytes) {
            *reinterpret_cast<uint4 *>(row + pos) = make_uint4(w0, w1, w2, w3);
        } else if (pos < bytes) {      // the ends of the row
            const uint32_t w[4] = {w0, w1, w2, w3};
#pragma unroll
            for (int i = 0; i < 16 / (int)sizeof(T); ++i) {
                const int o = pos + i * (int)sizeof(T);
                if (o < 0 || o >= bytes) continue;
                if constexpr (sizeof(T) == 2) *reinterpret_cast<uint16_t *>(row + o) = (uint16_t)(w[i >> 1] >> (16 * (i & 1)));
                else *reinterpret_cast<uint32_t *>(row + o) = w[i];
            }
        }
    }
    __device__ __forceinline__ void emit(int hb, const uint32_t (&cur)[NW], bool last)
    {
        uint32_t all[NW + 4], o[NW];
#pragma unroll
        for (int i = 0; i < NW + 4; ++i) all[i] = i < 4 ? prev[i] : cur[i - 4];
        shift_words<T, NW>(all, 16 - lag, o);
#pragma unroll
        for (int c = 0; c < NW / 4; ++c) put((hb * (NW / 4) + c) * 16 - lag, o[4 * c], o[4 * c + 1], o[4 * c + 2], o[4 * c + 3]);
#pragma unroll
        for (int i = 0; i < 4; ++i) prev[i] = cur[NW - 4 + i];
        if (last) {
            uint32_t end[8], e[4];
#pragma unroll
            for (int i = 0; i < 8; ++i) end[i] = i < 4 ? prev[i] : 0u;
            shift_words<T, 4>(end, 16 - lag, e);
            put((hb + 1) * (NW / 4) * 16 - lag, e[0], e[1], e[2], e[3]);
        }
    }
};

// byte offset of 16-byte chunk `chunk` of row `row` in a [rows x 32 B] SWIZZLE_32B tile (256-byte aligned)
__device__ __forceinline__ int sw32_offset(int row, int chunk) { return row * 32 + ((chunk ^ ((row >> 2) & 1)) << 4); }

// SW state warps share the states of the 32 channels; SPLIT gives the scalar work to two warps (warp 0 streams the
// tiles in and prepares the hand-offs, warp 1 finishes the outputs and streams them out) instead of one.  (2, false) is
// the layout described above: three warps, nine CTAs per SM, the choice whenever the grid fills the GPU.  The other two
// are for grids that leave the SMs partly empty (a batch divided over several GPUs), where a CTA's own serial chain per
// hand-off matters more than the number of CTAs an SM can hold: (2, true), four warps and six CTAs per SM, for up to
// 888 CTAs; (4, true), six warps (four states per lane) and four CTAs per SM, for up to 592.
template <typename T, int NS, bool SUMMARY, int SW, bool SPLIT, bool TMA>
__global__ void __launch_bounds__(32 * (SW + (SPLIT ? 2 : 1)), !SPLIT ? 9 : SW == 2 ? 6 : 4)
scan_stream_kernel(const mb200_scan_args a, const __grid_constant__ ScanMaps maps, const ScanSplit sp)
{
    using namespace tc;
    constexpr int TB = 32 / sizeof(T);                 // steps per tile (32 bytes of a row)
    constexpr int HPT = TB / kHB;                      // hand-offs per tile: 2 (16-bit) or 1 (fp32)
    constexpr int CPH = kHB * sizeof(T) / 16;          // 16-byte chunks per hand-off: 1 or 2
    constexpr int HS = NS / SW;                        // states per lane of a state warp
    constexpr int kScalarWarps = SPLIT ? 2 : 1;
    extern __shared__ __align__(256) uint8_t smem_raw[];
    using Smem = StreamSmem<T, NS, SW, SPLIT, TMA>;
    constexpr int NB = Smem::NB;
    Smem &sm = *reinterpret_cast<Smem *>(smem_raw);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int N = a.dstate;
    const int b = blockIdx.y / sp.nseg, seg = blockIdx.y % sp.nseg;
    const int t_begin = seg * sp.seg_len;              // a multiple of the tile length
    const int L = min(a.seqlen, t_begin + sp.seg_len) - t_begin;      // steps of my segment
    const int per_group = a.dim / a.ngroups, group_tiles = (per_group + kStreamCh - 1) / kStreamCh;
    const int g = blockIdx.x / group_tiles, ch0 = g * per_group + (blockIdx.x % group_tiles) * kStreamCh;
    const bool live = TMA || ch0 + lane < (g + 1) * per_group;       // (whole tiles of channels with TMA)
    const int d = live ? ch0 + lane : ch0;             // my channel; a lane without one shadows another and stores nothing
    const int ntiles = (L + TB - 1) / TB, nhb = (L + kHB - 1) / kHB;
    const bool has_z = !SUMMARY && a.z != nullptr;
    if (SUMMARY) pdl_trigger();
    if (SUMMARY && seg == sp.nseg - 1) return;         // the last segment's end state is the full launch's business
    if (L <= 0) return;                                // a segment past the end of a short sequence
    int *status = &g_scan_status;
    if (smem_u32(smem_raw) & 255u) {                   // the swizzle pattern of the tiles assumes this alignment
        if (threadIdx.x == 0) atomicCAS(status, 0, kStScanAlign);
        return;
    }

    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&sm.full[i], 1);
            mbar_init(&sm.zfull[i], 1);
        }
        for (int i = 0; i < NB; ++i) {
            mbar_init(&sm.ready[i], 1);
            mbar_init(&sm.ydone[i], SW);
            mbar_init(&sm.edone[i], 1);
        }
        mbar_fence_init();
    }
    __syncthreads();

    if (warp < kScalarWarps) {
        // ------------------------------------------------------------------ scalar warp(s)
        const bool in_side = warp == 0, out_side = warp == kScalarWarps - 1;
        [[maybe_unused]] constexpr uint32_t kTileBytes = 2 * kStreamCh * 32 + (SUMMARY ? 1 : 2) * NS * 32;      // a summary needs no C
        auto issue_tile = [&](int k) {          // lane 0 only
            if constexpr (TMA) {
                const int s = k & 1;
                mbar_expect_tx(&sm.full[s], kTileBytes);
                tma_load_3d(sm.t.u[s], &maps.u, &sm.full[s], t_begin + k * TB, ch0, b);
                tma_load_3d(sm.t.dt[s], &maps.dt, &sm.full[s], t_begin + k * TB, ch0, b);
                tma_load_4d(sm.t.B[s], &maps.B, &sm.full[s], t_begin + k * TB, 0, g, b);
                if (!SUMMARY) tma_load_4d(sm.t.C[s], &maps.C, &sm.full[s], t_begin + k * TB, 0, g, b);
            }
        };
        auto issue_z = [&](int k) {             // lane 0 only
            if constexpr (TMA) {
                const int s = k & 1;
                mbar_expect_tx(&sm.zfull[s], kStreamCh * 32);
                tma_load_3d(sm.t.z[s], &maps.z, &sm.zfull[s], t_begin + k * TB, ch0, b);
            }
        };
        int issued = 0, zissued = 0, waited = 0, zwaited = 0;     // tiles requested / consumed (uniform across the warp)
        if (TMA && lane == 0) {
            prefetch_tmap(&maps.u); prefetch_tmap(&maps.dt); prefetch_tmap(&maps.B);
            if (!SUMMARY) { prefetch_tmap(&maps.C); prefetch_tmap(&maps.out); }
            if (has_z) prefetch_tmap(&maps.z);
        }
        for (int k = 0; TMA && k < 2 && k < ntiles; ++k) {
            if (lane == 0 && in_side) issue_tile(k);
            if (lane == 0 && out_side && has_z) issue_z(k);
            ++issued; ++zissued;
        }
        const float bias = a.delta_bias ? a.delta_bias[d] : 0.f;
        const float Dd = a.D ? a.D[d] : 0.f;
        const int st_t = lane / NS, st_n = lane % NS;     // my (tensor, state row) in the B/C conversion
        const bool st_on = lane < (SUMMARY ? 1 : 2) * NS;
        bool ok = true;

        // TMA = false: my rows, and my slots of the rings
        [[maybe_unused]] GranuleRow row_u, row_dt, row_bc, row_z;
        [[maybe_unused]] GranuleOut<T, CPH * 4> row_out, row_pre;
        const bool pregate = !TMA && !SUMMARY && a.out_pregate != nullptr;
        if constexpr (!TMA) {
            auto at = [&](const void *p, const int64_t *st) { return static_cast<const T *>(p) + (int64_t)b * st[0] + (int64_t)d * st[1] + t_begin; };
            row_u = granule_row(at(a.u, a.u_stride), L);
            row_dt = granule_row(at(a.delta, a.delta_stride), L);
            const int64_t *bs = st_t == 0 ? a.B_stride : a.C_stride;
            row_bc = granule_row(static_cast<const T *>(st_t == 0 ? a.B : a.C) + (int64_t)b * bs[0] + (int64_t)g * bs[1] + (st_n < N ? st_n : 0) * bs[2] + t_begin, L);
            if (st_n >= N) row_bc.bytes = 0;           // states that pad the block: zeros
            row_z = has_z ? granule_row(at(a.z, a.z_stride), L) : row_u;
            row_out.init(const_cast<T *>(at(a.out, a.out_stride)), live ? L : 0);
            if (pregate) row_pre.init(const_cast<T *>(at(a.out_pregate, a.pregate_stride)), live ? L : 0);
        }
        auto fetch = [&](int hb) {              // the granules that begin in hand-off hb
            if constexpr (!TMA) {
                constexpr int R = decltype(sm.t)::R;
                auto one = [&](uint8_t *ring, const GranuleRow &r) {
#pragma unroll
                    for (int c = 0; c < CPH; ++c) {
                        const int o = (hb * CPH + c) * 16;
                        cp_async16(ring + ((hb % R) * CPH + c) * 512 + lane * 16, r.p + (o < r.bytes ? o : 0), o < r.bytes);
                    }
                };
                if (in_side) {
                    one(sm.t.u, row_u);
                    one(sm.t.dt, row_dt);
                    if (st_on) one(sm.t.bc, row_bc);
                }
                if (out_side && has_z) one(sm.t.z, row_z);
                cp_async_commit();              // one group per hand-off, empty ones included
            }
        };
        auto take = [&](const uint8_t *ring, int shift, int hb, uint32_t (&o)[CPH * 4]) {
            if constexpr (!TMA) {
                constexpr int R = decltype(sm.t)::R;
                uint32_t w[CPH * 4 + 4];
#pragma unroll
                for (int c = 0; c <= CPH; ++c) {
                    const int slot = c < CPH ? (hb % R) * CPH + c : ((hb + 1) % R) * CPH;
                    const uint4 v = *reinterpret_cast<const uint4 *>(ring + slot * 512 + lane * 16);
                    w[4 * c] = v.x; w[4 * c + 1] = v.y; w[4 * c + 2] = v.z; w[4 * c + 3] = v.w;
                }
                shift_words<T, CPH * 4>(w, shift, o);
            }
        };
        if constexpr (!TMA) {
            for (int i = 0; i < decltype(sm.t)::R; ++i) fetch(i);
        }

        auto prologue = [&](int hb) {
            const int k = hb / HPT, s = k & 1, part = hb % HPT, buf = hb % NB;
            if (SPLIT && hb >= NB) {    // the other scalar warp has finished with this buffer's D*u and partial outputs
                if (!mbar_wait(&sm.edone[buf], ((hb - NB) / NB) & 1, status, kStScanYdone)) { ok = false; return; }
            }
            uint32_t wd[CPH * 4], wu[CPH * 4], wb[CPH * 4];
            if constexpr (TMA) {
                if (part == 0) {
                    if (!mbar_wait(&sm.full[s], (k >> 1) & 1, status, kStScanFull)) { ok = false; return; }
                    ++waited;
                }
#pragma unroll
                for (int c = 0; c < CPH; ++c) {
                    const int off = sw32_offset(lane, part * CPH + c);
                    const uint4 rd = *reinterpret_cast<const uint4 *>(sm.t.dt[s] + off);
                    const uint4 ru = *reinterpret_cast<const uint4 *>(sm.t.u[s] + off);
                    wd[4 * c] = rd.x; wd[4 * c + 1] = rd.y; wd[4 * c + 2] = rd.z; wd[4 * c + 3] = rd.w;
                    wu[4 * c] = ru.x; wu[4 * c + 1] = ru.y; wu[4 * c + 2] = ru.z; wu[4 * c + 3] = ru.w;
                }
                if (st_on) {
                    const uint8_t *src = st_t ? sm.t.C[s] : sm.t.B[s];
#pragma unroll
                    for (int c = 0; c < CPH; ++c) {
                        const uint4 r = *reinterpret_cast<const uint4 *>(src + sw32_offset(st_n, part * CPH + c));
                        wb[4 * c] = r.x; wb[4 * c + 1] = r.y; wb[4 * c + 2] = r.z; wb[4 * c + 3] = r.w;
                    }
                }
            } else {
                // hand-offs hb and hb + 1 have landed.  Two scalar warps fetch hb + R after taking hb; one warp does so only after
                // finishing hb, one hand-off later.
                cp_async_wait<decltype(sm.t)::R - (SPLIT ? 2 : 3)>();
                take(sm.t.dt, row_dt.shift, hb, wd);
                take(sm.t.u, row_u.shift, hb, wu);
                if (st_on) take(sm.t.bc, row_bc.shift, hb, wb);
            }
            const int t0 = hb * kHB;
            const bool tail = t0 + kHB > L;             // only the last hand-off can run past the end
            float dl[kHB], dlu[kHB], skip[kHB];
#pragma unroll
            for (int i = 0; i < kHB; ++i) {
                float v = words_get<T>(wd, i) + bias;
                if (a.delta_softplus) v = TMA && sizeof(T) == 2 ? softplus20_lowprec(v) : fast_softplus20(v);
                float uu = words_get<T>(wu, i);
                if (tail && t0 + i >= L) {              // steps past the end are the identity (1, 0)
                    v = 0.f;
                    if (!TMA) uu = 0.f;                 // (a granule goes on with the next row's values, a tile with zeros)
                }
                dl[i] = v;
                dlu[i] = v * uu;
                skip[i] = Dd * uu;
            }
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int off = sw32_offset(lane, c);
                *reinterpret_cast<float4 *>(reinterpret_cast<uint8_t *>(sm.xd[buf][0]) + off) = make_float4(dl[4 * c], dl[4 * c + 1], dl[4 * c + 2], dl[4 * c + 3]);
                *reinterpret_cast<float4 *>(reinterpret_cast<uint8_t *>(sm.xd[buf][1]) + off) = make_float4(dlu[4 * c], dlu[4 * c + 1], dlu[4 * c + 2], dlu[4 * c + 3]);
                *reinterpret_cast<float4 *>(reinterpret_cast<uint8_t *>(sm.du[buf]) + off) = make_float4(skip[4 * c], skip[4 * c + 1], skip[4 * c + 2], skip[4 * c + 3]);
            }
            if (st_on) {
                float *dst = sm.bc[buf][st_t];
#pragma unroll
                for (int i = 0; i < kHB; ++i) dst[i * NS + st_n] = !TMA && tail && t0 + i >= L ? 0.f : words_get<T>(wb, i);
            }
            __syncwarp();
            if (lane == 0) {
                if (TMA && (part == HPT - 1 || hb == nhb - 1) && k + 2 < ntiles) issue_tile(k + 2);
                mbar_arrive(&sm.ready[buf]);
            }
            if constexpr (!TMA && SPLIT) fetch(hb + decltype(sm.t)::R);
            if (TMA && (part == HPT - 1 || hb == nhb - 1) && k + 2 < ntiles) ++issued;
        };

        auto epilogue = [&](int hb) {
            const int k = hb / HPT, s = k & 1, part = hb % HPT, buf = hb % NB;
            if (!mbar_wait(&sm.ydone[buf], (hb / NB) & 1, status, kStScanYdone)) { ok = false; return; }
            if (SUMMARY) {                      // nothing to put out: the wait only hands the buffers back
                if (SPLIT && lane == 0) mbar_arrive(&sm.edone[buf]);
                return;
            }
            if (TMA && part == 0) {
                if (has_z) {
                    if (!mbar_wait(&sm.zfull[s], (k >> 1) & 1, status, kStScanZ)) { ok = false; return; }
                    ++zwaited;
                }
                if (k >= 2) {       // the store that last read this output tile has finished reading it
                    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                    __syncwarp();
                }
            }
            float y[kHB];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int off = sw32_offset(lane, c);
                float4 p0 = *reinterpret_cast<const float4 *>(reinterpret_cast<const uint8_t *>(sm.yp[buf][0]) + off);
                const float4 p1 = *reinterpret_cast<const float4 *>(reinterpret_cast<const uint8_t *>(sm.yp[buf][1]) + off);
                if constexpr (SW == 4) {
                    const float4 p2 = *reinterpret_cast<const float4 *>(reinterpret_cast<const uint8_t *>(sm.yp[buf][2]) + off);
                    const float4 p3 = *reinterpret_cast<const float4 *>(reinterpret_cast<const uint8_t *>(sm.yp[buf][3]) + off);
                    p0 = make_float4(p0.x + p2.x, p0.y + p2.y, p0.z + p2.z, p0.w + p2.w);
                    p0 = make_float4(p0.x + p3.x, p0.y + p3.y, p0.z + p3.z, p0.w + p3.w);
                }
                const float4 sk = *reinterpret_cast<const float4 *>(reinterpret_cast<const uint8_t *>(sm.du[buf]) + off);
                y[4 * c] = (p0.x + p1.x) + sk.x;
                y[4 * c + 1] = (p0.y + p1.y) + sk.y;
                y[4 * c + 2] = (p0.z + p1.z) + sk.z;
                y[4 * c + 3] = (p0.w + p1.w) + sk.w;
            }
            if (SPLIT) {        // D*u and the partial outputs of this buffer are in registers: the other warp may refill it
                __syncwarp();
                if (lane == 0) mbar_arrive(&sm.edone[buf]);
            }
            uint32_t wo[CPH * 4];
            auto pack_out = [&]() {
                T *e = reinterpret_cast<T *>(wo);
#pragma unroll
                for (int i = 0; i < kHB; ++i) e[i] = from_float<T>(y[i]);
            };
            if (pregate) {
                pack_out();
                row_pre.emit(hb, wo, hb == nhb - 1);
            }
            if (has_z) {
                uint32_t wz[CPH * 4];
                if constexpr (TMA) {
#pragma unroll
                    for (int c = 0; c < CPH; ++c) {
                        const uint4 r = *reinterpret_cast<const uint4 *>(sm.t.z[s] + sw32_offset(lane, part * CPH + c));
                        wz[4 * c] = r.x; wz[4 * c + 1] = r.y; wz[4 * c + 2] = r.z; wz[4 * c + 3] = r.w;
                    }
                } else {
                    if constexpr (SPLIT) cp_async_wait<decltype(sm.t)::R - 2>();       // (one scalar warp: the hand-off after this has been waited for)
                    take(sm.t.z, row_z.shift, hb, wz);
                }
#pragma unroll
                for (int i = 0; i < kHB; ++i) {
                    const float zz = words_get<T>(wz, i);
                    if constexpr (TMA && std::is_same<T, __nv_bfloat16>::value) y[i] *= silu_for_bf16(zz);
                    else y[i] *= fast_silu(zz);
                }
            }
            pack_out();
            if constexpr (TMA) {
#pragma unroll
                for (int c = 0; c < CPH; ++c)
                    *reinterpret_cast<uint4 *>(sm.t.out[s] + sw32_offset(lane, part * CPH + c)) =
                        make_uint4(wo[4 * c], wo[4 * c + 1], wo[4 * c + 2], wo[4 * c + 3]);
                if (part == HPT - 1 || hb == nhb - 1) {
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) {
                        asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(&maps.out),
                                     "r"(smem_u32(sm.t.out[s])), "r"(t_begin + k * TB), "r"(ch0), "r"(b)
                                     : "memory");
                        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                        if (has_z && k + 2 < ntiles) issue_z(k + 2);
                    }
                    if (has_z && k + 2 < ntiles) ++zissued;
                }
            } else {
                row_out.emit(hb, wo, hb == nhb - 1);
                if constexpr (SPLIT) fetch(hb + decltype(sm.t)::R);
            }
        };

        if (!SPLIT) {
            prologue(0);
            for (int hb = 0; hb < nhb && ok; ++hb) {
                if (hb + 1 < nhb) prologue(hb + 1);
                if (ok) epilogue(hb);
                if constexpr (!TMA) fetch(hb + decltype(sm.t)::R);
            }
        } else if (in_side) {
            for (int hb = 0; hb < nhb && ok; ++hb) prologue(hb);
        } else {
            for (int hb = 0; hb < nhb && ok; ++hb) epilogue(hb);
        }
        if constexpr (!TMA) cp_async_wait<0>();
        if (TMA && lane == 0) {
            if (out_side) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            if (!ok) {      // stopped early: let the tiles already requested land before the CTA's shared memory goes away
                if (in_side)
                    for (int k = waited; k < issued; ++k) mbar_wait(&sm.full[k & 1], (k >> 1) & 1, status, kStScanFull);
                if (out_side && has_z)
                    for (int k = zwaited; k < zissued; ++k) mbar_wait(&sm.zfull[k & 1], (k >> 1) & 1, status, kStScanZ);
            }
        }
    } else {
        // ------------------------------------------------------------------ state warps
        const int w = warp - kScalarWarps;
        uint64_t A2[HS / 2], h[HS / 2];
#pragma unroll
        for (int j = 0; j < HS / 2; ++j) {
            float av[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int n = w * HS + 2 * j + e;
                av[e] = n < N ? a.A[(int64_t)d * a.A_stride[0] + (int64_t)n * a.A_stride[1]] * kLog2e : 0.f;
            }
            A2[j] = pack2(av[0], av[1]);
            float h0v[2] = {0.f, 0.f};
            if (sp.h0) {     // (the inputs may be on their way before the fold has ended)
                if (j == 0) pdl_wait();
                const float *hp = sp.h0 + (((int64_t)b * sp.nseg + seg) * a.dim + d) * N;
#pragma unroll
                for (int e = 0; e < 2; ++e)
                    if (w * HS + 2 * j + e < N) h0v[e] = hp[w * HS + 2 * j + e];
            }
            h[j] = pack2(h0v[0], h0v[1]);
        }
        float sum_dl = 0.f;          // SUMMARY: the decay product of the segment is 2^(A log2e * sum of dt)
        for (int hb = 0; hb < nhb; ++hb) {
            const int buf = hb % NB;
            if (!mbar_wait(&sm.ready[buf], (hb / NB) & 1, status, kStScanReady)) break;
            const float *Bt = sm.bc[buf][0] + w * HS, *Ct = sm.bc[buf][1] + w * HS;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int off = sw32_offset(lane, c);
                const float4 dlv = *reinterpret_cast<const float4 *>(reinterpret_cast<const uint8_t *>(sm.xd[buf][0]) + off);
                const float4 duv = *reinterpret_cast<const float4 *>(reinterpret_cast<const uint8_t *>(sm.xd[buf][1]) + off);
                const float dls[4] = {dlv.x, dlv.y, dlv.z, dlv.w}, dus[4] = {duv.x, duv.y, duv.z, duv.w};
                float ys[4];
#pragma unroll
                for (int i4 = 0; i4 < 4; ++i4) {
                    const int i = 4 * c + i4;
                    const uint64_t dl2 = pack2(dls[i4], dls[i4]), du2 = pack2(dus[i4], dus[i4]);
                    uint64_t bp[HS / 2], cp[HS / 2];
                    lds_pairs<HS>(Bt + i * NS, bp);
                    if (SUMMARY) {
                        sum_dl += dls[i4];
#pragma unroll
                        for (int j = 0; j < HS / 2; ++j) {
                            float x0, x1;
                            unpack2(mul2(dl2, A2[j]), x0, x1);
                            h[j] = fma2(pack2(ex2(x0), ex2(x1)), h[j], mul2(du2, bp[j]));
                        }
                        ys[i4] = 0.f;
                    } else {
                        lds_pairs<HS>(Ct + i * NS, cp);
                        uint64_t ya = pack2(0.f, 0.f), yb = pack2(0.f, 0.f);
#pragma unroll
                        for (int j = 0; j < HS / 2; ++j) {
                            float x0, x1;
                            unpack2(mul2(dl2, A2[j]), x0, x1);
                            h[j] = fma2(pack2(ex2(x0), ex2(x1)), h[j], mul2(du2, bp[j]));
                            if (j & 1) yb = fma2(h[j], cp[j], yb);
                            else ya = fma2(h[j], cp[j], ya);
                        }
                        float s0, s1, s2, s3;
                        unpack2(ya, s0, s1);
                        unpack2(yb, s2, s3);
                        ys[i4] = (s0 + s1) + (s2 + s3);
                    }
                }
                if (!SUMMARY) *reinterpret_cast<float4 *>(reinterpret_cast<uint8_t *>(sm.yp[buf][w]) + off) = make_float4(ys[0], ys[1], ys[2], ys[3]);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.ydone[buf]);
        }
        if (!live) return;
        if (SUMMARY) {
            const int64_t o = (((int64_t)b * sp.nseg + seg) * a.dim + d) * N;
#pragma unroll
            for (int j = 0; j < HS / 2; ++j) {
                float lo, hi, a0, a1;
                unpack2(h[j], lo, hi);
                unpack2(A2[j], a0, a1);
                const int n = w * HS + 2 * j;
                if (n < N) { sp.hend[o + n] = lo; sp.pdec[o + n] = ex2(a0 * sum_dl); }
                if (n + 1 < N) { sp.hend[o + n + 1] = hi; sp.pdec[o + n + 1] = ex2(a1 * sum_dl); }
            }
        } else if (a.last_state && seg == sp.nseg - 1) {
            float *ls = a.last_state + ((int64_t)b * a.dim + d) * N;
#pragma unroll
            for (int j = 0; j < HS / 2; ++j) {
                float lo, hi;
                unpack2(h[j], lo, hi);
                if (w * HS + 2 * j < N) ls[w * HS + 2 * j] = lo;
                if (w * HS + 2 * j + 1 < N) ls[w * HS + 2 * j + 1] = hi;
            }
        }
    }
}

// h0[b][s+1] = pdec[b][s] * h0[b][s] + hend[b][s] over the segments of a split sequence, one thread per (row, channel, state); all
// segments' values are asked for at once (with the loads behind the stores of the segment before: 4.4 us for 5120 channels x 8, now 2)
constexpr int kMaxSegments = 16;
__global__ void __launch_bounds__(256) scan_fold_segments_kernel(float *__restrict__ h0, const float *__restrict__ hend, const float *__restrict__ pdec, int nseg,
                                                                 int64_t per_seg, int64_t rows)
{
    pdl_trigger();
    pdl_wait();
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= rows * per_seg) return;
    const int64_t b = i / per_seg, e = i % per_seg, o = b * nseg * per_seg + e;
    float end[kMaxSegments - 1], dec[kMaxSegments - 1], h = 0.f;
#pragma unroll
    for (int s = 0; s < kMaxSegments - 1; ++s) {
        end[s] = s + 1 < nseg ? hend[o + s * per_seg] : 0.f;
        dec[s] = s + 1 < nseg ? pdec[o + s * per_seg] : 0.f;
    }
#pragma unroll
    for (int s = 0; s < kMaxSegments; ++s) {
        if (s < nseg) h0[o + s * per_seg] = h;
        if (s + 1 < kMaxSegments) h = fmaf(dec[s], h, end[s]);
    }
}

bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

template <typename T> int split_segments(const mb200_scan_args &a);

// The channel-parallel kernel works on tiles of 32 channels of one group.
int64_t channel_tiles(const mb200_scan_args &a) { return (int64_t)a.batch * a.ngroups * ((a.dim / a.ngroups + kStreamCh - 1) / kStreamCh); }

template <typename T> bool stream_tiles(const mb200_scan_args &a);

// Every row of u, delta, z and the outputs starts on a 16-byte boundary.
template <typename T>
bool rows_aligned(const mb200_scan_args &a)
{
    constexpr int VEC = 16 / sizeof(T);
    auto ok = [](const void *p, const int64_t *s) { return aligned16(p) && s[0] % VEC == 0 && s[1] % VEC == 0; };
    return ok(a.u, a.u_stride) && ok(a.delta, a.delta_stride) && ok(a.out, a.out_stride) && (!a.z || ok(a.z, a.z_stride)) &&
           (!a.z || !a.out_pregate || ok(a.out_pregate, a.pregate_stride));
}

// Which calls the channel-parallel kernel serves.  It keeps at most 16 states per channel in registers and takes its B and C from the
// input; fewer than kStreamMinChannels channels would leave most of the GPU idle unless the sequence can be cut.  Rows that TMA can
// describe need no more than that.  Where the lanes fetch the rows (stream_tiles is false), a pass is a chain of about 0.11 us per step
// however few the tiles, and lanes past the end of a group are idle, so that the time-parallel kernel -- which takes 512 steps of a
// channel at a time -- is often the faster one.  Measured, lanes / time-parallel, us, bf16 and 16 states unless said:
//   one pass, 999 steps:         2048 channels 105 / 55, 4128: 106 / 101, 5120: 115 / 134; 8 states, 6144: 121 / 109, 8192: 122 / 140
//   one pass, 133 steps:         1024 channels 21.5 / 24.6; 8 states, 2048: 22 / 20, 3072: 23 / 29
//   16 segments, 2048 steps:     1008 channels in groups of 24: 64 / 83; 4097 steps, 2048 channels: 163 / 201
//   8 segments, 1999 steps:      2048 channels 95 / 101, 3072: 151 / 176; 2000 channels in groups of 40 (800 CTAs): 113 / 93
//   groups that fill half of a tile, one pass, 2048 steps: 8192 channels 329 / 340, fp32 398 / 355; a quarter of a tile: 552 / 342
//   8 states, rows on 16-byte boundaries (which the time-parallel kernel loads in packets): 7680 channels in groups of 80: 245 / 203,
//   40960: 780 / 719
template <typename T>
bool stream_eligible(const mb200_scan_args &a)
{
    if (a.dstate > 16 || !a.B_variable || !a.C_variable) return false;
    const int64_t channels = (int64_t)a.batch * a.dim, tiles = channel_tiles(a);
    const int nseg = split_segments<T>(a);
    if (channels < kStreamMinChannels && nseg <= 1) return false;
    if (stream_tiles<T>(a)) return true;
    const bool few_states = a.dstate <= 8;
    if (channels * (few_states ? 24 : sizeof(T) == 4 ? 30 : 32) < tiles * kStreamCh * 16) return false;       // too few live lanes
    if (few_states && channels >= kStreamMinChannels && rows_aligned<T>(a)) return false;
    if (nseg > 1) return nseg > 8 || tiles * nseg <= 4 * 148 || channels >= 2688;
    const int64_t steps = a.seqlen;      // of the chain, against channels of the other kernel
    return channels >= (few_states ? std::min<int64_t>(7168, 12 * steps + 768) : std::min<int64_t>(4608, 10 * steps - 320));
}

// ... and its operands can be described to TMA: 16-byte aligned bases and row strides, whole groups of 32 channels, one output.
template <typename T>
bool stream_tiles(const mb200_scan_args &a)
{
    constexpr int VEC = 16 / sizeof(T);
    if (a.out_pregate || (a.dim / a.ngroups) % kStreamCh != 0) return false;
    // the output tile store clips the innermost dimension in 16-byte units, not in elements: a row (of a wider buffer)
    // that ends inside such a unit would have the bytes after its end overwritten
    if (((size_t)a.seqlen * sizeof(T)) % 16 != 0) return false;
    auto ok2 = [&](const void *p, const int64_t *s) { return aligned16(p) && s[0] > 0 && s[1] > 0 && s[0] % VEC == 0 && s[1] % VEC == 0; };
    auto ok3 = [&](const void *p, const int64_t *s) {
        return aligned16(p) && s[0] > 0 && s[1] > 0 && s[2] > 0 && s[0] % VEC == 0 && s[1] % VEC == 0 && s[2] % VEC == 0;
    };
    if (!ok2(a.u, a.u_stride) || !ok2(a.delta, a.delta_stride) || !ok2(a.out, a.out_stride)) return false;
    if (a.z && !ok2(a.z, a.z_stride)) return false;
    if (!ok3(a.B, a.B_stride) || !ok3(a.C, a.C_stride)) return false;
    return encode_fn() != nullptr;
}

// How many segments the sequence is cut into (1 = one pass).  Cutting pays when the channel groups alone leave most
// of the GPU idle: with G tiles of 32 channels, nseg is the largest power of two with G * nseg CTAs in one wave
// of 9 per SM.  It costs a second pass over every segment but the last, so it is used only from nseg = 8 up (fewer
// segments measured no faster than one pass), with segments of at least 128 steps, and only when the caller lent
// scratch for the summaries.
template <typename T>
int split_segments(const mb200_scan_args &a)
{
    const int64_t tiles = channel_tiles(a);
    int nseg = 1;
    while (nseg < kMaxSegments && tiles * nseg * 2 <= 9 * 148 && a.seqlen / (nseg * 2) >= 128) nseg *= 2;
    if (nseg < 8) return 1;
    const size_t need = 3 * sizeof(float) * (size_t)a.batch * nseg * a.dim * a.dstate;
    if (!a.scratch || a.scratch_bytes < need || (reinterpret_cast<uintptr_t>(a.scratch) & 15)) return 1;
    return nseg;
}

template <typename T>
int launch_stream(const mb200_scan_args &a, cudaStream_t stream)
{
    constexpr uint32_t TB = 32 / sizeof(T);
    const int dtype = sizeof(T) == 4 ? MB200_F32 : (std::is_same<T, __half>::value ? MB200_F16 : MB200_BF16);
    ScanMaps maps = {};
    auto rows = [&](CUtensorMap *m, const void *p, const int64_t *st) {
        const uint64_t dims[3] = {(uint64_t)a.seqlen, (uint64_t)a.dim, (uint64_t)a.batch};
        const uint64_t sb[2] = {(uint64_t)st[1] * sizeof(T), (uint64_t)st[0] * sizeof(T)};
        const uint32_t box[3] = {TB, (uint32_t)kStreamCh, 1};
        return encode_tiled(m, dtype, p, 3, dims, sb, box, CU_TENSOR_MAP_SWIZZLE_32B);
    };
    auto bc = [&](CUtensorMap *m, const void *p, const int64_t *st, uint32_t ns) {
        const uint64_t dims[4] = {(uint64_t)a.seqlen, (uint64_t)a.dstate, (uint64_t)a.ngroups, (uint64_t)a.batch};
        const uint64_t sb[3] = {(uint64_t)st[2] * sizeof(T), (uint64_t)st[1] * sizeof(T), (uint64_t)st[0] * sizeof(T)};
        const uint32_t box[4] = {TB, ns, 1, 1};
        return encode_tiled(m, dtype, p, 4, dims, sb, box, CU_TENSOR_MAP_SWIZZLE_32B);
    };
    const uint32_t ns = a.dstate <= 8 ? 8 : 16;
    // (the driver may refuse a map for unusual strides: the lanes' own loads take those)
    bool tiles = stream_tiles<T>(a) && rows(&maps.u, a.u, a.u_stride) && rows(&maps.dt, a.delta, a.delta_stride) && rows(&maps.out, a.out, a.out_stride) &&
              bc(&maps.B, a.B, a.B_stride, ns) && bc(&maps.C, a.C, a.C_stride, ns);
    if (a.z) tiles = tiles && rows(&maps.z, a.z, a.z_stride);
    else maps.z = maps.u;
    const int group_tiles = (a.dim / a.ngroups + kStreamCh - 1) / kStreamCh;
    int nseg = split_segments<T>(a);
    int seg_len = (int)((a.seqlen + TB - 1) / TB * TB);
    if (nseg > 1) {
        seg_len = (int)(((a.seqlen + nseg - 1) / nseg + TB - 1) / TB * TB);     // whole tiles per segment
        nseg = (a.seqlen + seg_len - 1) / seg_len;                              // rounding up may leave the last ones empty
    }
    // A grid that leaves the SMs partly empty runs the six- or four-warp layout (four / six CTAs of them fit an SM).
    auto go = [&](dim3 grid, const ScanSplit &split, bool summary) {
        const int64_t ctas = (int64_t)grid.x * grid.y;
        auto pick = [&](auto ns_c, auto sum_c, auto tma_c) {
            constexpr int NS = decltype(ns_c)::value;
            constexpr bool SUM = decltype(sum_c)::value, TMA = decltype(tma_c)::value;
            auto run = [&](auto sw_c, auto split_c) {
                constexpr int SW = decltype(sw_c)::value;
                constexpr bool SPLIT = decltype(split_c)::value;
                constexpr int threads = 32 * (SW + (SPLIT ? 2 : 1));
                constexpr size_t smem = sizeof(StreamSmem<T, NS, SW, SPLIT, TMA>);
                auto kernel = scan_stream_kernel<T, NS, SUM, SW, SPLIT, TMA>;
                launch_dependent_if(split.h0 != nullptr, kernel, grid, threads, smem, stream, a, maps, split);        // (after the fold)
            };
            // fp32 rows fetched by the lanes take two granules per hand-off, of which shared memory holds three: a single scalar warp would
            // wait for the last it asked for.  Rows off their 16-byte boundaries need twice the sectors, and the six-warp layout whatever
            // the grid (us: six, four, three warps; 8 x 5120 channels of 1999 steps: 901, 1466, 1720; 40960 channels in groups of 80, 2048
            // steps, aligned: 1122, 1073, 1268; 16000 of them, 600 CTAs: 598, 509, -).
            constexpr bool kLanes32 = sizeof(T) == 4 && !TMA;
            if (ctas <= 4 * 148 || (kLanes32 && !rows_aligned<T>(a))) run(std::integral_constant<int, 4>{}, std::true_type{});
            else if (ctas <= 6 * 148 || kLanes32) run(std::integral_constant<int, 2>{}, std::true_type{});
            else if constexpr (!kLanes32) run(std::integral_constant<int, 2>{}, std::false_type{});
        };
        auto with_ns = [&](auto ns_c) {
            if (tiles) summary ? pick(ns_c, std::true_type{}, std::true_type{}) : pick(ns_c, std::false_type{}, std::true_type{});
            else summary ? pick(ns_c, std::true_type{}, std::false_type{}) : pick(ns_c, std::false_type{}, std::false_type{});
        };
        if (ns == 8) with_ns(std::integral_constant<int, 8>{});
        else with_ns(std::integral_constant<int, 16>{});
    };
    if (nseg <= 1) {
        const ScanSplit one = {1, seg_len, nullptr, nullptr, nullptr};
        go(dim3(a.ngroups * group_tiles, a.batch), one, false);
        return MB200_OK;
    }
    // Few channel groups: the sequence is cut into nseg segments that run side by side.  A first launch summarises
    // every segment but the last from a zero state (end state + decay product), a fold turns the summaries into the
    // state entering each segment, a second launch runs every segment from there.
    const int64_t per_seg = (int64_t)a.dim * a.dstate, region = (int64_t)a.batch * nseg * per_seg;
    float *h0 = static_cast<float *>(a.scratch), *hend = h0 + region, *pdec = hend + region;
    const ScanSplit sum = {nseg, seg_len, nullptr, hend, pdec}, full = {nseg, seg_len, h0, nullptr, nullptr};
    dim3 grid(a.ngroups * group_tiles, a.batch * nseg);       // in the summary launch the CTAs of the last segment return at once
    go(grid, sum, true);
    launch_dependent(scan_fold_segments_kernel, dim3((unsigned)((a.batch * per_seg + 255) / 256)), 256, 0, stream, h0, hend, pdec, nseg, per_seg, a.batch);
    go(grid, full, false);
    return MB200_OK;
}

template <typename T>
int launch_scan(const mb200_scan_args &a, cudaStream_t stream)
{
    const int N = a.dstate;
    const int nblocks = (N + kStateBlock - 1) / kStateBlock;
    const int per_group = a.dim / a.ngroups;
    // more channels per staged B/C tile when the states fit one block and there is enough work
    int cpw = 1;
    if (nblocks == 1 && per_group >= 2 * kWarps && (int64_t)a.batch * a.dim >= 8 * kWarps * 2 * 148) cpw = 2;
    const int chans = kWarps * cpw;
    const int npad = N;
    const bool io_vec = rows_aligned<T>(a);
    // staging reads 4 elements at a time: 8 bytes for 16-bit types, 16 for fp32
    const int bc_align = sizeof(T) == 4 ? 16 : 8;
    bool bc_vec = true;
    if (a.B_variable)
        bc_vec = bc_vec && (reinterpret_cast<uintptr_t>(a.B) % bc_align == 0) && a.B_stride[0] % 4 == 0 &&
                 a.B_stride[1] % 4 == 0 && a.B_stride[2] % 4 == 0;
    if (a.C_variable)
        bc_vec = bc_vec && (reinterpret_cast<uintptr_t>(a.C) % bc_align == 0) && a.C_stride[0] % 4 == 0 &&
                 a.C_stride[1] % 4 == 0 && a.C_stride[2] % 4 == 0;
    const int vec_flags = (io_vec ? 1 : 0) | (bc_vec ? 2 : 0);
    if (stream_eligible<T>(a)) return launch_stream<T>(a, stream);
    // Four warps per channel while that is at most one CTA per SM; beyond, their barriers cost more than the shorter chain saves
    // (bf16, 777 steps, us, four warps / one: 512 channels of 16 states 27 / 45, 640: 43 / 45; of 8 states 22 / 31, 35 / 31).
    if (N <= kStateBlock && a.B_variable && a.C_variable && (int64_t)a.batch * a.ngroups * ((per_group + 3) / 4) <= 148) {
        auto go = [&](auto ch_c) {
            constexpr int CH = decltype(ch_c)::value;
            const cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void *>(&scan_few_kernel<T, CH>), (int)sizeof(FewSmem<CH>), a.device);
            if (e != cudaSuccess) return fail(MB200_ERR_LAUNCH, "selective_scan: shared memory opt-in (%zu B): %s", sizeof(FewSmem<CH>), cudaGetErrorString(e));
            launch_dependent(scan_few_kernel<T, CH>, dim3(a.ngroups * ((per_group + CH - 1) / CH), a.batch), CH * 128, sizeof(FewSmem<CH>), stream, a, vec_flags);
            return (int)MB200_OK;
        };
        return (int64_t)a.batch * a.dim > 2 * 148 ? go(std::integral_constant<int, 4>{}) : go(std::integral_constant<int, 2>{});
    }
    const size_t smem = sizeof(float) * (2 * kStateBlock * kTile + 2 * (size_t)chans * npad);
    static_assert(2 * kStateBlock * kTile * sizeof(float) + 2 * kWarps * 2 * 256 * sizeof(float) <= 227 * 1024, "smem budget");
    cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void *>(&scan_fwd_kernel<T>), (int)smem, a.device);
    if (e != cudaSuccess) return fail(MB200_ERR_LAUNCH, "selective_scan: shared memory opt-in (%zu B): %s", smem, cudaGetErrorString(e));
    const int tiles_per_group = (per_group + chans - 1) / chans;
    dim3 grid(a.ngroups * tiles_per_group, a.batch);
    scan_fwd_kernel<T><<<grid, kThreads, smem, stream>>>(a, cpw, nblocks, npad, vec_flags);
    return MB200_OK;
}

}  // namespace
}  // namespace mb200

extern "C" int mb200_scan_scratch_bytes(const mb200_scan_args *args, size_t *bytes)
{
    using namespace mb200;
    if (!args || !bytes) return fail(MB200_ERR_BAD_ARG, "scan_scratch_bytes: NULL argument");
    const mb200_scan_args &a = *args;
    *bytes = 0;
    if (a.batch <= 0 || a.dim <= 0 || a.dstate <= 0 || a.dstate > 16 || a.seqlen <= 0) return MB200_OK;
    // the size that would let the sequence be cut: ask the policy with a scratch that is certainly large enough
    mb200_scan_args probe = a;
    probe.scratch = reinterpret_cast<void *>(uintptr_t(256));
    probe.scratch_bytes = ~size_t(0);
    const int nseg = split_segments<float>(probe);
    if (nseg > 1) *bytes = 3 * sizeof(float) * (size_t)a.batch * nseg * a.dim * a.dstate;
    return MB200_OK;
}

extern "C" int mb200_scan_status(int device, int *status)
{
    using namespace mb200;
    if (!status) return fail(MB200_ERR_BAD_ARG, "scan_status: status is NULL");
    if (int rc = enter_device(device)) return rc;
    cudaError_t e = cudaMemcpyFromSymbol(status, g_scan_status, sizeof(int));
    int bwd = 0;
    if (e == cudaSuccess) e = scan_bwd_status(&bwd);
    if (e != cudaSuccess) return fail(MB200_ERR_LAUNCH, "scan_status: %s", cudaGetErrorString(e));
    if (*status == 0) *status = bwd;
    return MB200_OK;
}

extern "C" int mb200_selective_scan_fwd(const mb200_scan_args *args, void *stream_)
{
    using namespace mb200;
    if (!args) return fail(MB200_ERR_BAD_ARG, "selective_scan_fwd: args is NULL");
    const mb200_scan_args &a = *args;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    MB200_CHECK_ARG(a.batch >= 0 && a.dim > 0 && a.seqlen >= 0 && a.dstate > 0 && a.ngroups > 0,
                    "selective_scan_fwd: bad sizes (batch %d dim %d seqlen %d dstate %d ngroups %d)", a.batch, a.dim,
                    a.seqlen, a.dstate, a.ngroups);
    MB200_CHECK_ARG(a.dstate <= 256, "selective_scan only supports state dimension <= 256");
    MB200_CHECK_ARG(a.dim % a.ngroups == 0, "selective_scan_fwd: dim must be divisible by ngroups");
    MB200_CHECK_ARG(a.io_dtype == MB200_F32 || a.io_dtype == MB200_F16 || a.io_dtype == MB200_BF16,
                    "selective_scan_fwd: unknown io_dtype %d", a.io_dtype);
    MB200_CHECK_ARG(a.batch <= 65535, "selective_scan_fwd: batch must be <= 65535");
    MB200_CHECK_ARG(!a.out_pregate || a.z, "selective_scan_fwd: out_pregate is only meaningful with z");
    if (a.batch == 0) return MB200_OK;   // nothing to do; empty tensors carry NULL pointers
    MB200_CHECK_ARG(a.u && a.delta && a.A && a.B && a.C && a.out, "selective_scan_fwd: a required tensor is NULL");
    if (int rc = enter_device(a.device)) return rc;
    if (a.seqlen == 0) {
        if (a.last_state) {
            cudaError_t e = cudaMemsetAsync(a.last_state, 0, sizeof(float) * (size_t)a.batch * a.dim * a.dstate, stream);
            if (e != cudaSuccess) return fail(MB200_ERR_LAUNCH, "selective_scan_fwd: memset: %s", cudaGetErrorString(e));
        }
        return MB200_OK;
    }
    int rc;
    if (a.io_dtype == MB200_F32) rc = launch_scan<float>(a, stream);
    else if (a.io_dtype == MB200_BF16) rc = launch_scan<__nv_bfloat16>(a, stream);
    else rc = launch_scan<__half>(a, stream);
    if (rc) return rc;
    MB200_CHECK_LAUNCH("selective_scan_fwd");
    return MB200_OK;
}
