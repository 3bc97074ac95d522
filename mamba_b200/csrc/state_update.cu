// Single-token decode state update for sm_100a.
//
// The operator streams the recurrent state once (read + write in place); everything else is a
// few hundred bytes per (batch, head).  The fast kernel therefore gives every state row to a
// group of LPR lanes that each own one 16-byte packet of the row, and a lane has kRowsInFlight rows in work and as many of
// the next on their way, with what else their outputs need (x, dt, z, D: one row's in each quarter of the lanes), before it touches any of them; B, C, dt and
// exp(A dt) of the (batch, head) stay in registers.  The outputs of a group's rows are reduced together, each in a quarter of
// the lanes, so that they are also finished and stored together.
// Measured (fp32 state, 64 x 128 per head): 225 us for 256 x 80 heads (248 when a row's x, z and D were loaded when their turn
// came, behind the stores of the row before); 3.8 us for 1 x 80 heads (13.4 with one CTA per head).
// A general kernel (one warp per row, scalar strided accesses)
// serves layouts the packet path cannot: odd dstate, strided or unaligned state, any dtype mix.
#include "common.cuh"

namespace mb200 {

namespace {

constexpr int kThreads = 64;         // many small CTAs hide the per-(batch, head) set-up latency best
constexpr int kRowsInFlight = 4;     // state rows a lane group loads before it touches any of them
constexpr int kRowTile = 64;         // state rows per CTA (amortises the B / C / dt set-up) ...
constexpr int kFewCtas = 148 * 8;    // ... unless the grid would have fewer CTAs than this: then latency is what counts, and fewer rounds

// out rows of a padding entry (state_batch_indices < 0) are defined to be zero.
__device__ void zero_rows(const mb200_ssu_args &a, int b, int h, int p0, int rows)
{
    for (int r = threadIdx.x; r < rows; r += blockDim.x)
        store_any(a.out, a.x_dtype, (int64_t)b * a.out_stride[0] + (int64_t)h * a.out_stride[1] + (int64_t)(p0 + r) * a.out_stride[2], 0.f);
}

// VEC consecutive entries of a row of B, C or A, in one or two loads where they lie side by side on their own alignment
template <int VEC>
__device__ __forceinline__ void load_row(const void *p, int dtype, int64_t i, int64_t stride, float (&f)[VEC])
{
    const int size = dtype == MB200_F32 ? 4 : 2;
    const char *q = static_cast<const char *>(p) + i * size;
    if (stride == 1 && (reinterpret_cast<uintptr_t>(q) & ((VEC * size < 16 ? VEC * size : 16) - 1)) == 0) {
        if (dtype == MB200_F32) {
#pragma unroll
            for (int k = 0; k < VEC / 4; ++k) {
                const float4 v = reinterpret_cast<const float4 *>(q)[k];
                f[4 * k] = v.x; f[4 * k + 1] = v.y; f[4 * k + 2] = v.z; f[4 * k + 3] = v.w;
            }
        } else {
            uint32_t w[VEC / 2];
            if constexpr (VEC == 8) {
                const uint4 v = *reinterpret_cast<const uint4 *>(q);
                w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
            } else {
                const uint2 v = *reinterpret_cast<const uint2 *>(q);
                w[0] = v.x; w[1] = v.y;
            }
#pragma unroll
            for (int k = 0; k < VEC; ++k) {
                const uint16_t e = (uint16_t)(w[k >> 1] >> (16 * (k & 1)));
                f[k] = dtype == MB200_BF16 ? __uint_as_float((uint32_t)e << 16) : __half2float(__ushort_as_half(e));
            }
        }
    } else {
#pragma unroll
        for (int k = 0; k < VEC; ++k) f[k] = load_any(p, dtype, i + k * stride);
    }
}

template <typename StateT, int LPR, int NC, bool TIED>
__global__ void __launch_bounds__(kThreads) ssu_packet_kernel(const mb200_ssu_args a, const int row_tile)
{
    pdl_wait();
    pdl_trigger();
    constexpr int VEC = 16 / sizeof(StateT);
    constexpr int GROUPS = kThreads / LPR;
    const int b = blockIdx.y, h = blockIdx.z;
    const int p0 = blockIdx.x * row_tile;
    const int rows = min(row_tile, a.dim - p0);
    const int lir = threadIdx.x % LPR;   // lane within the row group
    const int group = threadIdx.x / LPR;

    int64_t sb = b;
    if (a.state_batch_indices) {
        const int idx = a.state_batch_indices[b];
        if (idx < 0) {
            zero_rows(a, b, h, p0, rows);
            return;
        }
        sb = idx;
    }
    StateT *state = static_cast<StateT *>(a.state) + sb * a.state_stride[0] + (int64_t)h * a.state_stride[1];
    const int g = h / (a.nheads / a.ngroups);
    const int64_t xo = (int64_t)b * a.x_stride[0] + (int64_t)h * a.x_stride[1];
    const int64_t dto = (int64_t)b * a.dt_stride[0] + (int64_t)h * a.dt_stride[1];
    const int64_t zo = (int64_t)b * a.z_stride[0] + (int64_t)h * a.z_stride[1];
    const int64_t oo = (int64_t)b * a.out_stride[0] + (int64_t)h * a.out_stride[1];

    // where the sums of my group's kRowsInFlight rows end up: row fin_u in the lanes of its quarter, finished by the first of them
    constexpr bool kTogether = LPR >= kRowsInFlight;
    const int fin_u = kTogether ? lir / (LPR / kRowsInFlight) : 0;
    const bool fin_lane = lir % (kTogether ? LPR / kRowsInFlight : LPR) == 0;

    struct Round {
        Vec16<StateT> pk[kRowsInFlight][NC];
        float x[kTogether ? 1 : kRowsInFlight], dt[kTogether ? 1 : kRowsInFlight];       // of the row that I finish, else of all
        float z, D;
    };
    auto load_round = [&](Round &q, int r0) {
#pragma unroll
        for (int u = 0; u < kRowsInFlight; ++u) {
            const int r = r0 + u * GROUPS;
            if (r < rows) {
                const StateT *row = state + (int64_t)(p0 + r) * a.state_stride[2];
#pragma unroll
                for (int c = 0; c < NC; ++c) q.pk[u][c].load(row + (c * LPR + lir) * VEC);
            }
        }
#pragma unroll
        for (int u = 0; u < (kTogether ? 1 : kRowsInFlight); ++u) {
            const int64_t p = p0 + min(r0 + (kTogether ? fin_u : u) * GROUPS, rows - 1);
            q.x[u] = load_any(a.x, a.x_dtype, xo + p * a.x_stride[2]);
            if (!TIED) {
                q.dt[u] = load_any(a.dt, a.dt_dtype, dto + p * a.dt_stride[2]);
                if (a.dt_bias) q.dt[u] += a.dt_bias[(int64_t)h * a.dt_bias_stride[0] + p * a.dt_bias_stride[1]];
            }
            if (kTogether) {
                q.z = a.z ? load_any(a.z, a.x_dtype, zo + p * a.z_stride[2]) : 0.f;
                q.D = a.D ? a.D[(int64_t)h * a.D_stride[0] + p * a.D_stride[1]] : 0.f;
            }
        }
    };
    // The state rows are the only real traffic: put the first round in flight before
    // the (latency-bound) per-(batch, head) set-up below.
    Round next;
    load_round(next, group);

    float Bv[NC][VEC], Cv[NC][VEC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        const int64_t n = (c * LPR + lir) * VEC;
        load_row<VEC>(a.B, a.bc_dtype, (int64_t)b * a.B_stride[0] + (int64_t)g * a.B_stride[1] + n * a.B_stride[2], a.B_stride[2], Bv[c]);
        load_row<VEC>(a.C, a.bc_dtype, (int64_t)b * a.C_stride[0] + (int64_t)g * a.C_stride[1] + n * a.C_stride[2], a.C_stride[2], Cv[c]);
    }

    float dt_tied = 0.f, dA_tied = 0.f;
    if (TIED) {
        const float Ah = a.A[(int64_t)h * a.A_stride[0]];
        dt_tied = load_any(a.dt, a.dt_dtype, dto);
        if (a.dt_bias) dt_tied += a.dt_bias[(int64_t)h * a.dt_bias_stride[0]];
        if (a.dt_softplus) dt_tied = softplus20(dt_tied);
        dA_tied = expf(Ah * dt_tied);
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
            for (int i = 0; i < VEC; ++i) Bv[c][i] *= dt_tied;   // B dt, shared by every row
    }

    // every thread runs the same number of rounds (the shuffles below need whole warps)
    for (int base = 0; base < rows; base += GROUPS * kRowsInFlight) {
        const int r0 = base + group;
        Round q = next;
        if (base + GROUPS * kRowsInFlight < rows) load_round(next, r0 + GROUPS * kRowsInFlight);
        float y[kRowsInFlight];
        if (!TIED && a.dt_softplus) {
#pragma unroll
            for (int u = 0; u < (kTogether ? 1 : kRowsInFlight); ++u) q.dt[u] = softplus20(q.dt[u]);
        }
#pragma unroll
        for (int u = 0; u < kRowsInFlight; ++u) {
            const int r = r0 + u * GROUPS;
            // with one row per lane, x and dt come from the lanes that have this one
            const float xv = kTogether ? __shfl_sync(0xffffffffu, q.x[0], u * (LPR / kRowsInFlight), LPR) : q.x[kTogether ? 0 : u];
            const float dtv = TIED ? dt_tied : kTogether ? __shfl_sync(0xffffffffu, q.dt[0], u * (LPR / kRowsInFlight), LPR) : q.dt[kTogether ? 0 : u];
            y[u] = 0.f;
            if (r < rows) {
                const int64_t p = p0 + r;
                StateT *row = state + p * a.state_stride[2];
                [[maybe_unused]] float Av[VEC];
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    if (!TIED)
                        load_row<VEC>(a.A, MB200_F32, (int64_t)h * a.A_stride[0] + p * a.A_stride[1] + (c * LPR + lir) * VEC * a.A_stride[2], a.A_stride[2], Av);
                    float s[VEC];
                    q.pk[u][c].unpack(s);
#pragma unroll
                    for (int i = 0; i < VEC; ++i) {
                        float dA, dBx;
                        if (TIED) {
                            dA = dA_tied;
                            dBx = Bv[c][i] * xv;
                        } else {
                            dA = __expf(Av[i] * dtv);
                            dBx = Bv[c][i] * dtv * xv;
                        }
                        s[i] = fmaf(s[i], dA, dBx);
                        y[u] = fmaf(s[i], Cv[c][i], y[u]);
                    }
                    q.pk[u][c].pack(s);
                    q.pk[u][c].store(row + (c * LPR + lir) * VEC);
                }
            }
        }
        auto finish = [&](int r, float v, float xv, float zv, float Dv) {
            if (a.D) v = fmaf(xv, Dv, v);
            if (a.z) v *= silu(zv);
            store_any(a.out, a.x_dtype, oo + (int64_t)(p0 + r) * a.out_stride[2], v);
        };
        if constexpr (kTogether) {       // four sums in six shuffles instead of twenty
            static_assert(kRowsInFlight == 4, "two halvings");
            const bool up = lir & (LPR / 2), up2 = lir & (LPR / 4);
            float k0 = up ? y[2] : y[0], k1 = up ? y[3] : y[1];
            k0 += __shfl_xor_sync(0xffffffffu, up ? y[0] : y[2], LPR / 2);
            k1 += __shfl_xor_sync(0xffffffffu, up ? y[1] : y[3], LPR / 2);
            float v = up2 ? k1 : k0;
            v += __shfl_xor_sync(0xffffffffu, up2 ? k0 : k1, LPR / 4);
#pragma unroll
            for (int o = LPR / 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            const int r = r0 + fin_u * GROUPS;
            if (fin_lane && r < rows) finish(r, v, q.x[0], q.z, q.D);
        } else {
#pragma unroll
            for (int u = 0; u < kRowsInFlight; ++u) {
                const int r = r0 + u * GROUPS;
                float v = y[u];
#pragma unroll
                for (int o = LPR / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (fin_lane && r < rows) {
                    const int64_t p = p0 + r;
                    finish(r, v, q.x[u], a.z ? load_any(a.z, a.x_dtype, zo + p * a.z_stride[2]) : 0.f,
                           a.D ? a.D[(int64_t)h * a.D_stride[0] + p * a.D_stride[1]] : 0.f);
                }
            }
        }
    }
}

// One warp per state row, every access scalar and fully strided.
__global__ void __launch_bounds__(128) ssu_general_kernel(const mb200_ssu_args a)
{
    pdl_wait();
    pdl_trigger();
    const int b = blockIdx.y, h = blockIdx.z;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int p = blockIdx.x * 4 + warp;
    if (p >= a.dim) return;
    const int64_t oi = (int64_t)b * a.out_stride[0] + (int64_t)h * a.out_stride[1] + (int64_t)p * a.out_stride[2];
    int64_t sb = b;
    if (a.state_batch_indices) {
        const int idx = a.state_batch_indices[b];
        if (idx < 0) {
            if (lane == 0) store_any(a.out, a.x_dtype, oi, 0.f);
            return;
        }
        sb = idx;
    }
    const int g = h / (a.nheads / a.ngroups);
    const float xv = load_any(a.x, a.x_dtype, (int64_t)b * a.x_stride[0] + (int64_t)h * a.x_stride[1] + (int64_t)p * a.x_stride[2]);
    float dtv = load_any(a.dt, a.dt_dtype, (int64_t)b * a.dt_stride[0] + (int64_t)h * a.dt_stride[1] + (int64_t)p * a.dt_stride[2]);
    if (a.dt_bias) dtv += a.dt_bias[(int64_t)h * a.dt_bias_stride[0] + (int64_t)p * a.dt_bias_stride[1]];
    if (a.dt_softplus) dtv = softplus20(dtv);
    const int64_t so = sb * a.state_stride[0] + (int64_t)h * a.state_stride[1] + (int64_t)p * a.state_stride[2];
    const float *Arow = a.A + (int64_t)h * a.A_stride[0] + (int64_t)p * a.A_stride[1];
    float y = 0.f;
    for (int n = lane; n < a.dstate; n += 32) {
        const float Bn = load_any(a.B, a.bc_dtype, (int64_t)b * a.B_stride[0] + (int64_t)g * a.B_stride[1] + (int64_t)n * a.B_stride[2]);
        const float Cn = load_any(a.C, a.bc_dtype, (int64_t)b * a.C_stride[0] + (int64_t)g * a.C_stride[1] + (int64_t)n * a.C_stride[2]);
        float s = load_any(a.state, a.state_dtype, so + (int64_t)n * a.state_stride[3]);
        s = fmaf(s, expf(Arow[(int64_t)n * a.A_stride[2]] * dtv), Bn * dtv * xv);
        store_any(a.state, a.state_dtype, so + (int64_t)n * a.state_stride[3], s);
        y = fmaf(s, Cn, y);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
    if (lane == 0) {
        if (a.D) y = fmaf(xv, a.D[(int64_t)h * a.D_stride[0] + (int64_t)p * a.D_stride[1]], y);
        if (a.z) y *= silu(load_any(a.z, a.x_dtype, (int64_t)b * a.z_stride[0] + (int64_t)h * a.z_stride[1] + (int64_t)p * a.z_stride[2]));
        store_any(a.out, a.x_dtype, oi, y);
    }
}

template <typename StateT, int LPR, int NC>
int launch_packet(const mb200_ssu_args &a, bool tied, cudaStream_t stream)
{
    constexpr int GROUPS = kThreads / LPR;
    const int round = GROUPS * kRowsInFlight;
    int row_tile = round < kRowTile ? kRowTile : round;
    while (row_tile > round && (int64_t)((a.dim + row_tile - 1) / row_tile) * a.batch * a.nheads < kFewCtas) row_tile /= 2;
    if (row_tile > a.dim) row_tile = a.dim;
    dim3 grid((a.dim + row_tile - 1) / row_tile, a.batch, a.nheads);
    if (tied)
        launch_dependent(ssu_packet_kernel<StateT, LPR, NC, true>, grid, kThreads, 0, stream, a, row_tile);
    else
        launch_dependent(ssu_packet_kernel<StateT, LPR, NC, false>, grid, kThreads, 0, stream, a, row_tile);
    return MB200_OK;
}

template <typename StateT>
bool try_packet(const mb200_ssu_args &a, bool tied, cudaStream_t stream)
{
    constexpr int VEC = 16 / sizeof(StateT);
    if (a.dstate % VEC) return false;
    const int packets = a.dstate / VEC;
    switch (packets) {
    case 2: launch_packet<StateT, 2, 1>(a, tied, stream); return true;
    case 4: launch_packet<StateT, 4, 1>(a, tied, stream); return true;
    case 8: launch_packet<StateT, 8, 1>(a, tied, stream); return true;
    case 16: launch_packet<StateT, 16, 1>(a, tied, stream); return true;
    case 32: launch_packet<StateT, 32, 1>(a, tied, stream); return true;
    case 64: launch_packet<StateT, 32, 2>(a, tied, stream); return true;
    default: return false;
    }
}

bool valid_dtype(int d) { return d == MB200_F32 || d == MB200_F16 || d == MB200_BF16; }

}  // namespace
}  // namespace mb200

extern "C" int mb200_selective_state_update(const mb200_ssu_args *args, void *stream_)
{
    using namespace mb200;
    if (!args) return fail(MB200_ERR_BAD_ARG, "selective_state_update: args is NULL");
    const mb200_ssu_args &a = *args;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    MB200_CHECK_ARG(a.batch >= 0 && a.nheads > 0 && a.dim > 0 && a.dstate > 0 && a.ngroups > 0,
                    "selective_state_update: sizes must be positive (batch %d nheads %d dim %d dstate %d ngroups %d)",
                    a.batch, a.nheads, a.dim, a.dstate, a.ngroups);
    MB200_CHECK_ARG(a.nheads % a.ngroups == 0, "nheads must be divisible by ngroups");
    MB200_CHECK_ARG(valid_dtype(a.state_dtype) && valid_dtype(a.x_dtype) && valid_dtype(a.dt_dtype) && valid_dtype(a.bc_dtype),
                    "selective_state_update: unknown dtype code");
    MB200_CHECK_ARG(a.batch <= 65535 && a.nheads <= 65535, "selective_state_update: batch and nheads must be <= 65535");
    if (a.batch == 0) return MB200_OK;   // nothing to do; empty tensors carry NULL pointers
    MB200_CHECK_ARG(a.state && a.x && a.dt && a.A && a.B && a.C && a.out, "selective_state_update: a required tensor is NULL");
    if (int rc = enter_device(a.device)) return rc;

    const bool tied = a.A_stride[1] == 0 && a.A_stride[2] == 0 && a.dt_stride[2] == 0 &&
                      (!a.dt_bias || a.dt_bias_stride[1] == 0);
    const int vec = 16 / dtype_size(a.state_dtype);
    const bool packet_ok = a.state_stride[3] == 1 && a.state_stride[2] % vec == 0 && a.state_stride[1] % vec == 0 &&
                           a.state_stride[0] % vec == 0 && (reinterpret_cast<uintptr_t>(a.state) & 15) == 0;
    bool done = false;
    if (packet_ok) {
        if (a.state_dtype == MB200_F32) done = try_packet<float>(a, tied, stream);
        else if (a.state_dtype == MB200_BF16) done = try_packet<__nv_bfloat16>(a, tied, stream);
        else done = try_packet<__half>(a, tied, stream);
    }
    if (!done) {
        dim3 grid((a.dim + 3) / 4, a.batch, a.nheads);
        launch_dependent(ssu_general_kernel, grid, 128, 0, stream, a);
    }
    MB200_CHECK_LAUNCH("selective_state_update");
    return MB200_OK;
}
