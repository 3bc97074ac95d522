// Mamba-2 SSD chunked forward for sm_100a: the stages, their order, and the first and the third of them.
//
// Stages (each one launch, all on the caller's stream, handing fp32 intermediates through the
// caller's scratch buffer):
//   1. chunk_cumsum   dt <- clamp(softplus(dt + bias)), dA_cum <- cumsum_Q(dt A)
//   2. chunk_state    S_c[p,n] = sum_k x[k,p] B[k,n] exp(min(dA_last - dA_k, 0)) dt_k
//   3. state_passing  H_{c+1} = exp(dA_last_c) H_c + S_c, slot c rewritten with H_c
//   4. chunk_cb       CB[m,k] = C_m . B_k   (lower block triangle)
//   5. chunk_scan     y_m = exp(dA_m) C_m.H_c + sum_{k<=m} CB[m,k] exp(min(dA_m - dA_k,0)) dt_k x_k + D x_m,
//                     then y_m * silu(z_m)
// The contractions, stages 2, 4 and 5, are ssd_split.cu's; for bf16/fp16 of the shape that most layers have ssd_tc.cu replaces stages 2 to 5.
#include <algorithm>

#include "ssd_common.cuh"

namespace mb200 {
namespace {

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
    pdl_trigger();
    pdl_wait();
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
    const bool cb_first = cb_early || (has_local && has_out && !tc_out);       // formed beside the chunk states
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
    auto state_passing = [&](const mb200_ssd_args &p, bool write_prev, void *to16) {
        if (PN % 4 == 0)
            launch_dependent(ssd_state_passing_kernel<4>, dim3((unsigned)((PN / 4 + 255) / 256), a.nheads, a.batch), 256, 0, stream, p, dAb, states, nc, write_prev, to16);
        else
            launch_dependent(ssd_state_passing_kernel<1>, dim3((unsigned)((PN + 255) / 256), a.nheads, a.batch), 256, 0, stream, p, dAb, states, nc, write_prev, to16);
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
        if (!tc_loc || cb_first)
            if (int rc = ssd_split_first(a, lay, !tc_loc, cb_first, stream)) return rc;
        if (fused_states) {
            if (int rc = ssd_tc_state_stream(a, lay, stream)) return rc;
        } else if (tc_loc) {
            if (int rc = ssd_tc_chunk_state(a, lay, stream)) return rc;
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
            if (!cb_ready && !cb_first)
                if (int rc = ssd_split_first(a, lay, false, true, stream)) return rc;
            if (int rc = ssd_split_scan(a, lay, stream)) return rc;
            if (varlen)
                if (int rc = ssd_split_varlen(a, lay, SsdStates::pn32, stream)) return rc;
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
