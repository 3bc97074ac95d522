// Shared definitions of the SSD (Mamba-2) chunked forward: scratch layout and stage entry points.
#pragma once

#include "common.cuh"

namespace mb200 {

constexpr int kTcChunk = 256;     // chunk length of the tensor-core stages

// Shapes and dtypes the tensor-core stages can take (pointers and strides decide the rest).
bool ssd_tc_shape(const mb200_ssd_args &a);

// Scratch the SSD stages hand to each other (fp32 unless said otherwise, each region 256-byte aligned):
//   dt      (batch, nheads, nchunks, Q)        dt after bias/softplus/clamp, 0 past seqlen
//   dA_cum  (batch, nheads, nchunks, Q)        inclusive cumsum of dt*A inside each chunk
//   states  (batch, nchunks, nheads, P, N)     chunk states; the inter-chunk recurrence then
//                                              overwrites slot c with the state ENTERING chunk c
//   cb      (batch, nchunks, ngroups, Q, Q)    C.B^T per chunk (lower block triangle only) of the general stages
//   prev16  (batch, nchunks, nheads, P, N)     16-bit copy of the state entering each chunk (tensor-core path); [n][p]
//                                              tiles when the fused state-stream kernel wrote it
//   aux     sequence-split hand-over of the fused state-stream path, written by the LOCAL phase for the OUTPUT
//           phase: prefix decay (batch, nheads, nchunks), the range's end state from a zero incoming state
//           (batch, nheads, P, N) and the range decay (batch, nheads)
//   seq     packed sequences on the tensor-core path: for every position the offset inside its chunk at which its
//           sequence starts (batch, nchunks, Q) uint8, and per chunk whether its first position continues the
//           sequence that ended the previous chunk (batch, nchunks) uint8
//   status  one int32 in the last 256 bytes    0 after a clean run; a kernel that gave up a bounded wait
//                                              leaves its code here (the output is then invalid)
struct SsdScratch {
    size_t off_dt, off_dA, off_states, off_cb, off_prev16, off_aux, off_aux_state, off_aux_decay, off_seq_start, off_seq_carry, off_status, total;
    int nchunks;
};

inline size_t align256(size_t v) { return (v + 255) & ~size_t(255); }

inline SsdScratch ssd_scratch_layout(const mb200_ssd_args &a)
{
    SsdScratch s;
    const int Q = a.chunk_size;
    s.nchunks = (a.seqlen + Q - 1) / Q;
    const size_t bc = (size_t)a.batch * s.nchunks;
    const size_t per = (size_t)a.batch * a.nheads * s.nchunks * Q * sizeof(float);
    s.off_dt = 0;
    s.off_dA = align256(s.off_dt + per);
    s.off_states = align256(s.off_dA + per);
    s.off_cb = align256(s.off_states + bc * a.nheads * a.headdim * a.dstate * sizeof(float));
    s.off_prev16 = align256(s.off_cb + bc * a.ngroups * Q * Q * sizeof(float));
    s.off_aux = align256(s.off_prev16 + (ssd_tc_shape(a) ? bc * a.nheads * a.headdim * a.dstate * 2 : 0));
    s.off_aux_state = align256(s.off_aux + (size_t)a.batch * a.nheads * s.nchunks * sizeof(float));
    s.off_aux_decay = align256(s.off_aux_state + (size_t)a.batch * a.nheads * a.headdim * a.dstate * sizeof(float));
    s.off_seq_start = align256(s.off_aux_decay + (size_t)a.batch * a.nheads * sizeof(float));
    s.off_seq_carry = align256(s.off_seq_start + bc * Q);
    s.off_status = align256(s.off_seq_carry + bc);
    s.total = s.off_status + 256;
    return s;
}

// The status word of a call: the caller's own if it gave one, else the one in the scratch.
inline int *ssd_status_word(const mb200_ssd_args &a, const SsdScratch &lay)
{
    return a.status ? reinterpret_cast<int *>(a.status) : reinterpret_cast<int *>(static_cast<char *>(a.scratch) + lay.off_status);
}

// Tensor-core stages (ssd_tc.cu): whether the call qualifies, and the launches.  The LOCAL stages read
// x, B and dt only; the OUTPUT stage adds C, z and out.  Each predicate looks at nothing else, so the two halves
// of a sequence split agree on how the LOCAL half ran although they are handed different C / z / out.
bool ssd_tc_local_eligible(const mb200_ssd_args &a);
bool ssd_tc_output_eligible(const mb200_ssd_args &a);
bool ssd_tc_cb_eligible(const mb200_ssd_args &a);      // C as the output kernel needs it
int ssd_tc_chunk_state(const mb200_ssd_args &a, const SsdScratch &lay, cudaStream_t stream);
// Chunk states and inter-chunk recurrence fused (one CTA per batch row and head); leaves the 16-bit entering
// states in [n][p] order, which the output and varlen launches are told through states_np.
bool ssd_tc_stream_eligible(const mb200_ssd_args &a);
int ssd_tc_state_stream(const mb200_ssd_args &a, const SsdScratch &lay, cudaStream_t stream);
int ssd_tc_output(const mb200_ssd_args &a, const SsdScratch &lay, bool states_np, cudaStream_t stream);
int ssd_tc_varlen(const mb200_ssd_args &a, const SsdScratch &lay, bool states_np, cudaStream_t stream);      // bf16 only
// OUTPUT phase of a sequence split on that path: adds the incoming state's share to the entering states the LOCAL
// phase left (H_c += prefix_decay_c * S_in) and forms the range's end state.
int ssd_tc_apply_incoming(const mb200_ssd_args &a, const SsdScratch &lay, cudaStream_t stream);

// The general stages (ssd_split.cu): chunk states and C.B^T, either or both; chunk outputs.  And the end states of packed sequences, from
// entering states of any form: fp32 or 16-bit in [p][n] order, or the 16-bit [n][p] tiles of the state stream.
enum class SsdStates { pn32, pn16, np16 };
int ssd_split_first(const mb200_ssd_args &a, const SsdScratch &lay, bool with_states, bool with_cb, cudaStream_t stream);
int ssd_split_scan(const mb200_ssd_args &a, const SsdScratch &lay, cudaStream_t stream);
int ssd_split_varlen(const mb200_ssd_args &a, const SsdScratch &lay, SsdStates entering, cudaStream_t stream);

}  // namespace mb200
