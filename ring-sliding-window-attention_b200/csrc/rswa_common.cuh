// Internal declarations shared by the kernels and the C-ABI layer.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/rswa.h"

namespace rswa {

constexpr int kTile = RSWA_TILE;       // rows of a query tile and of a key tile
constexpr int kHeadDim = 128;
// Heads of 64 elements have kernels of their own (the template argument kD): a tile is one TMA box instead of two,
// the products that contract over the head dimension take half as many instructions, the others are half as wide.
// Shared and tensor memory keep the 128-wide layout, half of each tile unused: neither leaves room for a second CTA
// per SM either way (the registers do not).  Training step, zero-padded to 128 by the host -> these kernels:
// 4 x 4096 tokens, 16 heads, window 512: 767 -> 342 us; 1024 tokens, 4 heads, window 128: 320 -> 91 us.
constexpr int kNarrowHeadDim = 64;
constexpr int kBoxBytes = 16384;       // one TMA box: 128 rows x 64 x 16-bit, 128-byte swizzle
constexpr int kTileBytes = 2 * kBoxBytes;
constexpr int kMaxEntries = 2 * RSWA_MAX_SPANS;

// device-side error codes written to the status word
enum : int {
  kErrWaitProducer = 101,
  kErrWaitMma = 102,
  kErrWaitSoftmax = 103,
  kErrWaitEpilogue = 104,
};

struct FwdKernelParams {
  CUtensorMap q_map;
  CUtensorMap k_map[RSWA_MAX_SPANS];
  CUtensorMap v_map[RSWA_MAX_SPANS];
  int span_pos[RSWA_MAX_SPANS];
  int span_len[RSWA_MAX_SPANS];
  int n_spans;
  int batch, q_len, hq, hkv, head_dim;
  int q_pos_start, window, n_sink;
  float scale_log2;  // softmax_scale * log2(e)
  const int* cu;
  int n_seqs;
  void* out;
  long long o_sb, o_st, o_sh;
  float* lse;
  long long l_sb, l_sh;
  int q_tile_begin, n_q_tiles;
  int carry;  // out / lse hold a partial result over other keys: continue it instead of starting over
  int* status;
  int* mirror;  // host-visible copy of the status word (or null)
};

struct BwdKernelParams {
  CUtensorMap q_map;
  CUtensorMap do_map;
  CUtensorMap k_map[RSWA_MAX_SPANS];
  CUtensorMap v_map[RSWA_MAX_SPANS];
  int span_pos[RSWA_MAX_SPANS];
  int span_len[RSWA_MAX_SPANS];
  int span_tile0[RSWA_MAX_SPANS + 1];  // prefix sum of key tiles per span
  void* dk[RSWA_MAX_SPANS];
  void* dv[RSWA_MAX_SPANS];
  long long dkv_sb[RSWA_MAX_SPANS], dkv_st[RSWA_MAX_SPANS], dkv_sh[RSWA_MAX_SPANS];
  int grad_fp32[RSWA_MAX_SPANS];
  int n_spans;
  int batch, q_len, hq, hkv, head_dim;
  int q_pos_start, window, n_sink;
  float scale_log2;
  float scale;
  const int* cu;
  int n_seqs;
  // rows prepared by the delta kernel, both [batch, hq, q_len_pad] fp32, 512-byte aligned per
  // 128-query tile and both NEGATED: -lse * log2(e) (-inf past q_len) and -delta = -rowsum(dO * O)
  // (0 past q_len)
  const float* lse2;
  const float* delta;
  long long d_sb, d_sh;
  void* dq;  // [batch, q_len, hq, 128], 16-bit, written by the dQ kernel
  int* dq_counter;   // work counter of the dQ kernel, zeroed before its launch
  int* dkv_counter;  // work counter of the dK/dV kernel, likewise
  int* gate;         // 0 until the dK/dV kernel hands what came before it on to an overlapping dQ kernel; null: no overlap
  long long dq_sb, dq_st, dq_sh;
  int* status;
  int* mirror;  // host-visible copy of the status word (or null)
  // Sink tokens are seen by every later query of their sequence.  When far_segs > 0 the dK/dV kernel treats
  // the queries beyond a sink token's window separately: the query axis is cut into far_segs segments
  // (see far_range); those that hold such queries (far_split) are work items of their own per KV head, whose dK / dV of
  // the sink rows go to far_ws as partial sums ([batch, hkv, far_segs + sequences, n_sink, 2, 128] fp32; the rows'
  // windowed part goes to the slot far_segs + sequence) and are added up by sink_sum_kernel.
  int far_segs, far_chunk, far_slots;  // far_chunk: positions per chunk, a multiple of the tile
  float* far_ws;
  int* far_list;  // number of segments that are work items, then these segments (written by begin_call)
};

// What the kernel in front of the tensor kernels needs of these (the whole struct is 3 KB of tensor maps).
struct FarParams {
  const int* cu;
  int n_seqs, q_pos_start, q_len, window, far_segs, far_chunk;
  int* far_list;
};

// Programmatic dependent launch.  The tensor kernels are launched with the attribute that lets a kernel start while
// the one before it on the stream still runs (launch_kernel below): griddep_wait() returns once every earlier
// kernel has finished and its writes are visible (at once if the kernel was launched the ordinary way),
// griddep_launch() says that the next kernel may be brought up as far as SMs are free (without it that is when
// the kernel ends: the launch itself is hidden then).  Nothing may be read from or written to global memory in
// front of griddep_wait(), with one exception: the dQ kernel, which overlaps the dK/dV kernel in front of it and needs what
// the kernels before THAT one wrote.  Starting behind its trigger promises no visibility (only griddep_wait() does, to
// the grid that waits), so the dK/dV kernel passes on what its own wait has made visible: tc05::gate_open() releases
// a word, tc05::gate_wait() acquires it.  (One load of a few hundred ns per dQ CTA, behind the barrier set-up.)
// Measured, one GPU: training step of 4096 tokens (32/4 heads, window 1000) 319 -> 290 us, prefill of 777 tokens
// 17.4 -> 15.4 us, 65536 tokens with 32/32 heads 5796 -> 5795 us.  A griddep_launch() in the forward kernel with
// an early delta kernel behind it made the large calls 1.5 to 5 % slower and gave the small ones nothing.
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// The code of an error already reported through the status word, or 0; the kernel then does no work, so as not to
// pile further time-outs on it.  The report also goes to the host-visible mirror, from where the host picks it
// up without a copy or a synchronisation.  For one thread.
__device__ __forceinline__ int status_code(const int* status, int* mirror) {
  const int code = *reinterpret_cast<const volatile int*>(status);
  if (mirror != nullptr && code != 0) *reinterpret_cast<volatile int*>(mirror) = code;
  return code;
}
__device__ __forceinline__ void raise_status(int* status, int* mirror, int code) {
  atomicCAS(status, 0, code);
  if (mirror != nullptr) *reinterpret_cast<volatile int*>(mirror) = code;
}

// Sequence [start, end) containing global position p.  cu has n_seqs + 1 entries.
// Returns its index (tokens past the last boundary form a sequence of their own, index n_seqs).
__device__ __forceinline__ int seq_of(const int* __restrict__ cu, int n_seqs, int p, int& start,
                                      int& end) {
  if (cu == nullptr) {
    start = 0;
    end = 0x7fffffff;
    return 0;
  }
  int lo = 0, hi = n_seqs;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (__ldg(cu + mid) <= p) lo = mid; else hi = mid - 1;
  }
  start = __ldg(cu + lo);
  end = (lo < n_seqs) ? __ldg(cu + lo + 1) : 0x7fffffff;
  return lo;
}

// The query axis of a call, cut at multiples of far_chunk from its first query and at sequence starts:
// segment e lies in one sequence and one chunk.  With i sequence starts and j chunk boundaries in front of
// it, e = i + j and it belongs to sequence i.  Fills the sequence's bounds and the positions [q_lo, q_hi] of the
// segment's queries that lie beyond the window of the sequence's first token (none if q_lo > q_hi).
template <typename Params>
__device__ __forceinline__ void far_range(const Params& p, int i, int j, int& s, int& e, int& q_lo, int& q_hi) {
  s = 0, e = 0x7fffffff;
  if (p.cu != nullptr) {
    s = __ldg(p.cu + i);
    if (i < p.n_seqs) e = __ldg(p.cu + i + 1);
  }
  const int q_end = p.q_pos_start + p.q_len;
  const int n_chunks = (p.q_len + p.far_chunk - 1) / p.far_chunk;
  const int a = p.q_pos_start + j * p.far_chunk;
  const int z = j + 1 < n_chunks ? a + p.far_chunk : q_end;
  q_lo = max(max(s, a), s > 0x7ffffffe - p.window ? 0x7fffffff : s + p.window + 1);
  q_hi = min(e, z) - 1;
}
// Whether the sequence [s, e) is treated that way: only if the queries beyond the window of its first token are more
// than one segment.  Fewer cost the sink tokens' key tile at most as many tile products again as an ordinary one has,
// and a segment item (its loads, its partial sums) costs more: 32768 tokens in 250 sequences of 131, 32/8
// heads, window 64, 4 sink tokens: 1086 us a training step without segments, 1280 us with one for each sequence.
template <typename Params>
__device__ __forceinline__ bool far_split(const Params& p, int s, int e) {
  if (p.far_segs == 0) return false;
  const int first = s > 0x7ffffffe - p.window ? 0x7fffffff : s + p.window + 1;
  return min(e, p.q_pos_start + p.q_len) - max(first, p.q_pos_start) > p.far_chunk;
}
// number of sequence starts among the first e of the merged boundaries (starts first on ties)
template <typename Params>
__device__ __forceinline__ int far_sequence(const Params& p, int e) {
  if (p.cu == nullptr) return 0;
  const int n_b = (p.q_len + p.far_chunk - 1) / p.far_chunk - 1;  // boundary j at q_pos_start + (j + 1) * far_chunk
  int lo = max(0, e - n_b), hi = min(e, p.n_seqs);                // start i at cu[i + 1]
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(p.cu + mid + 1) <= p.q_pos_start + (e - mid) * p.far_chunk) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// Optional in-kernel timeline (development builds only, -DRSWA_TRACE): one chosen CTA stamps clock64()
// into a per-file device array that a small extern "C" reader copies out.  Compiles to nothing otherwise.
#ifdef RSWA_TRACE
#ifndef RSWA_TRACE_CTA
#define RSWA_TRACE_CTA 2000
#endif
#define RSWA_TRACE_SLOTS 2048
#define RSWA_TRACE_DECL(name)                                                                    \
  static __device__ long long g_trace_##name[RSWA_TRACE_SLOTS];                                  \
  extern "C" int rswa_trace_read_##name(long long* out) {                                         \
    return static_cast<int>(cudaMemcpyFromSymbol(out, g_trace_##name, sizeof(g_trace_##name)));  \
  }
#define RSWA_TRC(name, cond, slot)                                                               \
  do {                                                                                           \
    if (blockIdx.x == RSWA_TRACE_CTA && (cond) && (slot) < RSWA_TRACE_SLOTS) g_trace_##name[slot] = clock64(); \
  } while (0)
#else
#define RSWA_TRACE_DECL(name)
#define RSWA_TRC(name, cond, slot) do { } while (0)
#endif

// host side -------------------------------------------------------------------------------
void set_error(const char* fmt, ...);
// 4-D map over a [batch, tokens, heads, head_dim] 16-bit tensor (strides in elements), box = 64
// elements x 1 head x 128 tokens x 1 batch, 128-byte swizzle, zero fill out of bounds.
int make_tile_map(CUtensorMap* map, const void* base, int dtype, int batch, int tokens, int heads, int head_dim,
                  long long sb, long long st, long long sh);
int check_geom(const rswa_geom_t& g, bool need_grads, int head_dim = kHeadDim);
int* status_mirror(const int* status);  // the mirror registered for a status word, or null
void count_launches(int n);             // kernels of this library launched (rswa_launch_count)
int sm_count();  // SMs of the current device (cached per device)

// A launch that may start before the kernel in front of it on the stream has finished (`early`; the kernel then
// waits with griddep_wait), or an ordinary one.
template <typename... Params, typename... Args>
cudaError_t launch_kernel(void (*kern)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t stream, bool early, Args... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(static_cast<unsigned>(threads));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = early ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, static_cast<Params>(args)...);
  if (e != cudaSuccess) cudaGetLastError();  // (reported here, not by whoever asks next)
  return e;
}

}  // namespace rswa
