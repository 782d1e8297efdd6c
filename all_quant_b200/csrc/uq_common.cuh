// Shared device/host helpers of libuq_b200: the FP4 codec arithmetic, the partial-slot layout of the
// caller's scratch, and the status record that bounded waits write to.
#pragma once
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "uq_params.h"

#define UQ_DEV __device__ __forceinline__

// ---- programmatic dependent launch ------------------------------------------------------------------
// The append, rotate, tensor-core verify and (behind that) combine kernels are launched as programmatic dependents of what precedes
// them on the stream: their blocks may be set up while that kernel's last blocks still run.  uq_pdl_wait() returns once everything
// before it on the stream has completed with its writes visible; every block of every such kernel executes it (a grid whose
// blocks left without it could complete before its predecessor, and the kernel after it would start too early), and none
// touches global memory before it.  uq_pdl_release() lets the next kernel be set up as soon as all blocks of this one have
// executed it (or left); the kernels execute it only when they are launched as dependents themselves, so that with the switch
// below off a launch is an ordinary one for its neighbours on both sides.
UQ_DEV void uq_pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// The wait, and the thread's index as a value that exists only from there on.  Loads through const __restrict__ pointers and __ldg are
// loads of memory that does not change while the kernel runs, which the compiler may move upwards across the wait; with an address
// made of this index there is nothing to load from before it.
UQ_DEV unsigned uq_pdl_wait_index() {
  unsigned t = threadIdx.x;
  asm volatile("griddepcontrol.wait;" : "+r"(t)::"memory");
  return t;
}
UQ_DEV void uq_pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// UQ_B200_CFG="pdl=0" (read at the first launch) makes every launch of the library an ordinary one.
inline bool uq_pdl_on() {
  static const bool on = !(std::getenv("UQ_B200_CFG") && std::strstr(std::getenv("UQ_B200_CFG"), "pdl=0"));
  return on;
}
template <typename... P, typename... A>
inline cudaError_t uq_launch(void (*kern)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t s, bool dependent, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = dependent ? 1 : 0;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
  if (e != cudaSuccess) cudaGetLastError();   // the caller gets it as a value; left behind, it would be the next launch check's
  return e;
}

// ---- what the host adds to UQParams for one launch -------------------------------------------------
struct UQLaunch {
  const int32_t* pos_offset;  // [B] global position of shard-local key 0 (nullptr = 0)
  const int32_t* tree_mask;   // [B, K] draft-visibility bitmasks of a tree-masked verify (nullptr = chain: draft j sees drafts 0..j)
  int ns_eff;                 // partial slots actually used per (sequence, kv head): <= p.nsplit
  int G;                      // Hq / Hkv
  int rows;                   // query rows per work item: per * G (K * G with one chunk)
  int BM;                     // row stride of the scratch (uq_block_m)
  float sc2;                  // sm_scale * log2(e) (times k_ts for an NVFP4 cache): scores live in the exp2 domain
  float out_scale;            // multiplies the normalised output: 1, or v_ts for an NVFP4 cache
  // A call with more query rows than the tensor-core kernel's tile takes (K * G > 64): the drafts of every (sequence, kv head)
  // are cut into `chunks` runs of `per` consecutive drafts, each a work item of its own on the whole sequence, with rows
  // chunk * per * G .. of the partial slots.  One chunk of K drafts otherwise.
  int chunks, per;
  int pdl;                    // launch the kernels as programmatic dependents of what precedes them on the stream
  unsigned int* status;       // this device's status record (4 words), see uq_report
  int expire_id;              // 0, or (for the test of the give-up path) 30: the softmax role never announces the query tile of a
                              // segment, so the wait on barrier 30 runs out after its full limit on an otherwise healthy kernel
};

// ---- where the combine of a context shard sends its packed partial (context split over peer memory) ----------------
// Every rank owns one exchange buffer, mapped on every other rank: [2 parities][world slots][slot_floats] floats, then
// [2][kMaxPeers] flag words, then one counter word.  A call with sequence number seq uses parity seq & 1: rank r stores its
// partial (o [rows, D], then lse2 [rows]) into slot r of every rank's buffer and then sets flag[parity][r] = seq there.
constexpr int kMaxPeers = 8;
struct UQPeerPush {
  float* slot[kMaxPeers];          // this rank's slot in every rank's buffer, parity applied (slot[rank] is the local one)
  unsigned int* flag[kMaxPeers];   // this rank's flag word in every rank's buffer, parity applied
  unsigned int* counter;           // local word counting the combine's finished blocks (zero between calls)
  size_t rows_total;               // rows of the call: the lse2 values follow rows_total * D floats of o
  int world;
  unsigned int seq;
};
__host__ __device__ inline size_t uq_peer_slot_floats(size_t rows, int D) { return (rows * (size_t)(D + 1) + 3) / 4 * 4; }
__host__ __device__ inline size_t uq_peer_data_bytes(int world, size_t slot_floats) { return ((size_t)2 * world * slot_floats * sizeof(float) + 255) / 256 * 256; }
__host__ __device__ inline size_t uq_peer_total_bytes(int world, size_t slot_floats) { return uq_peer_data_bytes(world, slot_floats) + 2 * kMaxPeers * sizeof(unsigned int) + 64; }

// Scratch slot (b, hk, s): rows are r = j * G + g (draft j, head g of the group), row stride BM.
UQ_DEV size_t uq_slot(const UQParams& p, int b, int hk, int s) { return ((size_t)b * p.HKV + hk) * p.nsplit + s; }

// The row of q / out that belongs to (sequence b, draft j).
UQ_DEV size_t uq_draft_row(const UQParams& p, int b, int j) { return (size_t)b * p.K + j; }

// Keys of sequence b held by this cache (whole context, or one shard of it).
UQ_DEV int uq_n_local(const UQParams& p, const UQLaunch& x, int b, int* off_out) {
  const int n = p.seq_lens[b];
  const int off = x.pos_offset ? x.pos_offset[b] : 0;
  *off_out = off;
  long long cap = (long long)p.max_pages * p.PAGE;
  long long nl = (long long)n - off;
  nl = nl < 0 ? 0 : (nl > cap ? cap : nl);
  return (int)nl;
}

// Does query (draft) j of sequence b see draft token t (the key at global position seq_len - K + t)?  Chain: t <= j.
// Tree (reference uqmt/tree.py:9-12): bit t of tree_mask[b, j].
UQ_DEV bool uq_sees_draft(const UQParams& p, const UQLaunch& x, int b, int j, int t) {
  return x.tree_mask ? ((static_cast<unsigned>(__ldg(x.tree_mask + (size_t)b * p.K + j)) >> t) & 1u) != 0u : t <= j;
}

// ---- status record ------------------------------------------------------------------------------------
// [0] code (0 none, 1 barrier wait ran out), [1] block, [2] barrier id, [3] tile.  First writer wins.
UQ_DEV void uq_report(unsigned int* status, unsigned code, unsigned bar, unsigned tile) {
  if (atomicCAS(&status[0], 0u, code) == 0u) {
    status[1] = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
    status[2] = bar;
    status[3] = tile;
  }
}

// ---- codec ------------------------------------------------------------------------------------------
// UE8M0 byte -> fp32 2^(s-127).  s = 0 gives the denormal 2^-127; s = 255 gives 2^128 = +inf in fp32
// (the reference's torch.exp2 does the same).
UQ_DEV float uq_scale_f32(unsigned s) {
  return s == 0 ? __int_as_float(0x00400000) : (s == 255 ? __int_as_float(0x7f800000) : __int_as_float((int)(s << 23)));
}

// NVFP4 block scale: e4m3fn byte -> fp32 (reference uqmt/quant.py:139-147 reads it with torch's float8_e4m3fn -> float).
// The low seven bits moved up by seven are an fp16 with the same mantissa and an exponent bias of 15 instead of 7, so one
// conversion and a multiply by 2^8 give the value, subnormals included; 0x7f / 0xff are the format's NaN.
UQ_DEV float uq_e4m3_f32(unsigned b) {
  const float v = __half2float(__ushort_as_half((unsigned short)(((b & 0x80u) << 8) | ((b & 0x7fu) << 7)))) * 256.f;
  return (b & 0x7fu) == 0x7fu ? __int_as_float(0x7fc00000) : v;
}

// e2m1 nibble -> exact fp32 value: (sign | code3 << 22) read as fp32 is value * 2^-126 (a denormal for
// 0.5, zero for 0), and one multiply by 2^126 normalises it without rounding.
UQ_DEV float uq_e2m1_f32(unsigned nib) {
  return __int_as_float((int)(((nib & 8u) << 28) | ((nib & 7u) << 22))) * 8.507059173023462e37f;
}
