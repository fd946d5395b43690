// Host-side helpers shared by the launchers: error codes of the C ABI, the
// tensor-map factory for [B, S, H, D] operands, and small shape utilities.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/rfa_b200.h"
#include "../../include/rfa_b200_debug.h"

namespace rfa {

// Per-device launcher state (function attributes, scratch addresses) is kept in arrays of this size.
constexpr int kMaxDevices = 64;

inline int round_up(int x, int m) { return (x + m - 1) / m * m; }
inline int ceil_div(int x, int m) { return (x + m - 1) / m; }

// Padded head dimension the kernels are instantiated for (64, 128 or 256), or 0.
inline int padded_head_dim(int d) {
  if (d <= 0 || d > 256 || (d % 8) != 0) return 0;
  if (d <= 64) return 64;
  if (d <= 128) return 128;
  return 256;
}

// Builds a 4-D tensor map over a contiguous [B, S, H, D] tensor of 16-bit
// elements.  The box is {64 elements of D, 1 head, box_rows rows of S, 1 batch}
// with the 128-byte swizzle; out-of-range elements read as zero, which is what
// pads ragged sequence tails and head dimensions below the padded size.
int make_tmap_bshd(CUtensorMap* out, const void* base, int dtype, int B, int S, int H, int D, int box_rows);

// Diagnostic event trace requested through rfa_debug_set_trace (null buffer = off).
struct TraceCfg {
  unsigned long long* buf;
  int ctas;
  int cap;
};
extern TraceCfg g_trace;
constexpr int kTraceRoles = 5;

// Buffers the backward's first kernel clears (16-byte aligned, sizes multiples of 16 bytes).
struct ClearList {
  uint4* ptr[3] = {nullptr, nullptr, nullptr};
  size_t n16[3] = {0, 0, 0};
  int n = 0;
  void add(void* p, size_t bytes) {
    ptr[n] = static_cast<uint4*>(p);
    n16[n] = bytes / 16;
    ++n;
  }
};
// delta and lse2 from out, dout, lse; clears the listed buffers.
int launch_bwd_prepare(const void* out, const void* dout, const float* lse, float* delta, float* lse2, int B, int Sq,
                       int Hq, int D, int dtype, const ClearList& clear, cudaStream_t stream);
// dq from its fp32 accumulator and, where dkdv (fp32 [2][B,Skv,Hkv,D]) is given, dk and dv from it, in one launch.
int launch_bwd_finish(const float* dq_acc, void* dq, const float* dkdv, void* dk, void* dv, int B, int Sq, int Skv, int Hq,
                      int Hkv, int D, int dtype, cudaStream_t stream);

// Translates a CUDA runtime error into an ABI error code (and clears it).
inline int cuda_status(cudaError_t e) {
  if (e == cudaSuccess) return RFA_OK;
  cudaGetLastError();
  return RFA_ERR_CUDA;
}

// Launches a kernel whose blocks may start while the previous kernel of the stream drains.  Such a kernel calls
// pdl_wait() before it touches global memory, so that what it reads is complete and what it overwrites is no longer
// read; what comes before (barriers, tensor memory, descriptors) overlaps the predecessor's tail.
template <typename... P, typename... A>
inline int launch_chained(void (*kern)(P...), unsigned grid, unsigned threads, size_t smem, cudaStream_t stream,
                          const A&... args) {
  cudaLaunchAttribute attr[1] = {};
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cuda_status(cudaLaunchKernelEx(&cfg, kern, P(args)...));
}

}  // namespace rfa
