// Launch parameters of the backward hop kernel and the split of K/V tiles over CTAs that evens out the grid.
#pragma once

#include <cuda_runtime.h>

#include "common.h"

namespace rfa {

struct BwdParams {
  const void* k;  // for head dim 256, where K is also copied into tensor memory
  const float* lse2;
  const float* delta;
  float* dq_acc;
  const float* dkdv_prev;
  float* dkdv_out;
  void* dk16;  // with these given and nothing to add (no split, no partial sums): dK, dV in the input dtype instead of
  void* dv16;  // the fp32 buffer, [B, Skv, Hkv, D] each
  int B, Sq, Skv, Hq, Hkv, D;
  int Spad;
  float scale, scale_log2;
  int accumulate_prev, causal;
  int q_begin;  // window (zigzag layout): only query rows >= q_begin contribute
  int kv_len;   // only keys < kv_len are processed; dK/dV rows beyond keep the previous partial sums (or zero)
  int nsplit;      // CTAs per (kv tile, kv head): each takes an equal run of the group's query tiles
  int reduce_out;  // 1: the epilogue adds into dkdv_out with vector reductions (nsplit > 1); 0: plain stores
  int* dq_order;   // ordered (bit-reproducible) dQ reductions: per-tile counters, cleared by the launcher; null = unordered
  int* status;
  unsigned long long* trace;
  int trace_ctas, trace_cap;
};

int bwd_check_args(const void* q, const void* k, const void* v, const void* dout, const float* lse2,
                   const float* delta, const float* dkdv_prev, const float* dkdv_out, int B, int Sq, int Skv, int Hq,
                   int Hkv, int D, int dtype, float softmax_scale, int accumulate_prev, int causal_diag, int q_begin,
                   int kv_len, const int* status);

// Work units are CTAs, one per SM at a time; a CTA costs its query tiles plus a fixed share (prologue, filling and
// draining the pipeline, epilogue: about kCtaOverhead tiles).  A grid that leaves SMs idle (fewer K/V tiles than SMs, a
// nearly empty last wave, a diagonal block whose first K/V tiles see most of the queries) is evened out by giving each
// K/V tile to several CTAs, whose partial dK/dV are added with vector reductions into a prepared buffer.
// Picks the split with the shortest estimated makespan, a larger one only for a gain of 5 %; runs shorter than three
// tiles cost more in reductions than they save (S = 256, 8 heads of 64: 14.3 us unsplit, 15.3 us in two).
// Measured, hop alone with the clearing of its buffer, unsplit / chosen (chosen split; neighbours), us:
//   S 2048, 32/8 heads of 128, diagonal 161 / 99 (2; 3: 114), full 179 (1; 2: 197);  16/2 heads, diagonal 291 / 60 (7; 6: 65,
//   8: 60), full 294 / 92 (4; 3: 114, 8: 99);  B 2, S 1500, 16/4 heads of 96, diagonal 120 / 64 (3; 2: 67, 4: 74), full
//   118 / 95 (3; 2: 128, 4: 113);  S 1024, 32 heads of 128, diagonal / full 45 / 63 (1; 2: 72 / 88).
// Two runs may be as short as two tiles, which gains up to 5 % at head dim 64 and 5 to 16 % above (unsplit / in two, us, full:
// S 512, 8 heads of 128 21.5 / 18.5, of 64 15.2 / 14.4, 16 heads of 128 21.7 / 20.5; S 256, 16/8 heads of 128 21.2 / 18.5, 8 heads
// of 256 20.8 / 18.5; S 128, 32/8 heads of 128 21.1 / 18.5; B 2, S 250, 4 heads of 160 20.1 / 17.7; S 600, 8 heads 23.8 / 20.5).
// An overhead of 2 or 3 tiles instead of 2.5 gains 7 % in places and loses as much in others (3: S 4096, 32/4 heads, diagonal
// 404 -> 385 us, B 2, S 1500, 16/4 heads of 96 65.8 -> 70.6).
// Without head groups (MHA) dK and dV keep the same bits from call to call, ordered mode or not: two runs may be added to
// the cleared buffer in either order, three, or two and the previous partial sums, may not.  This matters below some four
// heads (hop alone, any split / at most two: S 8192, 1 head of 128, diagonal 59 / 86 us; S 4096, 1 head of 64, diagonal / full
// 24.6, 26.7 / 39.4, 41.0; S 2048, 4 heads of 128 34.8, 34.8 / 32.8, 34.9), where the host takes longer than the kernels.
inline void choose_split(BwdParams& pr, long long base_units, int bq) {
  constexpr int kSMs = 148;
  constexpr double kCtaOverhead = 2.5;
  constexpr double kSplitGain = 0.95;
  constexpr int kMaxSplit = 16;
  constexpr int kMinRun = 3;
  const int G = pr.Hq / pr.Hkv;
  const int n_q = ceil_div(pr.Sq, bq);
  const int n_kv = ceil_div(pr.kv_len, 128);
  const double heaviest = static_cast<double>(G) * (n_q - pr.q_begin / bq);  // query tiles of the first K/V tile
  double mean = heaviest;                                                     // of all of them
  if (pr.causal) {
    double sum = 0;
    const int step = 128 / bq;
    for (int k = 0; k < n_kv; ++k) {
      const int first = k * step > pr.q_begin / bq ? k * step : pr.q_begin / bq;
      sum += n_q - first;
    }
    mean = G * sum / n_kv;
  }
  // the ordered mode has counters for as many K/V tiles as there are query tiles of 128 rows
  const bool may_split = pr.dq_order == nullptr ||
                         static_cast<long long>(pr.Hkv) * n_kv <= static_cast<long long>(pr.Hq) * ceil_div(pr.Sq, 128);
  const int max_split = !may_split ? 1 : (G > 1 || pr.dq_order != nullptr) ? kMaxSplit : pr.accumulate_prev ? 1 : 2;
  int best = 1;
  double best_t = 0;
  for (int ns = 1; ns <= max_split && (ns == 1 || heaviest >= (ns == 2 ? 2 : kMinRun) * ns); ++ns) {
    const double n = static_cast<double>(base_units) * ns;
    const double longest = heaviest / ns + kCtaOverhead;
    double t;
    if (n <= kSMs) t = longest;
    else if (!pr.causal) t = static_cast<double>((static_cast<long long>(n) + kSMs - 1) / kSMs) * longest;
    else {
      // heaviest first, so the tail is made of short CTAs: the mean load, plus half a short CTA
      const double load = (mean / ns + kCtaOverhead) * n / kSMs + kCtaOverhead;
      t = load > longest ? load : longest;
    }
    if (ns == 1 || t < best_t * kSplitGain) { best = ns; best_t = t; }
  }
  pr.nsplit = best;
  pr.reduce_out = best > 1 ? 1 : 0;
}

// Brings dkdv_out into the state the kernel expects where it adds into the buffer or leaves rows of it alone.
inline int prepare_dkdv(const BwdParams& pr, cudaStream_t stream) {
  // Rows of dkdv_out that the kernel does not write (keys beyond kv_len) must still hold prev (or zero): prepare the
  // whole buffer in that case too.
  const bool partial_rows = pr.kv_len < pr.Skv;
  if (pr.reduce_out || (partial_rows && (!pr.accumulate_prev || pr.dkdv_prev != pr.dkdv_out))) {
    const size_t bytes = static_cast<size_t>(2) * pr.B * pr.Skv * pr.Hkv * pr.D * sizeof(float);
    cudaError_t e = cudaSuccess;
    if (pr.accumulate_prev) {
      if (pr.dkdv_prev != pr.dkdv_out) e = cudaMemcpyAsync(pr.dkdv_out, pr.dkdv_prev, bytes, cudaMemcpyDeviceToDevice, stream);
    } else {
      e = cudaMemsetAsync(pr.dkdv_out, 0, bytes, stream);
    }
    if (e != cudaSuccess) { cudaGetLastError(); return RFA_ERR_CUDA; }
  }
  return RFA_OK;
}

}  // namespace rfa
