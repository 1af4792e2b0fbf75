// context.h -- the hbx_ctx of the C ABI (device, stream, memory pool).
#pragma once

#include <cuda_runtime.h>

#include <string>

#include "../../include/hbx.h"

struct hbx_ctx {
  int device = 0;
  int n_sm = 0;
  size_t smem_optin = 0;
  size_t smem_per_sm = 0;  // shared memory of one SM (all resident blocks)
  cudaStream_t stream = nullptr;
  cudaMemPool_t pool = nullptr;  // device memory of this context's sessions and servers
  hbx_opts opts{};
  std::string err;
  std::string device_name;  // keys the autotuner's cache
  // its sessions are windows under a memory budget: one dictionary at a time
  bool windows = false;
  bool sampled_on_device = false;  // the last streamed call's planner sample
  uint64_t window_peak = 0;  // most device memory a window of the last streamed call took
  void* h_ctr = nullptr;    // page-locked counters of the context's session runs
  void* h_few = nullptr;    // page-locked pairs of small one-shot results (on first use)
  // page-locked staging of larger ones: two chunks of h_out_chunk bytes, each
  // with the event of its device-to-host copy (as large as a result needed)
  void* h_out = nullptr;
  size_t h_out_chunk = 0;
  cudaEvent_t h_out_ev[2] = {nullptr, nullptr};
};
