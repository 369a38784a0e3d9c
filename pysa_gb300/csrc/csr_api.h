// csr_api.h -- host interface of the sparse-row Metropolis sweep.
#pragma once
#include <cuda_runtime.h>

#include "../../include/pysa_gb.h"
#include "common.cuh"

namespace pysa_gb {

struct SweepItem;

// Chains per CTA of the sparse-row sweep (a lane each), and its most warps.
constexpr int kCsrChains = 32;
constexpr int kCsrWarps = 32;

struct CsrArgs {
  pysa_gb_problems p;
  pysa_gb_state s;
  int32_t* perm;  // visiting orders with their level schedules (see
                  // launch_csr_schedule); may be null in sequential order
  int32_t perm_slots;
  int32_t num_items;
  const SweepItem* items;
  uint64_t seed;
  int32_t width;  // 0: grouped rows; 4/8/16/32: fixed records
  int32_t sms;    // SMs of the device
  // set by launch_csr: instances of every schedule, 1 narrow, 2 wide ones
  int32_t pick;
  PhiloxKeys keys;  // of seed
};

// The level schedule of every sparse instance's visiting order, written into
// the high halves of its row of `perm`: the current sweep's order (random,
// after it was made) or visiting order in slot 0 (sequential: one schedule
// serves every sweep).  Without `perm`, nothing: the sweep then takes one
// quad of positions after another.
cudaError_t launch_csr_schedule(const CsrArgs& a, bool random,
                                cudaStream_t st);
// One sweep of every work item (a CTA each).
cudaError_t launch_csr(CsrArgs a, bool random, cudaStream_t st);

}  // namespace pysa_gb
