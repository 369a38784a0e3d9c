// small_api.h -- host interface of the resident sweep of small dense
// instances.
#pragma once
#include <cuda_runtime.h>

#include "../../include/pysa_gb.h"

namespace pysa_gb {

// Widest instance of the resident small sweep: two positions per lane.
constexpr int kSmallMaxN = 64;

struct SmallArgs {
  pysa_gb_problems p;
  pysa_gb_state s;
  float* fields;
  int32_t field_ld;
  // set by launch_small: this launch's reads have above < R <= cap replicas,
  // taken by `warps` warps of a CTA
  int32_t above, cap, warps;
  uint64_t seed;
  int32_t num_sweeps;
  int32_t use_pt;
  int32_t exchange_every;
  int32_t log_omega_stride;
  int32_t advance;           // 1: this launch advances the sweep counter
  const int32_t* skip_inst;  // [num_instances] 1 = swept elsewhere; or null
};

// num_sweeps sweeps, each with its exchange and log-omega, of every read of
// the dense instances with at most kSmallMaxN spins (the others are left
// alone): one CTA per read.  sms: SMs of the device.
cudaError_t launch_small(SmallArgs a, bool random, int sms, cudaStream_t st);

}  // namespace pysa_gb
