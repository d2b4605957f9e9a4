// What the gather kernels of the commutator (commutator_122 by pair groups, the recoupling by orbit quadruples) need of
// the basis, for the FP64 and the mixed path alike: built once per context, on first use.
#pragma once
#include <cstdint>
#include <string>
#include <vector>

#include "comm122.h"
#include "recouple.h"

namespace imsrg {

struct GatherPlan {
  int state = 0;    // 1: ready, -1: the basis exceeds the kernels' index ranges (why)
  std::string why;
  // commutator_122 by pair-group sub-blocks (comm122.cu): the plan, its launch order for the current caps and its
  // device copies (tasks and runs sized for all tasks)
  G122Plan g122;
  G122Task* d_tasks = nullptr;
  int2* d_items = nullptr;
  const unsigned* d_codes = nullptr;
  int* d_counter = nullptr;   // the work counter, then the flag of k_check_mirror
  PairGroupsDev groups{};
  int nspb = 0;
  int per_sm[2] = {1, 1};     // resident CTAs of the FP32 and the FP64 kernel per SM
  double2* fb = nullptr;      // (fL, fR)(x, y) on every (l, j, tz) block (float2 in the mixed path)
  // orbit quadruples (i <= j, k <= l) of the particle-hole recoupling, and the column offset of every pair and J'
  std::vector<uint64_t> quads;
  const uint64_t* d_quads = nullptr;
  const int* d_xcol = nullptr;
  void* d_mem = nullptr;
  int num_sms = 1;
};

}  // namespace imsrg
