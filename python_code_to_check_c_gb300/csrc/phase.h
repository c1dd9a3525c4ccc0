// One kernel for a whole program phase (phase.cu).
#pragma once

#include <vector>

#include "engine.h"

namespace tdcc {

// The ops of one phase of a small FP64 program as one cooperative launch: the
// op records in device memory, grouped in levels of independent ops.
class PhaseKernel {
 public:
  // Builds the records (device allocation: not during a stream capture).
  // Leaves ok false where the phase does not qualify.
  void build(const Program& p, Program::Phase ph, std::vector<void*>& owned, long long& bytes);
  bool ok = false;
  // `blocks`: at most this many thread blocks (several phases may run at once)
  cudaError_t launch(const std::vector<void*>& bases, int blocks, cudaStream_t st) const;
  int* error_flag() const { return err_; }
  int wait = 0;  // polls of the grid barrier (0: the kernel's limit; negative: none, for tests)

 private:
  void* ops_ = nullptr;
  int* tab_ = nullptr;
  unsigned* bar_ = nullptr;
  int* err_ = nullptr;
  const void* outs_ = nullptr;
  int nops_ = 0, nlevels_ = 0, nslots_ = 0, widest_ = 0, nouts_ = 0;
  size_t smem_ = 0;
};

}  // namespace tdcc
