// Host interface of the NVRTC specialization of k_step (aq_jit.cu).
#pragma once

#include <cuda_runtime.h>

#include <string>

#include "../../include/aq.h"
#include "aq_step_config.h"

namespace aq {

bool jit_available();
// Compile (or fetch from the in-process cache) k_step<D, HF, HM, R, JitLayout,
// col, sparse> for layout L; returns a CUfunction, or null with *err set.
void* jit_k_step(int D, bool HF, bool HM, bool f64, bool col, bool sparse, const aq_layout& L, std::string* err);
std::string jit_layout_source(const aq_layout& L, int min_blocks);

// Whether the layout-specialized k_step keeps a record's words in registers
// rather than in a shared-memory slot per thread: short records, and records
// of unquantized values of any length, whose words are the values themselves
// and so take no registers of their own (3D FP32 state, 262,144 particles:
// 3.9 % faster than with slots; FP64 state, with the budget below, 19 %).
constexpr int kJitRegRecordMaxWords = 8;
inline bool jit_raw_record(const aq_layout& L) {
  for (int i = 0; i < L.n_slots; ++i)
    if (L.slot[i].kind != AQ_RAW_F32 && L.slot[i].kind != AQ_RAW_F64 && L.slot[i].kind != AQ_INT) return false;
  return true;
}
inline bool jit_reg_record(const aq_layout& L) { return L.n_words <= kJitRegRecordMaxWords || jit_raw_record(L); }
// CTAs per SM k_step's registers are budgeted for: short records 11 CTAs in 3D
// (254 us a substep of 2,097,152 quantized particles at rest, 261 with 12, 262
// with 13: of the bench layout ptxas still makes 80 registers, with fewer
// spills, and 12 CTAs fit) and 14 in 2D (73 registers; 300,000: 936 -> 829 us
// against 12), long ones 9 (113; 262,144 to 1,200,000 FP32 particles: +1.5 to
// -4 % against 8).
inline int jit_min_blocks(const aq_layout& L, int D) {
  if (L.n_words > kJitRegRecordMaxWords) return 576 / AQ_CH;
  return D == 2 ? 896 / AQ_CH : 704 / AQ_CH;
}
int jit_set_smem(void* fn, int bytes);
int jit_occupancy(void* fn, int block, size_t smem, int* out);
// launched while the kernel before it in the stream ends (the kernel waits, kernel_begin)
int jit_launch(void* fn, unsigned grid, unsigned block, size_t smem, cudaStream_t st, void** args);

}  // namespace aq
