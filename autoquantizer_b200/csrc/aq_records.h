// Launches of the bulk record kernels (aq_records.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/aq.h"

namespace aq {

// values (n x n_slots rows, FP32 or FP64) -> contiguous records and back
cudaError_t rec_encode_rows(const aq_layout& L, const void* values, bool f64, uint64_t* words, int64_t n,
                            const int32_t* pid, uint64_t sk, const float* uf, const double* ud, cudaStream_t st);
cudaError_t rec_decode_rows(const aq_layout& L, const uint64_t* words, void* values, bool f64, int64_t n,
                            cudaStream_t st);
// values -> grouped records at positions base + i, with ids base + i
cudaError_t rec_store(const aq_layout& L, const void* values, bool f64, uint64_t* words, int32_t* ids, int64_t base,
                      int64_t n, uint64_t sk, cudaStream_t st);
// grouped record i -> values row pid[i]
cudaError_t rec_fetch(const aq_layout& L, const uint64_t* words, const int32_t* pid, void* values, bool f64, int64_t n,
                      cudaStream_t st);
// grouped record i -> contiguous record pid[i] - base; contiguous records -> grouped, same order
cudaError_t rec_ungroup(const uint64_t* in, const int32_t* pid, uint64_t* out, int64_t n, int W, int64_t base,
                        cudaStream_t st);
cudaError_t rec_group(const uint64_t* in, uint64_t* out, int64_t n, int W, cudaStream_t st);
// per-slot statistics of grouped records, added to out (n_slots x 5)
cudaError_t rec_stats(const aq_layout& L, const uint64_t* words, const int32_t* pid, const void* ref, bool ref_f64,
                      int64_t n, double* out, cudaStream_t st);

}  // namespace aq
