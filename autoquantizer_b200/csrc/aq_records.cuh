// Records in bulk (sm_100a): encoding, decoding and moving whole buffers
// between rows of values, contiguous records and the simulator's grouped
// storage.
//
// All of these are bound by HBM: each byte is read and written once.  One
// thread per record with rows of ns values (100 bytes at 25 slots) or W words
// touched a sector per lane and access; here a warp takes 32 records, both
// sides are moved in runs of consecutive addresses through shared memory, and
// between them a lane holds one record.  2,097,152 records of 25 slots and 7
// words, FP32 values (values -> records -> words out -> values): 770 us
// before, see the figures at the kernels.
#pragma once

#include "aq_codec.cuh"

namespace aq {

// Two warps a CTA: shared memory per warp is up to 17 KB (32 slots of FP64
// values and 32 words a record), typically 5 KB.
constexpr int REC_T = 64;

// shared memory of a warp: words [W][32], row offsets [32], values [32][ns | 1]
struct RecSmem {
  uint64_t* words;
  int64_t* row;
  void* vals;
};

__host__ __device__ __forceinline__ int rec_vals_stride(int ns) { return ns | 1; }  // odd: no bank conflicts

__host__ __device__ __forceinline__ size_t rec_smem_warp(int W, int ns, size_t vsize) {
  return sizeof(uint64_t) * 32 * (size_t)W + sizeof(int64_t) * 32 +
         ((vsize * 32 * (size_t)rec_vals_stride(ns) + 15) & ~(size_t)15);
}

__device__ __forceinline__ RecSmem rec_smem(unsigned char* base, int W, int ns, size_t vsize) {
  unsigned char* p = base + (threadIdx.x >> 5) * rec_smem_warp(W, ns, vsize);
  RecSmem s;
  s.words = reinterpret_cast<uint64_t*>(p);
  s.row = reinterpret_cast<int64_t*>(p + sizeof(uint64_t) * 32 * (size_t)W);
  s.vals = p + sizeof(uint64_t) * 32 * (size_t)W + sizeof(int64_t) * 32;
  return s;
}

// a record in words [W][32]
struct SRec {
  const uint64_t* w;
  __device__ __forceinline__ uint64_t operator[](int k) const { return w[k * 32]; }
};

// The warp walks the 32 x m elements of 32 rows in order, 32 at a time:
// (r, k) of the lane's element.
struct RowWalk {
  int r, k, m;
  __device__ __forceinline__ RowWalk(int m_) : r(0), k(threadIdx.x & 31), m(m_) { wrap(); }
  __device__ __forceinline__ void wrap() {
    while (k >= m) {
      k -= m;
      ++r;
    }
  }
  __device__ __forceinline__ void next() {
    k += 32;
    wrap();
  }
};

// grouped records [32 g, 32 g + cnt) -> words [W][32]
__device__ __forceinline__ void rec_load_group(const uint64_t* __restrict__ words, int64_t g, int cnt, int W,
                                               uint64_t* sw) {
  const int lane = threadIdx.x & 31, W2 = W & ~1;
  const uint64_t* p = words + g * 32 * (int64_t)W;
  if (lane < cnt) {
#pragma unroll 4
    for (int k = 0; k < W2; k += 2) {
      const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2*>(p + (k >> 1) * 64 + 2 * lane));
      sw[k * 32 + lane] = v.x;
      sw[(k + 1) * 32 + lane] = v.y;
    }
    if (W & 1) sw[W2 * 32 + lane] = __ldg(p + W2 * 32 + lane);
  }
}

// the lane's record of words [W][32] -> grouped record r
__device__ __forceinline__ void rec_store_grouped(const uint64_t* sw, uint64_t* __restrict__ words, int64_t r, int W) {
  const int lane = threadIdx.x & 31, W2 = W & ~1, l = (int)(r & 31);
  uint64_t* p = words + (r >> 5) * 32 * (int64_t)W;
#pragma unroll 4
  for (int k = 0; k < W2; k += 2)
    *reinterpret_cast<ulonglong2*>(p + (k >> 1) * 64 + 2 * l) =
        make_ulonglong2(sw[k * 32 + lane], sw[(k + 1) * 32 + lane]);
  if (W & 1) p[W2 * 32 + l] = sw[W2 * 32 + lane];
}

// contiguous records [i0, i0 + cnt) <-> words [W][32]
__device__ __forceinline__ void rec_load_rows(const uint64_t* __restrict__ in, int64_t i0, int cnt, int W, uint64_t* sw) {
  const uint64_t* p = in + i0 * W;
  int e = threadIdx.x & 31;
  for (RowWalk w(W); w.r < cnt; w.next(), e += 32) sw[w.k * 32 + w.r] = __ldg(p + e);
}

// Encode a lane's values (stride 1) into words [W][32]: encode_record with
// the slots in a loop over the layout in constant memory, for layouts that
// are not compile-time constants.  Same codes.
template <class T>
__device__ __forceinline__ void encode_slots(const aq_layout& L, const T* v, uint64_t* out, uint64_t pk,
                                             const float* uf, const double* ud) {
  const bool f64 = L.compute_f64 != 0;
  const bool dith = L.use_dithering != 0;
  uint32_t gmax[AQ_MAX_GROUPS];
#pragma unroll
  for (int g = 0; g < AQ_MAX_GROUPS; ++g) gmax[g] = 0;
  if (L.n_groups > 0) {
    for (int s = 0; s < L.n_slots; ++s) {
      if (L.slot[s].kind != AQ_SHARED_EXP) continue;
      const uint32_t ex = (__float_as_uint((float)v[s]) >> 23) & 0xffu;
#pragma unroll
      for (int k = 0; k < AQ_MAX_GROUPS; ++k)
        if (L.slot[s].group == k) gmax[k] = max(gmax[k], ex);
    }
  }
  uint64_t acc = 0;
  int fill = 0;
  uint64_t* o = out;
  const auto put = [&](uint64_t code, int nb) {
    acc |= code << fill;
    const int nf = fill + nb;
    if (nf >= 64) {
      *o = acc;
      o += 32;
      acc = nf > 64 ? (code >> (64 - fill)) : 0ull;
      fill = nf - 64;
    } else {
      fill = nf;
    }
  };
  for (int s = 0; s < L.n_slots; ++s) {
    const aq_slot& S = L.slot[s];
    const T x = v[s];
    switch (S.kind) {
      case AQ_FIXED: {
        uint32_t q;
        if (f64) {
          double u = 0.0;
          if (dith) u = ud ? ud[s] : uniform_f64(pk, s);
          q = quant_fixed_f64(S, dith, (double)x, u);
        } else {
          float u = 0.0f;
          if (dith) u = uf ? uf[s] : uniform_f32(pk, s);
          q = quant_fixed_f32(S, dith, (float)x, u);
        }
        put(q, S.bits);
        break;
      }
      case AQ_INT: {
        uint32_t q = S.is_signed ? (uint32_t)__double2int_rz((double)x) : __double2uint_rz((double)x);
        if (S.bits < 32) q &= (1u << S.bits) - 1u;
        put(q, S.bits);
        break;
      }
      case AQ_FLOAT_EXP: {
        uint32_t d, e;
        quant_float_exp(S, (float)x, d, e);
        put(e, S.exp_bits);
        put(d, S.bits);
        break;
      }
      case AQ_SHARED_EXP: {
        uint32_t mx = 0;
#pragma unroll
        for (int k = 0; k < AQ_MAX_GROUPS; ++k)
          if (S.group == k) mx = gmax[k];
        if (S.exp_first) put(shared_exp_code(S.exp_bits, mx), S.exp_bits);
        put(quant_shared(S, (float)x, mx), S.bits);
        break;
      }
      case AQ_RAW_F32:
        put(__float_as_uint((float)x), 32);
        break;
      default:
        put((uint64_t)__double_as_longlong((double)x), 64);
        break;
    }
  }
  if (fill > 0) *o = acc;
}

// Values (n x n_slots rows) -> records.  GROUPED: into grouped storage at
// positions base + i, ids base + i also written to ids; else contiguous, with
// the dithering keyed on pid[i] (or i) and the uniforms given or drawn.
template <class T, bool GROUPED>
__global__ void __launch_bounds__(REC_T) k_encode(const __grid_constant__ aq_layout L, const T* __restrict__ values,
                                                  uint64_t* __restrict__ words, int64_t n,
                                                  const int32_t* __restrict__ pid, int32_t* __restrict__ ids,
                                                  int64_t base, uint64_t sk, const float* __restrict__ uf,
                                                  const double* __restrict__ ud) {
  extern __shared__ __align__(16) unsigned char rec_sm[];
  const int ns = L.n_slots, W = L.n_words, lane = threadIdx.x & 31, np = rec_vals_stride(ns);
  const int64_t i0 = ((int64_t)blockIdx.x * (REC_T / 32) + (threadIdx.x >> 5)) * 32;
  if (i0 >= n) return;
  const int cnt = (int)min((int64_t)32, n - i0);
  const RecSmem sm = rec_smem(rec_sm, W, ns, sizeof(T));
  T* const sv = static_cast<T*>(sm.vals);
  {
    const T* p = values + i0 * ns;
    int e = lane;
    for (RowWalk w(ns); w.r < cnt; w.next(), e += 32) sv[w.r * np + w.k] = __ldg(p + e);
  }
  __syncwarp();
  const int64_t i = i0 + lane;
  if (lane < cnt) {
    const int32_t id = GROUPED ? (int32_t)(base + i) : pid ? pid[i] : (int32_t)i;
    encode_slots<T>(L, sv + lane * np, sm.words + lane, particle_key(sk, id), uf ? uf + i * ns : nullptr,
                    ud ? ud + i * ns : nullptr);
    if (GROUPED) {
      rec_store_grouped(sm.words, words, base + i, W);
      ids[base + i] = id;
    }
  }
  if (!GROUPED) {
    __syncwarp();
    uint64_t* p = words + i0 * W;
    int e = lane;
    for (RowWalk w(W); w.r < cnt; w.next(), e += 32) p[e] = sm.words[w.k * 32 + w.r];
  }
}

// Records -> values rows.  GROUPED: from grouped storage, record i to row
// pid[i]; else contiguous records, row i.
template <class T, bool GROUPED>
__global__ void __launch_bounds__(REC_T) k_decode(const __grid_constant__ aq_layout L,
                                                  const uint64_t* __restrict__ words, const int32_t* __restrict__ pid,
                                                  T* __restrict__ values, int64_t n) {
  extern __shared__ __align__(16) unsigned char rec_sm[];
  const int ns = L.n_slots, W = L.n_words, lane = threadIdx.x & 31, np = rec_vals_stride(ns);
  const int64_t g = (int64_t)blockIdx.x * (REC_T / 32) + (threadIdx.x >> 5);
  if (g * 32 >= n) return;
  const int cnt = (int)min((int64_t)32, n - g * 32);
  const RecSmem sm = rec_smem(rec_sm, W, ns, sizeof(T));
  T* const sv = static_cast<T*>(sm.vals);
  if (GROUPED)
    rec_load_group(words, g, cnt, W, sm.words);
  else
    rec_load_rows(words, g * 32, cnt, W, sm.words);
  sm.row[lane] = lane < cnt ? (GROUPED ? (int64_t)__ldg(pid + g * 32 + lane) : g * 32 + lane) * ns : 0;
  __syncwarp();
  if (lane < cnt)
    for (int s = 0; s < ns; ++s) sv[lane * np + s] = decode_slot<T>(L, s, SRec{sm.words + lane});
  __syncwarp();
  for (RowWalk w(ns); w.r < cnt; w.next()) values[sm.row[w.r] + w.k] = sv[w.r * np + w.k];
}

// Records from the simulator's grouped storage to contiguous records in
// particle order (record i goes to out[pid[i] - base]; base: the id of out's
// first record, a streamed chunk's first particle).
static __global__ void __launch_bounds__(REC_T) k_words_ungroup(const uint64_t* __restrict__ in,
                                                                const int32_t* __restrict__ pid,
                                                                uint64_t* __restrict__ out, int64_t n, int W,
                                                                int64_t base) {
  extern __shared__ __align__(16) unsigned char rec_sm[];
  const int lane = threadIdx.x & 31;
  const int64_t g = (int64_t)blockIdx.x * (REC_T / 32) + (threadIdx.x >> 5);
  if (g * 32 >= n) return;
  const int cnt = (int)min((int64_t)32, n - g * 32);
  const RecSmem sm = rec_smem(rec_sm, W, 0, 0);
  rec_load_group(in, g, cnt, W, sm.words);
  sm.row[lane] = lane < cnt ? ((int64_t)__ldg(pid + g * 32 + lane) - base) * W : 0;
  __syncwarp();
  for (RowWalk w(W); w.r < cnt; w.next()) out[sm.row[w.r] + w.k] = sm.words[w.k * 32 + w.r];
}

// Contiguous records (record i at in[i W]) into grouped storage, same order.
static __global__ void __launch_bounds__(REC_T) k_words_group(const uint64_t* __restrict__ in,
                                                              uint64_t* __restrict__ out, int64_t n, int W) {
  extern __shared__ __align__(16) unsigned char rec_sm[];
  const int lane = threadIdx.x & 31;
  const int64_t i0 = ((int64_t)blockIdx.x * (REC_T / 32) + (threadIdx.x >> 5)) * 32;
  if (i0 >= n) return;
  const int cnt = (int)min((int64_t)32, n - i0);
  const RecSmem sm = rec_smem(rec_sm, W, 0, 0);
  rec_load_rows(in, i0, cnt, W, sm.words);
  __syncwarp();
  if (lane < cnt) rec_store_grouped(sm.words, out, i0 + lane, W);
}

inline size_t rec_smem_cta(int W, int ns, size_t vsize) { return (REC_T / 32) * rec_smem_warp(W, ns, vsize); }

}  // namespace aq
