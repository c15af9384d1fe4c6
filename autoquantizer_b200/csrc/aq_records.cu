// Records in bulk (sm_100a): encoding, decoding and moving whole buffers
// between rows of values, contiguous records and the simulator's grouped
// storage.
//
// All of these are bound by HBM: each byte is read and written once.  One
// thread per record with rows of ns values (100 bytes at 25 slots) or W words
// touched a sector per lane and access; here a warp takes 32 records, both
// sides are moved in runs of consecutive addresses through shared memory, and
// between them a lane holds one record, with eight loads in flight a lane.
// 2,097,152 records of 25 slots and 7 words, FP32 values, then -> now:
//   values -> grouped records   361 -> 158 us  (three passes then; 50 us of traffic)
//   grouped records -> values   368 -> 118 us  (50 us)
//   grouped records -> words     62 ->  50 us  (36 us)
// What is left above the traffic is the codec's own arithmetic, some 20
// instructions a slot.
#include <algorithm>

#include "aq_codec.cuh"
#include "aq_common.cuh"
#include "aq_records.h"

namespace aq {

// Two warps a CTA: shared memory per warp is up to 17 KB (32 slots of FP64
// values and 32 words a record), typically 5 KB.  CTAs stay and take one
// group of 32 records after another.
constexpr int REC_T = 64;

// ------------------------------------------------------------ slot plans
//
// The layout is not a compile-time constant here, so what a slot costs is
// mostly what is looked up and decided for it.  A CTA first writes a plan per
// slot to shared memory, two 16-byte reads, for the common kinds (fixed point
// computed in FP32, plain FP32), and runs of four signed fixed-point slots
// go side by side; everything else, and given uniforms, takes the codec's
// general functions.  (General functions for every slot: encoding 2,097,152
// records of 25 slots 182 us, decoding them 141; copying the layout's slots
// to shared memory too: 170 and 119.)
enum { PLAN_SIGNED = 0, PLAN_UNSIGNED = 1, PLAN_F32 = 2, PLAN_OTHER = 3 };

struct __align__(16) SlotPlan {
  int kind, bits, at;         // at: first bit; kind + 8: this and the next three slots are PLAN_SIGNED
  uint32_t mask;              // low `bits` bits
  float scale, offset;        // decoding: scale, offset; encoding: 1 / scale, offset
  uint32_t ja, jc;            // encoding: the slot's draw, x = ja key + jc (draw32)
};

__device__ __forceinline__ SlotPlan slot_plan(const aq_layout& L, int s, bool enc, bool given_uf) {
  const aq_slot& S = L.slot[s];
  SlotPlan p;
  p.kind = PLAN_OTHER;
  if (S.kind == AQ_FIXED && !L.compute_f64 && !given_uf)
    p.kind = S.is_signed ? PLAN_SIGNED : enc ? PLAN_OTHER : PLAN_UNSIGNED;
  if (S.kind == AQ_RAW_F32) p.kind = PLAN_F32;
  p.bits = S.bits;
  p.at = S.bit_offset;
  p.mask = 0xffffffffu >> (32 - (S.bits <= 32 ? S.bits : 32));
  p.scale = enc ? S.inv_scale_f32 : S.scale_f32;
  p.offset = S.offset_f32;
  p.ja = kLcgJumps.a[2 * s + 1];
  p.jc = kLcgJumps.c[2 * s + 1];
  return p;
}

// ---------------------------------------------------------- shared memory
//
// Per CTA the plans; per warp the words of 32 records as 32-bit halves
// [2 W + 1][32] (the last row is read but not used), the rows' offsets [32]
// and the values [32][ns | 1].
struct RecSmem {
  SlotPlan* plan;
  const aq_slot* slot;  // the layout's own (kernel parameter)
  int* shared;  // slots with a shared exponent: [0] how many, then which
  uint32_t* words;
  int64_t* row;
  void* vals;
};

__host__ __device__ __forceinline__ int rec_vals_stride(int ns) { return ns | 1; }  // odd: no bank conflicts

__host__ __device__ __forceinline__ size_t rec_smem_warp(int W, int ns, size_t vsize) {
  return sizeof(uint32_t) * 32 * (2 * (size_t)W + 1) + sizeof(int64_t) * 32 +
         ((vsize * 32 * (size_t)rec_vals_stride(ns) + 15) & ~(size_t)15);
}

__host__ __device__ __forceinline__ size_t rec_smem_plans(int ns) {
  return sizeof(SlotPlan) * ns + ((sizeof(int) * (ns + 1) + 15) & ~(size_t)15);
}

__device__ __forceinline__ RecSmem rec_smem(const aq_layout& L, unsigned char* base, int W, int ns, size_t vsize) {
  RecSmem s;
  s.plan = reinterpret_cast<SlotPlan*>(base);
  s.slot = L.slot;
  s.shared = reinterpret_cast<int*>(base + sizeof(SlotPlan) * ns);
  unsigned char* p = base + rec_smem_plans(ns) + (threadIdx.x >> 5) * rec_smem_warp(W, ns, vsize);
  s.row = reinterpret_cast<int64_t*>(p);
  s.words = reinterpret_cast<uint32_t*>(p + sizeof(int64_t) * 32);
  s.vals = p + sizeof(int64_t) * 32 + sizeof(uint32_t) * 32 * (2 * (size_t)W + 1);
  return s;
}

// the same without plans and values
__device__ __forceinline__ RecSmem rec_smem_words(unsigned char* base, int W) {
  RecSmem s;
  unsigned char* p = base + rec_smem_plans(0) + (threadIdx.x >> 5) * rec_smem_warp(W, 0, 0);
  s.row = reinterpret_cast<int64_t*>(p);
  s.words = reinterpret_cast<uint32_t*>(p + sizeof(int64_t) * 32);
  return s;
}

// a lane's record in words [2 W + 1][32]
struct SRec {
  const uint32_t* w;
  __device__ __forceinline__ uint64_t operator[](int k) const {
    return (uint64_t)w[2 * k * 32] | (uint64_t)w[(2 * k + 1) * 32] << 32;
  }
};

// How a warp walks rows of m <= 32 elements: lane l takes element k of the
// rows r, r + step, ..., as many whole rows at a time as 32 lanes hold.
struct RowWalk {
  int r, k, step;
  __device__ __forceinline__ RowWalk(int m) {
    const int lane = threadIdx.x & 31;
    step = 32 / m;
    r = lane / m;
    k = lane - r * m;
    if (r >= step) r = 32;  // no whole row left for this lane
  }
};

// The rows' elements, eight loads in flight a lane (a plain loop waited for
// each: encoding took 309 us instead of 186).
template <class T, class F>
__device__ __forceinline__ void load_rows(const T* __restrict__ p, int m, int cnt, const RowWalk& w, const F& put) {
  for (int r0 = w.r; r0 < cnt; r0 += 8 * w.step) {
    T t[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int r = r0 + j * w.step;
      t[j] = r < cnt ? __ldg(p + r * m + w.k) : T(0);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int r = r0 + j * w.step;
      if (r < cnt) put(r, w.k, t[j]);
    }
  }
}

__device__ __forceinline__ void rec_put(uint32_t* sw, int k, uint64_t v) {
  sw[2 * k * 32] = (uint32_t)v;
  sw[(2 * k + 1) * 32] = (uint32_t)(v >> 32);
}

// grouped records [32 g, 32 g + cnt) -> words
__device__ __forceinline__ void rec_load_group(const uint64_t* __restrict__ words, int64_t g, int cnt, int W,
                                               uint32_t* sw) {
  const int lane = threadIdx.x & 31, W2 = W & ~1;
  const uint64_t* p = words + g * 32 * (int64_t)W;
  if (lane < cnt) {
    for (int k0 = 0; k0 < W2; k0 += 8) {
      ulonglong2 t[4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (k0 + 2 * j < W2) t[j] = __ldg(reinterpret_cast<const ulonglong2*>(p + ((k0 >> 1) + j) * 64 + 2 * lane));
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (k0 + 2 * j < W2) {
          rec_put(sw + lane, k0 + 2 * j, t[j].x);
          rec_put(sw + lane, k0 + 2 * j + 1, t[j].y);
        }
    }
    if (W & 1) rec_put(sw + lane, W2, __ldg(p + W2 * 32 + lane));
  }
}

// the lane's record of words -> grouped record r
__device__ __forceinline__ void rec_store_grouped(const uint32_t* sw, uint64_t* __restrict__ words, int64_t r, int W) {
  const SRec rec{sw + (threadIdx.x & 31)};
  const int W2 = W & ~1, l = (int)(r & 31);
  uint64_t* p = words + (r >> 5) * 32 * (int64_t)W;
#pragma unroll 4
  for (int k = 0; k < W2; k += 2)
    *reinterpret_cast<ulonglong2*>(p + (k >> 1) * 64 + 2 * l) = make_ulonglong2(rec[k], rec[k + 1]);
  if (W & 1) p[W2 * 32 + l] = rec[W2];
}

// contiguous records [i0, i0 + cnt) -> words
__device__ __forceinline__ void rec_load_rows(const uint64_t* __restrict__ in, int64_t i0, int cnt, int W, uint32_t* sw) {
  load_rows(in + i0 * W, W, cnt, RowWalk(W), [&](int r, int k, uint64_t v) { rec_put(sw + r, k, v); });
}

// plans of the CTA
__device__ __forceinline__ void rec_plans(const aq_layout& L, const RecSmem& sm, bool enc, bool given_uf) {
  for (int s = threadIdx.x; s < L.n_slots; s += REC_T) {
    sm.plan[s] = slot_plan(L, s, enc, given_uf);
  }
  __syncthreads();
  if ((int)threadIdx.x + 3 < L.n_slots) {
    bool run = true;
    for (int j = 0; j < 4; ++j) run = run && (sm.plan[threadIdx.x + j].kind & 7) == PLAN_SIGNED;
    __syncwarp(__activemask());
    if (run) sm.plan[threadIdx.x].kind = PLAN_SIGNED + 8;
  }
  if (threadIdx.x == 0) {
    int m = 0;
    for (int s = 0; s < L.n_slots; ++s)
      if (L.slot[s].kind == AQ_SHARED_EXP) sm.shared[1 + m++] = s;
    sm.shared[0] = m;
  }
  __syncthreads();
}

// groups of 32 of n records that this warp takes: for (g = first; g * 32 < n; g += step)
__device__ __forceinline__ int64_t rec_first_group() { return (int64_t)blockIdx.x * (REC_T / 32) + (threadIdx.x >> 5); }
__device__ __forceinline__ int64_t rec_group_step() { return (int64_t)gridDim.x * (REC_T / 32); }

// The lane's record of words -> its values v[0, ns).
template <class T>
__device__ __forceinline__ void rec_decode(const RecSmem& sm, int ns, bool f64, const uint32_t* sw, T* v) {
  // dequant_fixed of a signed slot (q * scale is never -0, so adding a zero offset is exact)
  const auto fixed = [&](const SlotPlan& p) {
    const uint32_t* w = sw + (p.at >> 5) * 32;
    const int q = (int)(__funnelshift_r(w[0], w[32], p.at & 31) << (32 - p.bits)) >> (32 - p.bits);
    return (T)__fadd_rn(__fmul_rn(__int2float_rn(q), p.scale), p.offset);
  };
  for (int s = 0; s < ns; ++s) {
    const SlotPlan p = sm.plan[s];
    if (p.kind == PLAN_SIGNED + 8) {  // four slots, their chains side by side
      const SlotPlan p1 = sm.plan[s + 1], p2 = sm.plan[s + 2], p3 = sm.plan[s + 3];
      const T a = fixed(p), b = fixed(p1), c = fixed(p2), d = fixed(p3);
      v[s] = a;
      v[s + 1] = b;
      v[s + 2] = c;
      v[s + 3] = d;
      s += 3;
    } else if (p.kind == PLAN_SIGNED) {
      v[s] = fixed(p);
    } else if (p.kind == PLAN_OTHER) {
      v[s] = decode_of<T>(sm.slot[s], f64, SRec{sw});
    } else {
      const uint32_t* w = sw + (p.at >> 5) * 32;
      const uint32_t code = __funnelshift_r(w[0], w[32], p.at & 31);  // the next 32 bits
      if (p.kind == PLAN_F32)
        v[s] = (T)__uint_as_float(code);
      else
        v[s] = (T)__fadd_rn(__fmul_rn(__uint2float_rn(code & p.mask), p.scale), p.offset);
    }
  }
}

// The lane's values v[0, ns) -> its record in words: encode_record's codes.
// pk: particle key; uf / ud: given uniforms or null.
template <class T, bool DITH>
__device__ __forceinline__ void rec_encode(const RecSmem& sm, int ns, int W, bool f64, const T* v, uint32_t* sw,
                                           uint64_t pk, const float* uf, const double* ud) {
  uint32_t gmax[AQ_MAX_GROUPS];
#pragma unroll
  for (int g = 0; g < AQ_MAX_GROUPS; ++g) gmax[g] = 0;
  const int nsh = sm.shared[0];
  for (int i = 0; i < nsh; ++i) {
    const int s = sm.shared[1 + i], group = sm.slot[s].group;
    const uint32_t ex = (__float_as_uint((float)v[s]) >> 23) & 0xffu;
#pragma unroll
    for (int k = 0; k < AQ_MAX_GROUPS; ++k)
      if (group == k) gmax[k] = max(gmax[k], ex);
  }
  // quant_fixed_f32 of a signed slot (v - 0 == v, also for -0 and NaN)
  const auto fixed = [&](const SlotPlan& p, T x) {
    float c = __fmul_rn(__fsub_rn((float)x, p.offset), p.scale);
    if (DITH) {
      const uint32_t d = p.ja * (uint32_t)pk + p.jc;
      const float u = __fmul_rn(__uint2float_rn(d ^ (d >> 16) ^ (uint32_t)(pk >> 32)), 2.3283064365386963e-10f);
      c = __fsub_rn(__fadd_rn(c, u), 0.5f);
    }
    c = __fadd_rn(c, copysignf(0.5f, c));
    return (uint32_t)__float2int_rz(c) & p.mask;
  };
  // bit stream in 32-bit words; fill < 32 between fields
  uint32_t acc = 0;
  int fill = 0;
  uint32_t* o = sw;
  const auto put = [&](uint32_t code, int nb) {  // nb <= 32, code < 2^nb
    acc |= code << fill;
    const int nf = fill + nb;
    if (nf >= 32) {
      *o = acc;
      o += 32;
      acc = __funnelshift_rc(code, 0u, 32 - fill);  // 0 when the field ended on the word (fill 0)
      fill = nf - 32;
    } else {
      fill = nf;
    }
  };
  for (int s = 0; s < ns; ++s) {
    const SlotPlan p = sm.plan[s];
    if (p.kind == PLAN_SIGNED + 8) {  // four slots, their chains side by side
      const SlotPlan p1 = sm.plan[s + 1], p2 = sm.plan[s + 2], p3 = sm.plan[s + 3];
      const uint32_t a = fixed(p, v[s]), b = fixed(p1, v[s + 1]), c = fixed(p2, v[s + 2]), d = fixed(p3, v[s + 3]);
      put(a, p.bits);
      put(b, p1.bits);
      put(c, p2.bits);
      put(d, p3.bits);
      s += 3;
      continue;
    }
    const T x = v[s];
    if (p.kind == PLAN_SIGNED) {
      put(fixed(p, x), p.bits);
      continue;
    }
    if (p.kind == PLAN_F32) {
      put(__float_as_uint((float)x), 32);
      continue;
    }
    const aq_slot& S = sm.slot[s];
    switch (S.kind) {
      case AQ_FIXED: {
        if (f64) {
          double u = 0.0;
          if (DITH) u = ud ? ud[s] : uniform_f64(pk, s);
          put(quant_fixed_f64(S, DITH, (double)x, u), S.bits);
        } else {
          float u = 0.0f;
          if (DITH) u = uf ? uf[s] : uniform_f32(pk, s);
          put(quant_fixed_f32(S, DITH, (float)x, u), S.bits);
        }
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
      default: {
        const uint64_t f = (uint64_t)__double_as_longlong((double)x);
        put((uint32_t)f, 32);
        put((uint32_t)(f >> 32), 32);
        break;
      }
    }
  }
  // the record's last word, and the other half of its 64-bit word
  if (fill > 0) {
    *o = acc;
    o += 32;
  }
  if (o < sw + 2 * W * 32) *o = 0;
}

// Values (n x n_slots rows) -> records.  GROUPED: into grouped storage at
// positions base + i, ids base + i also written to ids; else contiguous, with
// the dithering keyed on pid[i] (or i) and the uniforms given or drawn.
template <class T, bool GROUPED, bool DITH>
__global__ void __launch_bounds__(REC_T) k_encode(const __grid_constant__ aq_layout L, const T* __restrict__ values,
                                                  uint64_t* __restrict__ words, int64_t n,
                                                  const int32_t* __restrict__ pid, int32_t* __restrict__ ids,
                                                  int64_t base, uint64_t sk, const float* __restrict__ uf,
                                                  const double* __restrict__ ud) {
  extern __shared__ __align__(16) unsigned char rec_sm[];
  const int ns = L.n_slots, W = L.n_words, lane = threadIdx.x & 31, np = rec_vals_stride(ns);
  const RecSmem sm = rec_smem(L, rec_sm, W, ns, sizeof(T));
  T* const sv = static_cast<T*>(sm.vals);
  const RowWalk vw(ns);
  rec_plans(L, sm, true, uf != nullptr);
  for (int64_t g = rec_first_group(); g * 32 < n; g += rec_group_step()) {
    const int64_t i0 = g * 32, i = i0 + lane;
    const int cnt = (int)min((int64_t)32, n - i0);
    load_rows(values + i0 * ns, ns, cnt, vw, [&](int r, int k, T v) { sv[r * np + k] = v; });
    __syncwarp();
    if (lane < cnt) {
      const int32_t id = GROUPED ? (int32_t)(base + i) : pid ? pid[i] : (int32_t)i;
      rec_encode<T, DITH>(sm, ns, W, L.compute_f64 != 0, sv + lane * np, sm.words + lane, particle_key(sk, id),
                          uf ? uf + i * ns : nullptr, ud ? ud + i * ns : nullptr);
      if (GROUPED) {
        rec_store_grouped(sm.words, words, base + i, W);
        ids[base + i] = id;
      }
    }
    __syncwarp();
    if (!GROUPED) {
      const RowWalk w(W);
#pragma unroll 4
      for (int r = w.r; r < cnt; r += w.step) words[(i0 + r) * W + w.k] = SRec{sm.words + r}[w.k];
      __syncwarp();
    }
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
  const RecSmem sm = rec_smem(L, rec_sm, W, ns, sizeof(T));
  T* const sv = static_cast<T*>(sm.vals);
  const RowWalk vw(ns);
  const bool f64 = L.compute_f64 != 0;
  rec_plans(L, sm, false, false);
  for (int64_t g = rec_first_group(); g * 32 < n; g += rec_group_step()) {
    const int cnt = (int)min((int64_t)32, n - g * 32);
    if (GROUPED)
      rec_load_group(words, g, cnt, W, sm.words);
    else
      rec_load_rows(words, g * 32, cnt, W, sm.words);
    sm.row[lane] = lane < cnt ? (GROUPED ? (int64_t)__ldg(pid + g * 32 + lane) : g * 32 + lane) * ns : 0;
    __syncwarp();
    if (lane < cnt) rec_decode<T>(sm, ns, f64, sm.words + lane, sv + lane * np);
    __syncwarp();
#pragma unroll 8
    for (int r = vw.r; r < cnt; r += vw.step) values[sm.row[r] + vw.k] = sv[r * np + vw.k];
    __syncwarp();
  }
}

// Records from the simulator's grouped storage to contiguous records in
// particle order (record i goes to out[pid[i] - base]; base: the id of out's
// first record, a streamed chunk's first particle).
__global__ void __launch_bounds__(REC_T) k_words_ungroup(const uint64_t* __restrict__ in,
                                                                const int32_t* __restrict__ pid,
                                                                uint64_t* __restrict__ out, int64_t n, int W,
                                                                int64_t base) {
  extern __shared__ __align__(16) unsigned char rec_sm[];
  const int lane = threadIdx.x & 31;
  const RecSmem sm = rec_smem_words(rec_sm, W);
  const RowWalk w(W);
  for (int64_t g = rec_first_group(); g * 32 < n; g += rec_group_step()) {
    const int cnt = (int)min((int64_t)32, n - g * 32);
    rec_load_group(in, g, cnt, W, sm.words);
    sm.row[lane] = lane < cnt ? ((int64_t)__ldg(pid + g * 32 + lane) - base) * W : 0;
    __syncwarp();
#pragma unroll 4
    for (int r = w.r; r < cnt; r += w.step) out[sm.row[r] + w.k] = SRec{sm.words + r}[w.k];
    __syncwarp();
  }
}

// Contiguous records (record i at in[i W]) into grouped storage, same order.
__global__ void __launch_bounds__(REC_T) k_words_group(const uint64_t* __restrict__ in,
                                                              uint64_t* __restrict__ out, int64_t n, int W) {
  extern __shared__ __align__(16) unsigned char rec_sm[];
  const int lane = threadIdx.x & 31;
  const RecSmem sm = rec_smem_words(rec_sm, W);
  for (int64_t g = rec_first_group(); g * 32 < n; g += rec_group_step()) {
    const int cnt = (int)min((int64_t)32, n - g * 32);
    rec_load_rows(in, g * 32, cnt, W, sm.words);
    __syncwarp();
    if (lane < cnt) rec_store_grouped(sm.words, out, g * 32 + lane, W);
    __syncwarp();
  }
}

static size_t rec_smem_cta(int W, int ns, size_t vsize) {
  return rec_smem_plans(ns) + (REC_T / 32) * rec_smem_warp(W, ns, vsize);
}

// CTAs for n records: all that fit at once, and no more than there are groups
static unsigned rec_grid(int64_t n, size_t smem) {
  const int per_sm = (int)std::min<size_t>(2048 / REC_T, std::max<size_t>(1, (size_t)220 * 1024 / (smem + 1024)));
  return (unsigned)std::min<int64_t>((n + REC_T - 1) / REC_T, (int64_t)num_sms() * per_sm);
}

// k_encode with or without dithering; smem and grid as above
template <class T, bool GROUPED>
static cudaError_t launch_encode(const aq_layout& L, const T* values, uint64_t* words, int64_t n, const int32_t* pid,
                                 int32_t* ids, int64_t base, uint64_t sk, const float* uf, const double* ud,
                                 cudaStream_t st) {
  const size_t smem = rec_smem_cta(L.n_words, L.n_slots, sizeof(T));
  const unsigned grid = rec_grid(n, smem);
  if (L.use_dithering)
    k_encode<T, GROUPED, true><<<grid, REC_T, smem, st>>>(L, values, words, n, pid, ids, base, sk, uf, ud);
  else
    k_encode<T, GROUPED, false><<<grid, REC_T, smem, st>>>(L, values, words, n, pid, ids, base, sk, uf, ud);
  return cudaGetLastError();
}

template <class T, bool GROUPED>
static cudaError_t launch_decode(const aq_layout& L, const uint64_t* words, const int32_t* pid, T* values, int64_t n,
                                 cudaStream_t st) {
  const size_t smem = rec_smem_cta(L.n_words, L.n_slots, sizeof(T));
  k_decode<T, GROUPED><<<rec_grid(n, smem), REC_T, smem, st>>>(L, words, pid, values, n);
  return cudaGetLastError();
}

// Per-slot statistics of the decoded state (features of the sensitivity
// surrogate); out[slot * 5 + k] accumulates
// k = 0: sum |v|, 1: sum v, 2: sum v^2, 3: max |v| (as the bit pattern of a
// non-negative double, which orders like the value), 4: sum |v - ref|
// (ref: n x n_slots values in particle order, or null).
//
// A warp decodes 32 records at a time, a lane per record, into shared memory
// and then takes them a lane per slot, so that the sums stay in the lane's
// registers and the rows of ref are read in contiguous runs.  (One pass over
// the records per slot: 1,000,003 records of 24 slots with a float ref took
// 406 us, now 121.)
// V: the values' type in shared memory, float where every value of the layout
// is one (half the shared memory, twice the warps).
template <class T, class V>
__global__ void __launch_bounds__(REC_T) k_field_stats(const __grid_constant__ aq_layout L,
                                                       const uint64_t* __restrict__ words,
                                                       const int32_t* __restrict__ pid, const T* __restrict__ ref,
                                                       int64_t n, double* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char rec_sm[];
  __shared__ double sh[REC_T / 32][5][32];
  const int ns = L.n_slots, W = L.n_words, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, np = rec_vals_stride(ns);
  const RecSmem sm = rec_smem(L, rec_sm, W, ns, sizeof(V));
  V* const sv = static_cast<V*>(sm.vals);
  double a[5] = {0, 0, 0, 0, 0};
  V top = 0;
  const bool f64 = L.compute_f64 != 0;
  rec_plans(L, sm, false, false);
  for (int64_t g = rec_first_group(); g * 32 < n; g += rec_group_step()) {
    const int cnt = (int)min((int64_t)32, n - g * 32);
    sm.row[lane] = lane < cnt ? (int64_t)__ldg(pid + g * 32 + lane) * ns : 0;
    rec_load_group(words, g, cnt, W, sm.words);
    __syncwarp();
    if (lane < cnt) rec_decode<V>(sm, ns, f64, sm.words + lane, sv + lane * np);
    __syncwarp();
    if (lane < ns) {
      for (int r0 = 0; r0 < cnt; r0 += 16) {
        T t[16];
        if (ref) {
#pragma unroll
          for (int j = 0; j < 16; ++j) t[j] = r0 + j < cnt ? __ldg(ref + sm.row[r0 + j] + lane) : T(0);
        }
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (r0 + j < cnt) {
            const V x = sv[(r0 + j) * np + lane];
            const double v = (double)x;
            top = fmax(top, fabs(x));
            a[0] += fabs(v);
            a[1] += v;
            a[2] += v * v;
            if (ref) a[4] += fabs(v - (double)t[j]);
          }
      }
    }
    __syncwarp();
  }
  a[3] = (double)top;
#pragma unroll
  for (int j = 0; j < 5; ++j) sh[warp][j][lane] = a[j];
  __syncthreads();
  for (int e = threadIdx.x; e < 5 * ns; e += REC_T) {
    const int s = e / 5, j = e - 5 * s;
    double t = sh[0][j][s];
#pragma unroll
    for (int w = 1; w < REC_T / 32; ++w) t = j == 3 ? fmax(t, sh[w][j][s]) : t + sh[w][j][s];
    if (j == 3)
      atomicMax(reinterpret_cast<unsigned long long*>(out + e), (unsigned long long)__double_as_longlong(t));
    else
      atomicAdd(out + e, t);
  }
}

// --------------------------------------------------------------- launches

cudaError_t rec_encode_rows(const aq_layout& L, const void* values, bool f64, uint64_t* words, int64_t n,
                            const int32_t* pid, uint64_t sk, const float* uf, const double* ud, cudaStream_t st) {
  return f64 ? launch_encode<double, false>(L, (const double*)values, words, n, pid, nullptr, 0, sk, uf, ud, st)
             : launch_encode<float, false>(L, (const float*)values, words, n, pid, nullptr, 0, sk, uf, ud, st);
}

cudaError_t rec_decode_rows(const aq_layout& L, const uint64_t* words, void* values, bool f64, int64_t n,
                            cudaStream_t st) {
  return f64 ? launch_decode<double, false>(L, words, nullptr, (double*)values, n, st)
             : launch_decode<float, false>(L, words, nullptr, (float*)values, n, st);
}

cudaError_t rec_store(const aq_layout& L, const void* values, bool f64, uint64_t* words, int32_t* ids, int64_t base,
                      int64_t n, uint64_t sk, cudaStream_t st) {
  return f64 ? launch_encode<double, true>(L, (const double*)values, words, n, nullptr, ids, base, sk, nullptr, nullptr, st)
             : launch_encode<float, true>(L, (const float*)values, words, n, nullptr, ids, base, sk, nullptr, nullptr, st);
}

cudaError_t rec_fetch(const aq_layout& L, const uint64_t* words, const int32_t* pid, void* values, bool f64, int64_t n,
                      cudaStream_t st) {
  return f64 ? launch_decode<double, true>(L, words, pid, (double*)values, n, st)
             : launch_decode<float, true>(L, words, pid, (float*)values, n, st);
}

cudaError_t rec_ungroup(const uint64_t* in, const int32_t* pid, uint64_t* out, int64_t n, int W, int64_t base,
                        cudaStream_t st) {
  const size_t smem = rec_smem_cta(W, 0, 0);
  k_words_ungroup<<<rec_grid(n, smem), REC_T, smem, st>>>(in, pid, out, n, W, base);
  return cudaGetLastError();
}

cudaError_t rec_group(const uint64_t* in, uint64_t* out, int64_t n, int W, cudaStream_t st) {
  const size_t smem = rec_smem_cta(W, 0, 0);
  k_words_group<<<rec_grid(n, smem), REC_T, smem, st>>>(in, out, n, W);
  return cudaGetLastError();
}

cudaError_t rec_stats(const aq_layout& L, const uint64_t* words, const int32_t* pid, const void* ref, bool ref_f64,
                      int64_t n, double* out, cudaStream_t st) {
  bool narrow = true;  // every value is a float
  for (int k = 0; k < L.n_slots; ++k) {
    const aq_slot& S = L.slot[k];
    if (S.kind == AQ_RAW_F64 || (S.kind == AQ_FIXED && L.compute_f64) || (S.kind == AQ_INT && S.bits > 24)) narrow = false;
  }
  const size_t smem = rec_smem_cta(L.n_words, L.n_slots, narrow ? sizeof(float) : sizeof(double));
  const unsigned grid = rec_grid(n, smem);
  if (ref_f64 && narrow)
    k_field_stats<double, float><<<grid, REC_T, smem, st>>>(L, words, pid, (const double*)ref, n, out);
  else if (ref_f64)
    k_field_stats<double, double><<<grid, REC_T, smem, st>>>(L, words, pid, (const double*)ref, n, out);
  else if (narrow)
    k_field_stats<float, float><<<grid, REC_T, smem, st>>>(L, words, pid, (const float*)ref, n, out);
  else
    k_field_stats<float, double><<<grid, REC_T, smem, st>>>(L, words, pid, (const float*)ref, n, out);
  return cudaGetLastError();
}

}  // namespace aq
