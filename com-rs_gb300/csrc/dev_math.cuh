// Device helpers shared by every decoder, also compiled at run time by NVRTC for the
// graph-specialised decoder (layered_nr.cuh): explicitly rounded arithmetic, the min
// helpers of the row updates, the L2 policy of the check-node state and the block-wide
// syndrome test on packed hard decisions.  No includes but <cstdint> under nvcc.
#pragma once
#ifndef __CUDACC_RTC__
#include <cstdint>
#else
typedef unsigned char uint8_t;
typedef unsigned short uint16_t;
typedef unsigned int uint32_t;
typedef int int32_t;
typedef unsigned long long uint64_t;
typedef long long int64_t;
typedef unsigned long long uintptr_t;
#endif

namespace cbk {
namespace {

template <typename T>
__device__ __forceinline__ T add_rn(T a, T b);
template <>
__device__ __forceinline__ double add_rn<double>(double a, double b) { return __dadd_rn(a, b); }
template <>
__device__ __forceinline__ float add_rn<float>(float a, float b) { return __fadd_rn(a, b); }
template <typename T>
__device__ __forceinline__ T sub_rn(T a, T b);
template <>
__device__ __forceinline__ double sub_rn<double>(double a, double b) { return __dsub_rn(a, b); }
template <>
__device__ __forceinline__ float sub_rn<float>(float a, float b) { return __fsub_rn(a, b); }
template <typename T>
__device__ __forceinline__ T mul_rn(T a, T b);
template <>
__device__ __forceinline__ double mul_rn<double>(double a, double b) { return __dmul_rn(a, b); }
template <>
__device__ __forceinline__ float mul_rn<float>(float a, float b) { return __fmul_rn(a, b); }

// The bit pattern of |x| from that of a double x: the AND as inline PTX, opaque to the
// compiler's recognition of `bits & 0x7fff...` as fabs, whose result it then forms on the
// FP64 pipe when the consumer is an integer comparison
__device__ __forceinline__ long long abs_bits(long long b) {
  long long r;
  asm("and.b64 %0, %1, 0x7fffffffffffffff;" : "=l"(r) : "l"(b));
  return r;
}

template <typename T>
__device__ __forceinline__ T infinity();
template <>
__device__ __forceinline__ double infinity<double>() { return __longlong_as_double(0x7ff0000000000000ll); }
template <>
__device__ __forceinline__ float infinity<float>() { return __int_as_float(0x7f800000); }

// ---- syndrome test on packed hard decisions
// post < 0 for the hard decision: in f64 the sign bit (an integer test), since the
// posteriors are never -0.0 or NaN
__device__ __forceinline__ uint32_t is_negative(double v) {
  return (uint32_t)((unsigned long long)__double_as_longlong(v) >> 63);
}
__device__ __forceinline__ uint32_t is_negative(float v) { return (uint32_t)(v < 0.0f); }

// hd holds, per base column j, the hard decisions of its Z bits packed 32 per word
// (ceil(Z/32) words, then one zero word).  The parity of the 32 lifted rows
// [32g, 32g + 32) of layer L is the XOR over the layer's entries (j, s) of the
// Z-bit circular window of column j starting at (32g + s) mod Z.
template <typename T>
__device__ __forceinline__ void build_hard_decisions(const T* post, uint32_t* hd, int ncol, int z, int tid, int nt) {
  const int wz = (z + 31) >> 5, ws = wz + 1;
  const int lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  for (int task = warp; task < ncol * wz; task += nw) {
    const int j = task / wz, w = task - j * wz;
    const int r = w * 32 + lane;
    const uint32_t word = __ballot_sync(0xffffffffu, r < z && is_negative(post[j * z + r]));
    if (lane == 0) {
      hd[j * ws + w] = word;
      if (w == wz - 1) hd[j * ws + wz] = 0u;
    }
  }
}

// 32 bits of a packed column from bit o (bits at or beyond Z read as 0)
__device__ __forceinline__ uint32_t window32(const uint32_t* col, int o) {
  return __funnelshift_r(col[o >> 5], col[(o >> 5) + 1], o & 31);
}

// Stage 2 of the syndrome test: every row on packed hard decisions.  Block-wide.
template <typename T>
__device__ __forceinline__ bool some_packed_check_fails(const T* post, uint32_t* hd, const uint32_t* ent,
                                                        const uint16_t* lstart, int rows_n, int ncol, int z, int tid,
                                                        int nt) {
  int bad = 0;
  build_hard_decisions(post, hd, ncol, z, tid, nt);
  __syncthreads();
  const int wz = (z + 31) >> 5, ws = wz + 1;
  for (int task = tid; task < rows_n * wz && !bad; task += nt) {
    const int L = task / wz, g = task - L * wz;
    const int r0 = g * 32, nrows = min(32, z - r0);
    uint32_t par = 0;
    for (int t = lstart[L]; t < lstart[L + 1]; t++) {
      const uint32_t en = ent[t];
      const uint32_t* col = hd + (en >> 16) * ws;
      int o = r0 + (int)(en & 0xffffu);
      o -= (o >= z) ? z : 0;
      uint32_t win = window32(col, o);
      if (o + nrows > z) win |= window32(col, 0) << (z - o);
      par ^= win;
    }
    const uint32_t mask = nrows == 32 ? 0xffffffffu : ((1u << nrows) - 1u);
    bad = (par & mask) != 0u;
  }
  return __syncthreads_or(bad) != 0;
}

// Stage 1 of the syndrome test: the rows of the first two layers, read directly (each thread its
// own row, stopping at the first failure).  Block-wide.
template <typename T>
__device__ __forceinline__ bool first_rows_fail(const T* post, const uint32_t* ent, const uint16_t* lstart, int z,
                                                int tid) {
  int bad = 0;
  if (tid < z) {
    for (int L = 0; L < 2 && !bad; L++) {
      uint32_t par = 0;
      for (int t = lstart[L]; t < lstart[L + 1]; t++) {
        const uint32_t en = ent[t];
        int cc = tid + (int)(en & 0xffffu);
        cc -= (cc >= z) ? z : 0;
        par ^= is_negative(post[(int)(en >> 16) * z + cc]);
      }
      bad = (int)par;
    }
  }
  return __syncthreads_or(bad) != 0;
}

// Whether some check fails on the hard decisions of post (hard_decisions_are_a_codeword,
// ldpc.rs:555-557).  Block-wide.  While the decoder has not converged stage 1 almost always
// finds a failing check.  Only when every one of its rows is satisfied does stage 2 test all
// rows on packed hard decisions.  Either way the answer is exactly "H c != 0".
template <typename T>
__device__ __forceinline__ bool some_check_fails(const T* post, uint32_t* hd, const uint32_t* ent,
                                                 const uint16_t* lstart, int rows_n, int ncol, int z, int tid,
                                                 int nt) {
  if (first_rows_fail(post, ent, lstart, z, tid)) return true;
  return some_packed_check_fails(post, hd, ent, lstart, rows_n, ncol, z, tid, nt);
}

// some_check_fails after an iteration: `own` forms the own columns of skipped rows (see
// unsent_rows) before stage 2 reads them
template <typename T, class Own>
__device__ __forceinline__ bool some_check_fails_after(const T* post, uint32_t* hd, const uint32_t* ent,
                                                       const uint16_t* lstart, int rows_n, int ncol, int z, int tid,
                                                       int nt, const Own& own) {
  if (first_rows_fail(post, ent, lstart, z, tid)) return true;
  own();
  return some_packed_check_fails(post, hd, ent, lstart, rows_n, ncol, z, tid, nt);
}

// Magnitudes beyond which a codeword runs every row: those in which a skipped row may change
// more than its own column.  Such a row sends zero because its own variable comes in with
// magnitude zero, what the row made of it less its old message, while that is finite: from
// an infinite one inf - inf is NaN, which the minimum passes over, and the row's other
// variables get messages.  Every skipped row has an edge in one of the watched base columns
// (0 and 1, in base graph 2 also 2 and 10; cbh::live_rows asks for it), so its smallest magnitude
// is finite while those columns are.  A posterior that is not finite never is again, so the plain
// rules, which make no magnitude larger (cbk::decoder_rows), are tested at a codeword's end; a
// learned scale may (up to cbd::kSkipMaxScale), so there the test follows every iteration.
// A codeword that fails it is decoded again.  The channel LLRs are tested where they are
// loaded: infinite ones end in the watched columns anyway, and beside a NaN the pairwise
// minimum search finds another second minimum.  (Tested after every iteration the plain
// decoders took 1-2 % longer.)
__device__ __forceinline__ bool beyond_skipping(float v) { return (__float_as_uint(v) & 0x7fffffffu) >= (127u + 100u) << 23; }
__device__ __forceinline__ bool beyond_skipping(double v) {
  return ((uint32_t)__double2hiint(v) & 0x7fffffffu) >= (1023u + 1000u) << 20;
}
// the watched variables of lifted row r
template <typename T>
__device__ __forceinline__ bool beyond_skipping(const T* post, int r, int z, int bg) {
  return beyond_skipping(post[r]) || beyond_skipping(post[z + r]) ||
         (bg == 2 && (beyond_skipping(post[2 * z + r]) || beyond_skipping(post[10 * z + r])));
}
// whether some of a thread's values is beyond the bound, an instruction a value in f32
// (tested one by one the loads of a rate 1/2 codeword took 1 % of its decoding)
template <typename T>
struct Widest;
template <>
struct Widest<float> {
  float most = 0.0f;
  __device__ __forceinline__ void add(float v) { asm("max.NaN.f32 %0, %0, %1;" : "+f"(most) : "f"(fabsf(v))); }
  __device__ __forceinline__ bool beyond() const { return beyond_skipping(most); }
};
template <>
struct Widest<double> {
  bool some = false;
  __device__ __forceinline__ void add(double v) { some = some || beyond_skipping(v); }
  __device__ __forceinline__ bool beyond() const { return some; }
};

// The own parity columns of the base rows [live, rows): columns that are not sent and in no
// other row (cbh::live_rows).  What such a row makes of its variable is 0 + the message
// from the row's other variables, whose messages from the row are zero: their smallest
// magnitude through `mag` (the rule; entry of the own column, lifted row, magnitude) with the
// product of their signs.  The own column is the row's last entry.
template <typename T, class Mag>
__device__ __forceinline__ void unsent_rows(T* post, const uint32_t* ent, const uint16_t* lstart, int live, int rows,
                                            int z, int tid, int nt, const Mag mag) {
  for (int task = tid; task < (rows - live) * z; task += nt) {
    const int q = task / z, r = task - q * z, own = lstart[live + q + 1] - 1;
    T m = infinity<T>();
    uint32_t neg = 0;
    for (int t = lstart[live + q]; t < own; t++) {
      const uint32_t en = ent[t];
      int cc = r + (int)(en & 0xffffu);
      cc -= (cc >= z) ? z : 0;
      const T v = post[(int)(en >> 16) * z + cc];
      neg ^= is_negative(v);
      m = fmin(m, fabs(v));
    }
    const uint32_t en = ent[own];
    int cc = r + (int)(en & 0xffffu);
    cc -= (cc >= z) ? z : 0;
    const T o = mag(own, r, m);
    post[(int)(en >> 16) * z + cc] = add_rn((T)0, neg ? -o : o);
  }
}

// the same out of line: called once a codeword, and inlined its registers made the iteration of
// the graph-specialised decoder spill
template <typename T, class Mag>
__device__ __noinline__ void unsent_rows_call(T* post, const uint32_t* ent, const uint16_t* lstart, int live, int rows,
                                              int z, int tid, int nt, const Mag mag) {
  unsent_rows(post, ent, lstart, live, rows, z, tid, nt, mag);
}

__device__ __forceinline__ float ld_post(const float* post, int off) {
  return *reinterpret_cast<const float*>(reinterpret_cast<const char*>(post) + off);
}
__device__ __forceinline__ void st_post(float* post, int off, float v) {
  *reinterpret_cast<float*>(reinterpret_cast<char*>(post) + off) = v;
}
// |d| = min(|a|, |b|), sign(d) = sign(a) xor sign(b)
__device__ __forceinline__ float min_xorsign_abs(float a, float b) {
  float d;
  asm("min.xorsign.abs.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ float min3f(float a, float b, float c) {
  float d;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// The state records of all resident CTAs (64 MB at BG1 Z = 384) fit in L2, but the LLR
// stream of a launch (830 MB for 8192 codewords) would evict them: the records are read
// and written with an L2 evict-last policy, the LLRs with streaming loads.
__device__ __forceinline__ uint64_t l2_evict_last_policy() {
  uint64_t pol;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}

}  // namespace
}  // namespace cbk
