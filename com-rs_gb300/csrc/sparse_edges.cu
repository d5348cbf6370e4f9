// Layered sum-product decoding of small generic codes, an edge per thread.
//
// In f64 the sum-product row is bound by the FP64 pipe, which GB300 has little of (2 lanes
// per SM and clock: a warp instruction holds its quarter of the pipe for 64 cycles however
// many of its lanes work).  A thread per row (sparse_group_kernel) left half of the lanes
// idle, levels having few rows (15 of 32 at work on PEG(1024, 512)), and its threads ran a
// row's six tanh and six atanh one after the other, 15 us a level, while every codeword of
// the group waited for the slowest.  Here
//   * a codeword has a slot of its own: posteriors and messages in shared memory, `warps`
//     warps that a named barrier holds together, and the next codeword from the work
//     counter as soon as it is done;
//   * the edges of a level are spread over the slot's lanes: each computes its tanh, then,
//     after a barrier, the product of the row's other tanh values and its own outgoing
//     message.
// Measured (GB300, words with the copies): the link of 512 trials, 4096 words of PEG(1024, 512),
// 76.7 -> 33.0 ms; PEG(576, 288), 2000 words of 3 iterations, some of 50, 20.7 -> 5.6 ms
// (15.3 -> 4.6 on another box).  PEG codes of 301 to 4000 bits, 1 to 3000 words: f64 1.3 to
// 4.3 times faster, f32 1.0 to 2.2.  What is left in f64 is the FP64 pipe, 81-85 % busy.
// The product is formed as check_row (sparse.cu) forms it: the running product of the
// edges before, first to last, times that of the edges after, last to first, so the results
// are the same bits.
#include <cuda_runtime.h>

#include "kernels.h"
#include "sparse_math.cuh"

namespace cbk {
namespace {

__device__ __forceinline__ void slot_sync(int bar, int n) { asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(n) : "memory"); }

// The edges of a level are grouped by the size of |l|, so that the lanes of a warp have arguments of
// one kind: it orders the work and nothing else.  The high word of 21/16, the fastest value of
// those tried (sixteenths from 18 to 24, and 1/2, 1, 2 and 3) by the time of the whole decode:
// the link of 512 trials at 2.5 dB 91 ms, with 20/16 97, 22/16 98, 18/16 103 and 24/16 102; at 4 dB
// 33.0 ms, 33.6 to 34.1, 34.5, 35.0 and 35.0, with 1 36.5, 3 36.5 and one group 36.7.
constexpr int kGroupSplitHi = 0x3ff50000;

// x / 2, for doubles by the exponent field (off the FP64 pipe) unless the result could be
// subnormal or x is not finite
__device__ __forceinline__ float half_of(float x) { return mul_rn(x, 0.5f); }
__device__ __forceinline__ double half_of(double x) {
  const uint32_t hi = (uint32_t)__double2hiint(x);
  if (((hi >> 20) & 0x7ffu) - 2u < 0x7fdu) return __hiloint2double((int)(hi - 0x100000u), __double2loint(x));
  return mul_rn(x, 0.5);
}

// x < 0 as a bit
__device__ __forceinline__ int below_zero(float x) { return (int)(x < 0.0f); }
__device__ __forceinline__ int below_zero(double x) {
  // the sign bit of a nonzero, non-NaN x
  const long long b = __double_as_longlong(x), a = abs_bits(b);
  return (int)(b < 0 && a != 0 && a <= 0x7ff0000000000000ll);
}

// whether some row of the slot's codeword fails; `flag` starts and is left at 0
template <typename T>
__device__ __forceinline__ bool slot_check_fails(const EdgeDev& c, const T* post, const uint32_t* edge,
                                                 const uint16_t* row, int lt, int nt, int bar, volatile int* flag) {
  int bad = 0;
  for (int r = lt; r < c.m && !bad; r += nt) {
    int par = 0;
    for (int e = row[r]; e < row[r + 1]; e++) par ^= below_zero(post[edge[e] & 0xffffu]);
    bad = par;
  }
  if (bad) *flag = 1;
  slot_sync(bar, nt);
  const int f = *flag;
  slot_sync(bar, nt);
  if (lt == 0) *flag = 0;
  return f != 0;
}

template <typename T>
__global__ void __launch_bounds__(kEdgeThreads, 1) sparse_edges_kernel(const __grid_constant__ EdgeArgs<T> a) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ long long s_cw[kEdgeMaxSlots];
  __shared__ int s_flag[kEdgeMaxSlots];
  __shared__ int s_cnt[kEdgeMaxSlots][2][2];  // f64: a level's edges of large and small argument, by parity
  const EdgeDev& c = a.code;
  const int nt = c.warps * 32, slot = threadIdx.x / nt, lt = threadIdx.x - slot * nt, bar = slot + 1;
  // shared memory: the slots' posteriors, messages and tanh values of a level, then the tables
  const size_t per = (size_t)c.n + c.edges + c.max_level_edges;
  T* post = reinterpret_cast<T*>(smem) + slot * per;
  T* msg = post + c.n;
  T* tb = msg + c.edges;
  uint32_t* edge = reinterpret_cast<uint32_t*>(reinterpret_cast<T*>(smem) + a.slots * per);
  uint16_t* row = reinterpret_cast<uint16_t*>(edge + c.edges);
  uint16_t* level = row + c.m + 1;
  uint16_t* list = level + c.levels + 1 + slot * c.max_level_edges;  // f64
  for (int i = threadIdx.x; i < c.edges; i += blockDim.x) edge[i] = c.edge[i];
  for (int i = threadIdx.x; i <= c.m; i += blockDim.x) row[i] = (uint16_t)c.row[i];
  for (int i = threadIdx.x; i <= c.levels; i += blockDim.x) level[i] = (uint16_t)c.level[i];
  if (threadIdx.x < kEdgeMaxSlots) {
    s_flag[threadIdx.x] = 0;
    for (int i = 0; i < 4; i++) s_cnt[threadIdx.x][i >> 1][i & 1] = 0;
  }
  __syncthreads();
  int parity = 0;
  for (;;) {
    if (lt == 0) s_cw[slot] = (long long)atomicAdd(a.work_counter, 1ull);
    slot_sync(bar, nt);
    const long long cw = s_cw[slot];
    if (cw >= a.n_frames) break;
    const T* llr = a.llr + (size_t)cw * c.n;
    for (int v = lt; v < c.n; v += nt) post[v] = llr[v];
    for (int e = lt; e < c.edges; e += nt) msg[e] = (T)0;
    slot_sync(bar, nt);
    int it = 0;
    if (slot_check_fails(c, post, edge, row, lt, nt, bar, &s_flag[slot])) {
      it = a.max_iterations;
      for (int iter = 1; iter <= a.max_iterations; iter++) {
        for (int L = 0; L < c.levels; L++) {
          const int e0 = level[L], e1 = level[L + 1];
          // each edge's tanh(l / 2), and l into its posterior (no other row of the level
          // touches the variable)
          if constexpr (sizeof(T) == 4) {
            for (int e = e0 + lt; e < e1; e += nt) {
              const int v = (int)(edge[e] & 0xffffu);
              const T l = sub_rn(post[v], msg[e]);
              post[v] = l;
              tb[e - e0] = tanh_t(half_of(l));
            }
          } else {
            // large arguments at the front of the list, small ones at its back
            int* cnt = s_cnt[slot][parity];
            for (int b = e0; b < e1; b += nt) {
              const int e = b + lt;
              const bool in = e < e1;
              bool small = false;
              if (in) {
                const int v = (int)(edge[e] & 0xffffu);
                const T l = sub_rn(post[v], msg[e]);
                post[v] = l;
                small = (__double2hiint(l) & 0x7fffffff) < kGroupSplitHi;
              }
              const unsigned ms = __ballot_sync(0xffffffffu, in && small), ml = __ballot_sync(0xffffffffu, in && !small);
              int at = 0;
              if ((lt & 31) < 2) at = atomicAdd(&cnt[lt & 31], __popc((lt & 31) ? ms : ml));
              const int al = __shfl_sync(0xffffffffu, at, 0), as = __shfl_sync(0xffffffffu, at, 1);
              const unsigned below = (1u << (lt & 31)) - 1u;
              if (in) list[small ? e1 - e0 - 1 - as - __popc(ms & below) : al + __popc(ml & below)] = (uint16_t)e;
            }
            slot_sync(bar, nt);
            const int nl = cnt[0], ns = e1 - e0 - nl, pad = (nl + 31) & ~31;
            parity ^= 1;
            if (lt < 2) s_cnt[slot][parity][lt] = 0;
            for (int i = lt; i < pad + ns; i += nt) {
              if (i < nl || i >= pad) {
                const int e = list[i < nl ? i : i - pad + nl];
                tb[e - e0] = tanh_t(half_of(post[edge[e] & 0xffffu]));
              }
            }
          }
          slot_sync(bar, nt);
          for (int e = e0 + lt; e < e1; e += nt) {
            const uint32_t w = edge[e];
            const int v = (int)(w & 0xffffu), k = (int)((w >> 16) & 0xffu), d = (int)(w >> 24);
            const T* t = tb + (e - e0 - k);
            T pre = k > 0 ? t[0] : (T)1, suf = k < d - 1 ? t[d - 1] : (T)1;
            // each step multiplies the next factor onto the product before the edge or,
            // when that is complete, onto the one after it: one multiplication a step for
            // every lane, whatever its place in the row
            for (int i = 0, j = d - 2; i < d - 2; i++) {
              const bool before = i < k - 1, after = !before && j > k;
              const T f = before ? t[i + 1] : after ? t[j] : (T)1;
              const T p = mul_rn(before ? pre : suf, f);
              pre = before ? p : pre;
              suf = before ? suf : p;
              j -= after;
            }
            const T o = twice_atanh_t(mul_rn(pre, suf));
            msg[e] = o;
            post[v] = add_rn(post[v], o);
          }
          slot_sync(bar, nt);
        }
        if (!slot_check_fails(c, post, edge, row, lt, nt, bar, &s_flag[slot])) {
          it = iter;
          break;
        }
      }
    }
    if (a.post_out)
      for (int v = lt; v < c.n; v += nt) a.post_out[(size_t)cw * c.n + v] = post[v];
    if (lt == 0 && a.iters_out) a.iters_out[cw] = it;
    slot_sync(bar, nt);
  }
}

}  // namespace

size_t sparse_edges_slot_bytes(int n, int edges, int max_level_edges, int precision) {
  return ((size_t)n + edges + max_level_edges) * (precision == 0 ? 8 : 4) + (precision == 0 ? 2 * (size_t)max_level_edges : 0);
}
size_t sparse_edges_table_bytes(int edges, int m, int levels) {
  return (size_t)edges * 4 + ((size_t)m + levels + 2) * 2;
}

void* sparse_edges_kernel_ptr(int precision) {
  return precision == 0 ? (void*)sparse_edges_kernel<double> : (void*)sparse_edges_kernel<float>;
}

}  // namespace cbk
