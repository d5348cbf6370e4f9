// Layered belief propagation on codes whose rows form a chain (irregular
// repeat-accumulate codes: DVB-S2, dual-diagonal parity), the layered schedule of
// sparse.cu run in blocks of consecutive rows.
//
// Row r of such a code closes on the parity bits p(r - 1) and p(r), so every row shares a
// variable with the one before it, the level schedule has one row per level, and a warp
// per row spends an iteration on m dependent steps of about 0.8 us (DVB-S2 short rate
// 1/2: 9000 rows, 7.2 ms an iteration, one warp of the SM at work, issue 11 %).  But the
// only dependence inside a run of rows is one number, the posterior that row r hands to
// row r + 1; the other variables of about 60 consecutive rows are distinct in every DVB-S2
// code.  A block of such rows (sparse_host.h, ChainBlocks) is decoded in three phases:
//   1. all edges but the link-in ones at once, a group of G lanes per row: incoming
//      messages, tanh values and prefix products (min-sum: the row's minimum and sign);
//   2. two warps solve the chain x(r + 1) = f_r(x(r)), a row per thread, by sweeps that
//      evaluate every f_r at the current inputs and hand the results on, until no input
//      changes by a bit.  The system is triangular, so the fixed point is the sequential
//      result exactly, whatever the starting values; after k sweeps the first k rows hold
//      it, so a block of b rows takes at most b sweeps.  A check row damps what
//      comes in (its other edges bound the output), so a few sweeps do;
//   3. the outgoing messages and posteriors of all edges.
// The products are associated as check_row_warp of sparse.cu associates them (a scan over
// the row's edges), so posteriors and iteration counts are the same bits as that path's.
//
// Bound: the latency of the chain sweeps (a tanh and an atanh each), two warps of a CTA.
// The next block's variables and messages are loaded during the sweeps.  Measured on
// DVB-S2 short rate 1/2, f32 sum-product, 152 words of 5.8 iterations (9 at most): 65 ms
// with a warp per row, 5.8 ms with the chain on one warp (two rows a lane: 10.6 sweeps a
// block of 670 cycles, phase 1 1940 and phase 3 940 cycles), 4.5 ms on two.
#include <cuda_runtime.h>

#include "decode_common.cuh"
#include "kernels.h"
#include "sparse_math.cuh"

namespace cbk {
namespace {

constexpr unsigned kFull = 0xffffffffu;

template <typename T>
__device__ __forceinline__ bool same_bits(T a, T b);
template <>
__device__ __forceinline__ bool same_bits<float>(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }
template <>
__device__ __forceinline__ bool same_bits<double>(double a, double b) {
  return __double_as_longlong(a) == __double_as_longlong(b);
}

// what phase 1 leaves for the chain, and the chain for phase 3, per row of a block
template <typename T>
struct ChainRow {
  // sum-product: the factors that the scan multiplies onto the link-in edge's tanh, in
  // order; min-sum: f[0] the smallest magnitude and f[1] the sign (+-1) of the edges
  // before the last two
  T f[5];
  T xl;     // the second to last edge: its incoming message, or (linked) its old message
  T xr;     // the last edge's incoming message
  T tl;     // out: tanh(xl / 2)
  T outr;   // out: the last edge's outgoing message
};

template <typename T>
__device__ __forceinline__ T scaled_mag(T mag, T alpha, bool oms) {
  return oms ? fmax(sub_rn(mag, alpha), (T)0) : mul_rn(alpha, mag);
}

// the last edge's outgoing message from the second to last edge's incoming message
template <typename T, bool SPA, int G>
__device__ __forceinline__ T chain_message(const T (&f)[5], T xl, bool has_left, T alpha, bool oms, T& tl) {
  if constexpr (SPA) {
    tl = has_left ? tanh_t(mul_rn(xl, (T)0.5)) : (T)1;
    T p = mul_rn(f[0], tl);
    p = mul_rn(f[1], p);
    p = mul_rn(f[2], p);
    if constexpr (G > 8) p = mul_rn(f[3], p);
    if constexpr (G > 16) p = mul_rn(f[4], p);
    return twice_atanh_t(p);
  } else {
    tl = (T)0;
    T m = f[0];
    T s = f[1];
    if (has_left) {
      const T a = fabs(xl);
      if (a < m) m = a;
      if (xl < (T)0) s = -s;
    }
    return mul_rn(s, scaled_mag(m, alpha, oms));
  }
}

// whether the predicate holds for every thread of the chain's warps, which it synchronises
__device__ __forceinline__ bool chain_all(bool p) {
  int all;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\tbarrier.cta.red.and.pred q, 1, %2, p;\n\t"
      "selp.s32 %0, 1, 0, q;\n\t}"
      : "=r"(all)
      : "r"((int)p), "n"(kChainBlockRows)
      : "memory");
  return all != 0;
}

template <typename T, bool SPA, int G, int NT>
__global__ void __launch_bounds__(NT) sparse_chain_kernel(const __grid_constant__ ChainArgs<T> a) {
  constexpr int R = kChainBlockRows * G / NT;  // edges per thread of a full block
  static_assert(R * NT == kChainBlockRows * G && R >= 1, "a block's edges split evenly over the threads");
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ ChainRow<T> s_row[kChainBlockRows];
  __shared__ T s_next[2][kChainBlockRows + 1];  // the posterior handed to each row, by sweep parity
  __shared__ long long s_cw;
  const ChainDev& c = a.code;
  const int tid = threadIdx.x, lane = tid & 31, k = tid & (G - 1);
  const size_t msgs = (size_t)c.m * G;
  T* msg = a.slots + (size_t)blockIdx.x * (msgs + (a.post_in_smem ? 0 : (size_t)c.n));
  T* post = a.post_in_smem ? reinterpret_cast<T*>(smem) : msg + msgs;
  const T alpha = (T)a.alpha;
  const bool oms = a.oms != 0;
  for (;;) {
    if (tid == 0) s_cw = (long long)atomicAdd(a.work_counter, 1ull);
    __syncthreads();
    const long long cw = s_cw;
    if (cw >= a.n_frames) break;
    const T* llr = a.llr + (size_t)cw * c.n;
    for (int v = tid; v < c.n; v += NT) post[v] = llr[v];
    __syncthreads();
    int it = 0;
    // the rows' parities, a group of G lanes per row
    auto some_row_fails = [&]() {
      int bad = 0;
      for (int r0 = 0; r0 < c.m && !bad; r0 += NT / G) {
        const int r = r0 + tid / G;
        const int v = r < c.m ? c.vars[(size_t)r * G + k] : -1;
        unsigned neg = __ballot_sync(kFull, v >= 0 && post[v] < (T)0);
        if (G < 32) neg = (neg >> (lane & ~(G - 1))) & ((1u << (G & 31)) - 1u);
        bad = __any_sync(kFull, __popc(neg) & 1);
      }
      return __syncthreads_or(bad) != 0;
    };
    if (some_row_fails()) {
      it = a.max_iterations;
      for (int iter = 1; iter <= a.max_iterations; iter++) {
        int nv[R];   // the block's variables and old messages (loaded a block ahead)
        T nm[R];
        uint32_t ni[R];  // their rows: bits 0-5 the degree, then the link flags
        auto load = [&](int b) {
          const int r0 = c.block_start[b], rows = c.block_start[b + 1] - r0;
#pragma unroll
          for (int j = 0; j < R; j++) {
            const int rl = (tid + j * NT) / G;
            const size_t e = (size_t)(r0 + rl) * G + k;
            nv[j] = rl < rows ? c.vars[e] : -1;
            ni[j] = rl < rows ? c.row_info[r0 + rl] : 0u;
            nm[j] = (nv[j] >= 0 && iter > 1) ? msg[e] : (T)0;
          }
        };
        load(0);
        for (int b = 0; b < c.blocks; b++) {
          const int r0 = c.block_start[b], rows = c.block_start[b + 1] - r0;
          int vv[R];
          T x[R], t[R], pre[R];
          uint32_t info[R];
          // ---- phase 1
#pragma unroll
          for (int j = 0; j < R; j++) {
            const int rl = (tid + j * NT) / G;
            const T old = nm[j];
            vv[j] = nv[j];
            info[j] = ni[j];
            const int d = (int)(info[j] & 63u);
            const bool linked = (info[j] & kChainLinkIn) != 0 && k == d - 2;
            x[j] = linked || vv[j] < 0 ? (T)0 : sub_rn(post[vv[j]], old);
            if constexpr (SPA) {
              t[j] = vv[j] < 0 || linked ? (T)1 : tanh_t(mul_rn(x[j], (T)0.5));
              // the scan; lane d - 2 keeps the factors that it multiplies onto its value
              T inc = t[j], f[5];
#pragma unroll
              for (int s = 0; s < 5; s++) {
                f[s] = (T)1;
                if ((1 << s) < G) {
                  const T u = __shfl_up_sync(kFull, inc, 1 << s, G);
                  if (k >= (1 << s)) {
                    f[s] = u;
                    inc = mul_rn(u, inc);
                  }
                }
              }
              const T exc = __shfl_up_sync(kFull, inc, 1, G);
              pre[j] = k == 0 ? (T)1 : exc;
              if (rl < rows && (k == d - 2 || (d == 1 && k == 0))) {
#pragma unroll
                for (int s = 0; s < 5; s++) s_row[rl].f[s] = d == 1 ? (T)1 : f[s];
              }
            } else {
              // smallest magnitude and sign of the edges before the last two
              t[j] = pre[j] = (T)0;
              const bool in = vv[j] >= 0 && k < d - 2;
              T m = in && fabs(x[j]) < infinity<T>() ? fabs(x[j]) : infinity<T>();
              int neg = in && x[j] < (T)0;
#pragma unroll
              for (int o = G / 2; o > 0; o >>= 1) {
                const T om = __shfl_xor_sync(kFull, m, o, G);
                neg ^= __shfl_xor_sync(kFull, neg, o, G);
                m = om < m ? om : m;
              }
              if (rl < rows && k == 0) {
                s_row[rl].f[0] = m;
                s_row[rl].f[1] = neg ? (T)-1 : (T)1;
              }
            }
            if (rl < rows) {
              if (k == d - 2) s_row[rl].xl = linked ? old : x[j];
              if (k == d - 1) s_row[rl].xr = x[j];
            }
          }
          if (b + 1 < c.blocks) load(b + 1);
          __syncthreads();
          // ---- phase 2: the chain, a row per thread of the first two warps
          if (tid < kChainBlockRows) {
            const int rl = tid;
            const uint32_t ri = rl < rows ? c.row_info[r0 + rl] : 0u;
            const int d = (int)(ri & 63u);
            const bool linked = (ri & kChainLinkIn) != 0, left = d >= 2, feeds = (ri & kChainLinkOut) != 0;
            T f[5], tl, out;
#pragma unroll
            for (int s = 0; s < 5; s++) f[s] = rl < rows ? s_row[rl].f[s] : (T)1;
            const T xl = left ? s_row[rl].xl : (T)0, xr = d >= 1 ? s_row[rl].xr : (T)0;
            // the first guess: every row leaves its last variable as it is
            const size_t e = (size_t)(r0 + rl) * G + d;
            T in = linked ? post[c.vars[e - 2]] : (T)0;
            T handed = feeds ? post[c.vars[e - 1]] : (T)0;  // what this row's follower uses
            T xi;
            for (int sweep = 0;; sweep++) {
              xi = linked ? sub_rn(in, xl) : xl;
              out = chain_message<T, SPA, G>(f, xi, left, alpha, oms, tl);
              const T next = add_rn(xr, out);
              s_next[sweep & 1][rl + 1] = next;
              const bool same = !feeds || same_bits(next, handed);
              handed = next;
              if (chain_all(same) || sweep >= kChainBlockRows) break;
              if (linked) in = s_next[sweep & 1][rl];
            }
            if (rl < rows) {
              s_row[rl].xl = xi;
              s_row[rl].tl = tl;
              s_row[rl].outr = out;
            }
          }
          __syncthreads();
          // ---- phase 3
#pragma unroll
          for (int j = 0; j < R; j++) {
            const int rl = (tid + j * NT) / G;
            const int d = (int)(info[j] & 63u);
            if ((info[j] & kChainLinkIn) != 0 && k == d - 2) {
              x[j] = s_row[rl].xl;
              t[j] = s_row[rl].tl;
            }
            T o;
            if constexpr (SPA) {
              T inc = t[j];
#pragma unroll
              for (int s = 1; s < G; s <<= 1) {
                const T u = __shfl_down_sync(kFull, inc, s, G);
                if (k + s < G) inc = mul_rn(u, inc);
              }
              const T exc = __shfl_down_sync(kFull, inc, 1, G);
              o = k == d - 1 ? s_row[rl].outr : twice_atanh_t(mul_rn(pre[j], k == G - 1 ? (T)1 : exc));
            } else {
              // minimum, its first edge and second minimum of the whole row (sparse.cu)
              const T av = fabs(x[j]);
              const bool in = vv[j] >= 0;
              int neg = in && x[j] < (T)0;
              const bool fin = in && av < infinity<T>();
              T m1 = fin ? av : infinity<T>(), m2 = infinity<T>();
              int i1 = fin ? k : 0x7fffffff;
#pragma unroll
              for (int w = G / 2; w > 0; w >>= 1) {
                const T bm1 = __shfl_xor_sync(kFull, m1, w, G), bm2 = __shfl_xor_sync(kFull, m2, w, G);
                const int bi1 = __shfl_xor_sync(kFull, i1, w, G);
                neg ^= __shfl_xor_sync(kFull, neg, w, G);
                const bool mine = m1 < bm1 || (m1 == bm1 && i1 < bi1);
                const T w2 = mine ? m2 : bm2, l1 = mine ? bm1 : m1;
                m1 = mine ? m1 : bm1;
                i1 = mine ? i1 : bi1;
                m2 = w2 < l1 ? w2 : l1;
              }
              const T s = mul_rn(neg ? (T)-1 : (T)1, x[j] < (T)0 ? (T)-1 : (T)1);
              o = mul_rn(s, scaled_mag(k == i1 ? m2 : m1, alpha, oms));
            }
            if (vv[j] >= 0) {
              msg[(size_t)(r0 + rl) * G + k] = o;
              // a last variable that the next row takes over is written by that row
              if (!((info[j] & kChainLinkOut) != 0 && k == d - 1)) post[vv[j]] = add_rn(x[j], o);
            }
          }
          __syncthreads();
        }
        if (!some_row_fails()) {
          it = iter;
          break;
        }
      }
    }
    if (a.post_out)
      for (int v = tid; v < c.n; v += NT) a.post_out[(size_t)cw * c.n + v] = post[v];
    if (tid == 0 && a.iters_out) a.iters_out[cw] = it;
    __syncthreads();
  }
}

template <typename T, bool SPA>
void* chain_kernel_for(int group) {
  if (group == 8) return (void*)sparse_chain_kernel<T, SPA, 8, 256>;
  if (group == 16) return (void*)sparse_chain_kernel<T, SPA, 16, 512>;
  return (void*)sparse_chain_kernel<T, SPA, 32, 512>;
}

}  // namespace

int sparse_chain_threads(int group) { return group == 8 ? 256 : 512; }

void* sparse_chain_kernel_ptr(int precision, int rule, int group) {
  const bool spa = rule == cbd::RULE_SUM_PRODUCT;
  if (precision == 0) return spa ? chain_kernel_for<double, true>(group) : chain_kernel_for<double, false>(group);
  return spa ? chain_kernel_for<float, true>(group) : chain_kernel_for<float, false>(group);
}

}  // namespace cbk
