// Learned (neural) min-sum: the layered min-sum of decode.cu with a scale and an offset
// per iteration and per edge, trained by hand-written reverse-mode differentiation of
// the unrolled iterations.  No counterpart in the reference; the plain normalised
// min-sum is its special case alpha = 0.75, beta = 0 and remains its fallback.
//
// Check message at iteration t, edge e of a row (the row's other edges k != e):
//   y_e = s_e * max(alpha[t, e] * m_e - beta[t, e], 0)  (the product and the difference
//   rounded once, as one fused multiply-add),
//   s_e = prod sign(x_k), m_e = min |x_k|, x_k = post[v_k] - c2v_k (ldpc.rs:468-491),
// then post[v_e] = x_e + y_e and c2v_e = y_e.  Weights are indexed [t][entry][r] (one per
// lifted edge) or [t][entry] (one per base-graph edge, shared across Z); the edge
// storage is [entry][r], so a layer's Z threads touch consecutive words.
//
// Training loss: the mean over frames and over the codeword bits [0, loss_bits) (all n_full
// bits, or the K' information bits) of softplus(-(1 - 2 c_v) post_v), the binary
// cross-entropy of the soft output: of the
// last iteration, or (multi-loss) a weighted mean over the outputs of all T iterations,
// whose posteriors the forward then saves: weights 1/T, or a ramp 2(t+1)/(T(T+1)).
// Backward: for t = T-1..0 and the layers in reverse, each row recomputes its forward
// quantities from its saved record and propagates
//   g_y = g_post[v] + g_c2v, g_a = g_y s [a > 0], dL/dalpha += g_a m, dL/dbeta -= g_a,
//   g_m = g_a alpha flows to |x| of the argmin (or of the second argmin for the argmin),
//   g_x = g_post[v] + sign(x) g_|x|, then g_post[v] = g_x and g_c2v = -g_x.
//
// The tape.  Everything the backward pass needs of a row is a function of its smallest and
// second smallest |x|, their edges and the signs of x, so the forward pass saves these, 12
// bytes a row and iteration (a plane of the two magnitudes, a plane of meta words), instead
// of x itself, 4 bytes an edge (BG1: 27 bytes a row), and reads the previous iteration's
// record where it kept the messages before: y follows from it and the previous iteration's
// weights, the same bits.
//
// Rows from c.rows_live on (cbh::live_rows: their own parity column is not sent and in no
// other row) send the other variables zero while their offsets are not negative, which
// learned_live_kernel tests before each pass over the frames.  Such a row is then only what
// it makes of its own column, m the smallest |post| of its other variables:
//   post_own = s max(alpha m - beta, 0)
// (a frame whose magnitudes approach infinity runs again with every row, beyond_skipping),
// and backward the gradient of post_own's own loss, through alpha m, onto m's variable.  Its
// record is m, m's variable and two signs.  (Half of base graph 1's rows at rate 1/2, three
// quarters of base graph 2's: 61 % of its edges.)
//
// Bound: forward, issue (57-65 %); backward, the latency of the message gradients, 4 bytes
// an edge read and written per iteration, more than L2 holds for BG1's resident frames.
// Measured on GB300, shared weights: a step of 512 frames of BG1 Z = 384, 8 iterations, 10.3
// -> 3.3 ms (forward 3.57, backward 6.52 before; 1.43 and 2.15 with every row run); 1024
// frames of BG2 Z = 52, 10 iterations, forward 0.98 -> 0.36 ms (0.46 with every row) and
// backward 1.78 -> 0.44 (0.67).  Before: x on the tape, messages and weights read from global memory
// in the rows, ten shuffles per edge for the weight gradients and their sums by shared-memory
// atomics.  Loading the next row's message gradients ahead, in registers, measured 5-10 %
// slower.
#include <cuda_runtime.h>

#include <cmath>

#include "decode_common.cuh"
#include "kernels.h"

namespace cbk {
namespace {

constexpr unsigned kFull = 0xffffffffu;
// the edges of a level at most (the dense core rows of base graph 1)
constexpr int kMaxLevelEdges = 19;
constexpr int kOwnGroup = 8;  // skipped rows whose gradients are summed together
// meta word: bits 0-4 the first edge of the smallest |x| (0 when that is infinite), bits
// 5-9 that of the second smallest (likewise), bits 31, 30, .. the signs of x of edges 0, 1, ..
constexpr uint32_t kMetaSigns = 0xffffe000u;

// weight of iteration t's output in the multi-loss: 1/T each (mode 1), or a linear ramp
// 2 (t + 1) / (T (T + 1)) that leans on the last iterations (mode 2)
__device__ __forceinline__ float iter_loss_weight(int mode, int t, int T) {
  return mode == 2 ? 2.f * (float)(t + 1) / ((float)T * (float)(T + 1)) : 1.f / (float)T;
}

__device__ __forceinline__ float softplus_f(float x) { return x > 0.f ? x + log1pf(__expf(-x)) : log1pf(__expf(x)); }
__device__ __forceinline__ float sigmoid_f(float x) { return 1.f / (1.f + __expf(-x)); }

// the records of one frame and iteration: {m1, m2} per lifted row, then the meta words
struct Tape {
  float2* mag;
  uint32_t* meta;
  __device__ __forceinline__ Tape(unsigned char* base, int lifted)
      : mag(reinterpret_cast<float2*>(base)), meta(reinterpret_cast<uint32_t*>(base + (size_t)lifted * 8)) {}
};

// the posteriors (or their gradients) at the start of a kernel's shared memory
__host__ __device__ inline size_t learned_post_bytes(int n_full) { return ((size_t)n_full * 4 + 15) & ~(size_t)15; }

// The (scale, offset) of entry i for lifted row r in one iteration: shared weights staged
// in shared memory as pairs, or one per lifted edge in global memory.  `none`: the iteration
// before the first, whose scale 0 and offset +inf make every message 0.
template <bool SHARED>
struct RowWeights;
template <>
struct RowWeights<true> {
  const float2* w;
  __device__ __forceinline__ float2 at(int i, int, int) const { return w[i]; }
};
template <>
struct RowWeights<false> {
  const float *al, *be;
  bool none;
  __device__ __forceinline__ float2 at(int i, int z, int r) const {
    const size_t k = (size_t)i * z + r;
    return none ? make_float2(0.f, INFINITY) : make_float2(al[k], be[k]);
  }
};

// The magnitude max(alpha m - beta, 0) of a message.  A zero's sign is of no account: it is
// added to or subtracted from posteriors that are never -0.0 (they start as 0.0 + LLR or 30.0).
__device__ __forceinline__ float learned_mag(float2 w, float m) { return fmaxf(__fmaf_rn(w.x, m, -w.y), 0.f); }

// bit 31 of a word of signs shifted left by an edge's number, on a value
__device__ __forceinline__ float flip_sign(float v, uint32_t signs) {
  return __uint_as_float(__float_as_uint(v) ^ (signs & 0x80000000u));
}

// forward of one lifted row, degree D, entries s0 ..; (o, om) the previous iteration's
// record, wp and wc the previous and this iteration's weights
template <int D, bool SHARED>
__device__ __forceinline__ void learned_row_fwd(const LearnedArgs& a, float* post, int s0, int r, int z,
                                                const RowWeights<SHARED>& wp, const RowWeights<SHARED>& wc, float2 o,
                                                uint32_t om, float2& n, uint32_t& nm) {
  const EdgeAddrTable addr{a.code.eaddr + s0, r, 4 * r, 4 * z};
  int off[D];
  float x[D];
  const int oi1 = (int)(om & 31u);
  // the signs to add the old messages with: the opposite of the product of the others'
  const uint32_t os = (__popc(om & kMetaSigns) & 1) ? om : ~om;
#pragma unroll
  for (int e = 0; e < D; e++) {
    off[e] = addr(e);
    const float mag = learned_mag(wp.at(s0 + e, z, r), e == oi1 ? o.y : o.x);
    x[e] = __fadd_rn(ld_post(post, off[e]), flip_sign(mag, os << e));
  }
  // the two smallest magnitudes, two edges at a time (NaN counts as infinite)
  float m1 = INFINITY, m2 = INFINITY;
#pragma unroll
  for (int e = 0; e + 1 < D; e += 2) {
    const float p = fminf(fabsf(x[e]), INFINITY), q = fminf(fabsf(x[e + 1]), INFINITY);
    const float lo = fminf(p, q);
    m2 = min3f(m2, fmaxf(m1, lo), fmaxf(p, q));
    m1 = fminf(m1, lo);
  }
  if (D & 1) {
    const float p = fminf(fabsf(x[D - 1]), INFINITY);
    m2 = fminf(m2, fmaxf(m1, p));
    m1 = fminf(m1, p);
  }
  uint32_t sg = 0, at1 = 0, at2 = 0;
#pragma unroll
  for (int e = 0; e < D; e++) {
    sg = __funnelshift_l(__float_as_uint(x[e]), sg, 1);
    if (fabsf(x[e]) == m2) at2 |= 1u << e;
  }
  sg <<= 32 - D;
  const uint32_t ns = (__popc(sg) & 1) ? ~sg : sg;  // the product of the other signs
#pragma unroll
  for (int e = 0; e < D; e++) {
    const bool first = fabsf(x[e]) == m1;  // (on a tie m1 = m2)
    if (first) at1 |= 1u << e;
    const float mag = learned_mag(wc.at(s0 + e, z, r), first ? m2 : m1);
    st_post(post, off[e], __fadd_rn(x[e], flip_sign(mag, ns << e)));
  }
  // their first edges, as a scan with strict comparisons finds them
  const uint32_t rest = m1 == m2 ? at1 & (at1 - 1) : at2;
  const uint32_t i1 = m1 < INFINITY ? __ffs(at1) - 1 : 0, i2 = m2 < INFINITY ? __ffs(rest) - 1 : 0;
  n = make_float2(m1, m2);
  nm = i1 | i2 << 5 | sg;
}

// The sums of N values over the warp's lanes in about N + 5 shuffles: each step halves
// the values a lane holds, the lanes of one half keeping the first half's sums and the others
// the second's.  Lane l is left with v[j] = the sum of value index(j), j < (N + 31) / 32.
template <int N, int O>
struct WarpSums {
  static constexpr int H = (N + 1) / 2;
  using Next = WarpSums<H, O / 2>;
  static constexpr int left = Next::left;
  static __device__ __forceinline__ void sum(float* v, int lane) {
    const bool up = (lane & O) != 0;
#pragma unroll
    for (int i = 0; i < H; i++) {
      if (i + H < N) {
        const float send = up ? v[i] : v[i + H], keep = up ? v[i + H] : v[i];
        v[i] = keep + __shfl_xor_sync(kFull, send, O);
      } else {
        v[i] += __shfl_xor_sync(kFull, v[i], O);
      }
    }
    Next::sum(v, lane);
  }
  // the value that slot j of this lane sums, -1 for a copy of another lane's
  static __device__ __forceinline__ int index(int j, int lane) {
    const int i = Next::index(j, lane);
    if (i < 0) return -1;
    if ((lane & O) == 0) return i;
    return i + H < N ? i + H : -1;
  }
};
template <int N>
struct WarpSums<N, 0> {
  static constexpr int left = N;
  static __device__ __forceinline__ void sum(float*, int) {}
  static __device__ __forceinline__ int index(int j, int) { return j; }
};

// the warp's sums of N values to red[0], red[1], ..
template <int N>
__device__ __forceinline__ void put_warp_sums(float (&v)[N], float* red, int lane) {
  using Sums = WarpSums<N, 16>;
  Sums::sum(v, lane);
#pragma unroll
  for (int j = 0; j < Sums::left; j++) {
    const int i = Sums::index(j, lane);
    if (i >= 0) red[i] = v[j];
  }
}

// Backward of one lifted row from its record.  `gr` points at the row's message gradients, S
// floats from edge to edge (a constant, so that their addresses are immediates; 0: z, with weights
// per lifted edge, whose atomics hide it).  With
// shared weights `red` receives the warp's sums of the gradients: D scales, then D offsets with the
// opposite sign (every lane of the warp takes part; the lanes without a row with zeros).
template <int D, bool SHARED, int S>
__device__ __forceinline__ void learned_row_bwd(const LearnedArgs& a, float* gp, float* gr, float2 n, uint32_t nm,
                                                int t, int s0, int r, int z, bool active, bool last,
                                                const RowWeights<SHARED>& w, float* red, int lane) {
  const int i1 = (int)(nm & 31u), st = S ? S : z;
  float ga[D];  // the gradients of max(alpha m - beta, 0): of the offsets, negated
  if (active) {
    const EdgeAddrTable addr{a.code.eaddr + s0, r, 4 * r, 4 * z};
    int off[D];
    int i2 = (int)((nm >> 5) & 31u);
    const uint32_t sg = nm & kMetaSigns, ns = (__popc(sg) & 1) ? ~sg : sg;
#pragma unroll
    for (int e = 0; e < D; e++) ga[e] = last ? 0.f : gr[e * st];
    float g1 = 0.f, g2 = 0.f;  // gradients of |x_i1| and |x_i2|
#pragma unroll
    for (int e = 0; e < D; e++) {
      off[e] = addr(e);
      const float gy = ld_post(gp, off[e]) + ga[e];
      const float2 ab = w.at(s0 + e, z, r);
      const bool min = e == i1;
      const float m = min ? n.y : n.x;
      ga[e] = __fmaf_rn(ab.x, m, -ab.y) > 0.f ? flip_sign(gy, ns << e) : 0.f;
      if constexpr (!SHARED) {
        const size_t k = ((size_t)t * a.code.n_entries + s0 + e) * z + r;
        atomicAdd(&a.g_alpha[k], ga[e] * m);
        atomicAdd(&a.g_beta[k], -ga[e]);
      }
      const float gm = ga[e] * ab.x;
      if (min) g2 = gm;
      else g1 += gm;
    }
    // only the two smallest inputs' posteriors receive a gradient: x = post - c2v there
    // adds sign(x) g_|x|, everywhere else the row leaves the posterior's gradient as it is
    g1 = flip_sign(g1, sg << i1);
    g2 = flip_sign(g2, sg << i2);
    if (i2 == i1) i2 = 31;
#pragma unroll
    for (int e = 0; e < D; e++) {
      const bool at1 = e == i1, at2 = e == i2;
      const float gx = ld_post(gp, off[e]) + (at1 ? g1 : at2 ? g2 : 0.f);
      if (at1 || at2) st_post(gp, off[e], gx);
      if (t > 0) gr[e * st] = -gx;
    }
  } else {
#pragma unroll
    for (int e = 0; e < D; e++) ga[e] = 0.f;
  }
  if constexpr (SHARED) {
    if constexpr (D <= 10) {
      float v[2 * D];
#pragma unroll
      for (int e = 0; e < D; e++) {
        v[e] = ga[e] * (e == i1 ? n.y : n.x);
        v[D + e] = ga[e];
      }
      put_warp_sums(v, red, lane);
    } else {  // (two sums: 2 D values at once spill)
      float v[D];
#pragma unroll
      for (int e = 0; e < D; e++) v[e] = ga[e] * (e == i1 ? n.y : n.x);
      put_warp_sums(v, red, lane);
      put_warp_sums(ga, red + D, lane);
    }
  }
}

// forward of one row that only makes its own column: lifted row r of entries [s0, s0 + d), own = the
// last one, with its weights w
__device__ __forceinline__ void own_column_fwd(const LearnedArgs& a, float* post, int s0, int d, int r, int z, float2 w,
                                               float2& n, uint32_t& nm) {
  const EdgeAddrTable addr{a.code.eaddr + s0, r, 4 * r, 4 * z};
  float m = INFINITY;
  int at = addr(0);
  uint32_t neg = 0, neg_at = 0;
  for (int e = 0; e + 1 < d; e++) {
    const int o = addr(e);
    const float x = ld_post(post, o), av = fabsf(x);
    const uint32_t s = x < 0.f;
    neg ^= s;
    if (av < m || e == 0) neg_at = s;
    if (av < m) {
      m = av;
      at = o;
    }
  }
  const float y = learned_mag(w, m);
  st_post(post, addr(d - 1), __fadd_rn(0.f, neg ? -y : y));
  n = make_float2(__int_as_float(at), m);
  nm = neg | neg_at << 1;
}

// *live: the rows that a pass with shared weights runs: c.rows_live, or all when a skipped row
// has a negative offset on another edge than its own column's, or there weights that could make
// a magnitude below beyond_skipping's bound infinite
__global__ void __launch_bounds__(256) learned_live_kernel(const __grid_constant__ LearnedArgs a) {
  const cbd::DevCode& c = a.code;
  const int first = c.layer_start[c.rows_live], count = c.n_entries - first;
  int bad = 0;
  for (int i = threadIdx.x; i < a.T * count; i += blockDim.x) {
    const int t = i / count, e = first + i - t * count;
    const size_t w = (size_t)t * c.n_entries + e;
    bool own = false;
    for (int L = c.rows_live; L < c.rows_n; L++) own = own || e + 1 == c.layer_start[L + 1];
    if (own ? !cbd::skippable_own_weights(a.alpha[w], a.beta[w]) : a.beta[w] < 0.f) bad = 1;
  }
  bad = __syncthreads_or(bad);
  if (threadIdx.x == 0) *a.live = bad ? c.rows_n : c.rows_live;
}

#define CB_LEARNED_DEGREES(ROW) \
  switch (d) {                  \
    case 3: ROW(3) break;       \
    case 4: ROW(4) break;       \
    case 5: ROW(5) break;       \
    case 6: ROW(6) break;       \
    case 7: ROW(7) break;       \
    case 8: ROW(8) break;       \
    case 9: ROW(9) break;       \
    case 10: ROW(10) break;     \
    default: ROW(19) break;     \
  }

// the weights of iteration t: staged in `buf` (shared; visible after the caller's next
// barrier) or in global memory
template <bool SHARED>
__device__ __forceinline__ RowWeights<SHARED> iteration_weights(const LearnedArgs& a, float2* buf, int t) {
  const int ne = a.code.n_entries;
  if constexpr (SHARED) {
    for (int i = threadIdx.x; i < ne; i += blockDim.x)
      buf[i] = make_float2(a.alpha[(size_t)t * ne + i], a.beta[(size_t)t * ne + i]);
    return {buf};
  } else {
    const size_t per = (size_t)ne * a.code.z;
    return {a.alpha + t * per, a.beta + t * per, false};
  }
}

template <bool SHARED>
__global__ void __launch_bounds__(384, 2) learned_forward_kernel(const __grid_constant__ LearnedArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const cbd::DevCode& c = a.code;
  const int z = c.z, nt = blockDim.x, tid = threadIdx.x;
  const int ne = c.n_entries, lifted = c.rows_n * z;
  float* post = reinterpret_cast<float*>(smem);
  float2* wbuf = reinterpret_cast<float2*>(smem + learned_post_bytes(c.n_full));  // two iterations' (shared)
  __shared__ float s_loss;
  __shared__ int s_wide;  // the frame left the magnitudes in which rows may be skipped
  const long long f = blockIdx.x;
  if (f >= a.n_frames) return;
  if (tid == 0) {
    s_loss = 0.f;
    s_wide = 0;
  }
  int live = SHARED ? *a.live : c.rows_n;
  unsigned char* tape = a.tape + (size_t)f * a.tape_frame;
  const float* llr = a.llr + (size_t)f * c.e;
again:
  for (int v = tid; v < c.n_full; v += nt) post[v] = 0.f;
  __syncthreads();
  Widest<float> widest;
  auto put = [&](int v, float l) {
    const float x = __fadd_rn(0.f, l);
    if constexpr (SHARED) widest.add(x);
    post[v] = x;
  };
  if (c.map_is_offset) {
    for (int t = tid; t < c.e; t += nt) put(2 * z + t, llr[t]);
  } else if (!c.has_repeats) {
    for (int t = tid; t < c.e; t += nt) put(c.map[t], llr[t]);
  } else {
    for (int v = tid; v < c.n_full; v += nt) {
      int b0 = c.inv_start[v], b1 = c.inv_start[v + 1];
      if (b0 == b1) continue;
      float s = 0.f;
      for (int i = b0; i < b1; i++) s = __fadd_rn(s, llr[c.inv_t[i]]);
      put(v, s);
    }
  }
  if (SHARED && widest.beyond()) s_wide = 1;
  __syncthreads();
  for (int v = c.k_info + tid; v < c.k; v += nt) post[v] = cbd::kKnownBitLlr;
  __syncthreads();
  const bool multi = a.multi_loss && a.P && a.cw_bits && a.loss;
  const bool active = tid < z;
  const int run = live < c.rows_n ? c.rows_run : c.rows_n;
  float lsum = 0.f;  // this thread's share of the loss
  // before the first iteration there are no messages: weights that make them 0
  RowWeights<SHARED> wp, wc;
  if constexpr (SHARED) {
    wc = {wbuf + ne};
    for (int i = tid; i < ne; i += nt) wbuf[ne + i] = make_float2(0.f, INFINITY);
  } else {
    wc = {a.alpha, a.beta, true};
  }
  for (int t = 0; t < a.T; t++) {
    wp = wc;
    wc = iteration_weights<SHARED>(a, wbuf + (t & 1) * ne, t);
    __syncthreads();
    if (SHARED && live < c.rows_n && s_wide) {
      live = c.rows_n;
      __syncthreads();
      goto again;
    }
    const Tape old(tape + (t > 0 ? (size_t)(t - 1) * a.tape_iter : 0), lifted);
    const Tape cur(tape + (size_t)t * a.tape_iter, lifted);
    // the next row's old record is loaded a row ahead
    float2 o = make_float2(0.f, 0.f);
    uint32_t om = 0;
    if (active && t > 0) {
      const int i = c.layer_order[0] * z + tid;
      o = old.mag[i];
      om = old.meta[i];
    }
    for (int q = 0; q < run; q++) {
      const int L = c.layer_order[q];
      float2 on = o;
      uint32_t omn = om;
      if (active && t > 0 && q + 1 < run) {
        const int i = c.layer_order[q + 1] * z + tid;
        on = old.mag[i];
        omn = old.meta[i];
      }
      if (active && L < live) {  // (a skipped row may share the last live level)
        const int s0 = c.layer_start[L], d = c.layer_start[L + 1] - s0;
        float2 n;
        uint32_t nm;
#define CB_ROW(DD) learned_row_fwd<DD, SHARED>(a, post, s0, tid, z, wp, wc, o, om, n, nm);
        CB_LEARNED_DEGREES(CB_ROW)
#undef CB_ROW
        cur.mag[L * z + tid] = n;
        cur.meta[L * z + tid] = nm;
      }
      o = on;
      om = omn;
      if (c.level_end[q]) __syncthreads();
    }
    if (SHARED && live < c.rows_n && active && beyond_skipping(post, tid, z, c.bg)) s_wide = 1;
    // the skipped rows' own columns, where the loss or the output reads them
    if (SHARED && live < c.rows_n && (t == a.T - 1 || (multi && a.loss_bits > (c.cols_k + live) * z))) {
      if (active) {
        for (int L = live; L < c.rows_n; L++) {
          const int s0 = c.layer_start[L], s1 = c.layer_start[L + 1];
          float2 n;
          uint32_t nm;
          own_column_fwd(a, post, s0, s1 - s0, tid, z, wc.at(s1 - 1, z, tid), n, nm);
          cur.mag[L * z + tid] = n;
          cur.meta[L * z + tid] = nm;
        }
      }
      __syncthreads();
    }
    if (multi) {
      const int wpc = (c.n_full + 31) >> 5;
      const float wt = iter_loss_weight(a.multi_loss, t, a.T);
      float* Pt = a.P + ((size_t)f * a.T + t) * c.n_full;
      for (int v = tid; v < a.loss_bits; v += nt) {
        Pt[v] = post[v];
        int bit = (a.cw_bits[(size_t)f * wpc + (v >> 5)] >> (v & 31)) & 1;
        lsum += softplus_f(bit ? post[v] : -post[v]) * wt;
      }
    }
  }
  // outputs
  if (SHARED && tid == 0) a.frame_live[f] = live;
  if (a.post_out)
    for (int v = tid; v < c.n_full; v += nt) a.post_out[(size_t)f * c.n_full + v] = post[v];
  if (a.cw_bits && a.loss) {
    if (!multi) {
      const int wpc = (c.n_full + 31) >> 5;
      for (int v = tid; v < a.loss_bits; v += nt) {
        int bit = (a.cw_bits[(size_t)f * wpc + (v >> 5)] >> (v & 31)) & 1;
        lsum += softplus_f(bit ? post[v] : -post[v]);
      }
    }
    for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(kFull, lsum, o);
    if ((tid & 31) == 0) atomicAdd(&s_loss, lsum);
    __syncthreads();
    if (tid == 0) atomicAdd(a.loss, s_loss / (float)a.loss_bits);
  }
}

// Backward of the skipped rows' own columns at iteration t, kOwnGroup rows at a time: gp of an
// own column holds this iteration's loss gradient alone, and is cleared for the next one.  Returns
// the buffer of sums to use next.  (Out of line: inlined, its registers made the rows spill.)
__device__ __noinline__ int own_columns_bwd(const LearnedArgs& a, float* gp, Tape cur, int live, int t,
                                            const float2* w, float* red, int buf) {
  const cbd::DevCode& c = a.code;
  const int z = c.z, nt = blockDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  constexpr int RW = 2 * kMaxLevelEdges;
  const bool active = tid < z;
  for (int L0 = live; L0 < c.rows_n; L0 += kOwnGroup) {
    float v[2 * kOwnGroup];
    float2 n[kOwnGroup];
    uint32_t nm[kOwnGroup];
#pragma unroll
    for (int j = 0; j < kOwnGroup; j++) {
      n[j] = make_float2(0.f, 0.f);
      nm[j] = 0;
      if (active && L0 + j < c.rows_n) {
        n[j] = cur.mag[(L0 + j) * z + tid];
        nm[j] = cur.meta[(L0 + j) * z + tid];
      }
    }
#pragma unroll
    for (int j = 0; j < kOwnGroup; j++) {
      v[2 * j] = v[2 * j + 1] = 0.f;
      if (active && L0 + j < c.rows_n) {
        const float2 ab = w[c.layer_start[L0 + j + 1] - 1];
        float* own = gp + (c.cols_k + L0 + j) * z + tid;
        const float g = *own, m = n[j].y;
        *own = 0.f;
        const float ga = __fmaf_rn(ab.x, m, -ab.y) > 0.f ? ((nm[j] & 1u) ? -g : g) : 0.f;
        const float gm = ga * ab.x;
        v[2 * j] = ga * m;
        v[2 * j + 1] = ga;
        // (two rows may meet on a variable)
        atomicAdd(reinterpret_cast<float*>(reinterpret_cast<char*>(gp) + __float_as_int(n[j].x)),
                  (nm[j] & 2u) ? -gm : gm);
      }
    }
    put_warp_sums(v, red + ((size_t)buf * nw + warp) * RW, lane);
    __syncthreads();
    for (int i = tid; i < 2 * kOwnGroup; i += nt) {
      const int L = L0 + (i >> 1);
      if (L < c.rows_n) {
        const float* rd = red + (size_t)buf * nw * RW + i;
        float sum = 0.f;
        for (int k = 0; k < nw; k++) sum += rd[k * RW];
        const size_t wi = (size_t)t * c.n_entries + c.layer_start[L + 1] - 1;
        atomicAdd((i & 1) ? &a.g_beta[wi] : &a.g_alpha[wi], (i & 1) ? -sum : sum);
      }
    }
    buf ^= 1;
  }
  return buf;
}

template <bool SHARED, int S>
__global__ void __launch_bounds__(384, 2) learned_backward_kernel(const __grid_constant__ LearnedArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const cbd::DevCode& c = a.code;
  const int z = c.z, nt = blockDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  const int lifted = c.rows_n * z;
  float* gp = reinterpret_cast<float*>(smem);
  float2* wbuf = reinterpret_cast<float2*>(smem + learned_post_bytes(c.n_full));
  // the warps' sums of a level's weight gradients, in two buffers by turns (shared weights)
  float* red = reinterpret_cast<float*>(wbuf + c.n_entries);
  constexpr int RW = 2 * kMaxLevelEdges;
  const long long f = blockIdx.x;
  if (f >= a.n_frames) return;
  const int st = S ? S : z;
  float* gc = a.c2v + (size_t)f * c.n_entries * st + tid;  // this thread's message gradients
  const int wpc = (c.n_full + 31) >> 5;
  const bool multi = a.multi_loss && a.P;
  const bool active = tid < z;
  const int live = SHARED ? a.frame_live[f] : c.rows_n, run = live < c.rows_n ? c.rows_run : c.rows_n;
  const bool own_loss = live < c.rows_n && a.loss_bits > (c.cols_k + live) * z;  // on a skipped row's column
  const float scale = 1.f / ((float)a.loss_bits * (float)a.n_frames);
  for (int v = tid; v < c.n_full; v += nt) gp[v] = 0.f;
  __syncthreads();
  int buf = 0;
  for (int t = a.T - 1; t >= 0; t--) {
    const RowWeights<SHARED> w = iteration_weights<SHARED>(a, wbuf, t);
    // the loss of iteration t's output (every iteration, or the last one)
    if (multi || t == a.T - 1) {
      const float* p = multi ? a.P + ((size_t)f * a.T + t) * c.n_full : a.post_out + (size_t)f * c.n_full;
      const float sc = multi ? scale * iter_loss_weight(a.multi_loss, t, a.T) : scale;
      // eight posteriors in flight: one at a time, their latency was a third of the kernel
      constexpr int U = 8;
      for (int v0 = tid; v0 < a.loss_bits; v0 += U * nt) {
        float q[U];
        uint32_t cw[U];
#pragma unroll
        for (int j = 0; j < U; j++) {
          const int v = v0 + j * nt;
          q[j] = v < a.loss_bits ? p[v] : 0.f;
          cw[j] = v < a.loss_bits ? a.cw_bits[(size_t)f * wpc + (v >> 5)] : 0u;
        }
#pragma unroll
        for (int j = 0; j < U; j++) {
          const int v = v0 + j * nt;
          if (v >= a.loss_bits) break;
          const float sgn = ((cw[j] >> (v & 31)) & 1) ? -1.f : 1.f;
          gp[v] += -sgn * sigmoid_f(-sgn * q[j]) * sc;
        }
      }
    }
    __syncthreads();
    const Tape cur(a.tape + (size_t)f * a.tape_frame + (size_t)t * a.tape_iter, lifted);
    // the next row's record is loaded a row ahead: zeros for a skipped row that shares the last
    // live level, whose record the forward pass does not write in every iteration (the
    // level's sums form 0 times the record's magnitudes, NaN if they were infinite)
    float2 n;
    uint32_t nm;
    auto record = [&](int q, float2& mag, uint32_t& meta) {
      mag = make_float2(0.f, 0.f);
      meta = 0;
      const int L = c.layer_order[q];
      if (active && L < live) {
        mag = cur.mag[L * z + tid];
        meta = cur.meta[L * z + tid];
      }
    };
    record(run - 1, n, nm);
    // the skipped rows, the last of the forward pass
    if constexpr (SHARED) {
      if (own_loss && (multi || t == a.T - 1)) buf = own_columns_bwd(a, gp, cur, live, t, wbuf, red, buf);
    }
    for (int q = run - 1; q >= 0;) {
      // the rows of a level, then a barrier, then the level's sums into the gradients
      int at = 0, qe = q;
      do {
        const int L = c.layer_order[qe];
        const int s0 = c.layer_start[L], d = c.layer_start[L + 1] - s0;
        float2 nn = n;
        uint32_t nmn = nm;
        if (qe > 0) record(qe - 1, nn, nmn);
        float* rd = red + ((size_t)buf * nw + warp) * RW + 2 * at;
#define CB_ROW(DD)                                                                                                 \
  learned_row_bwd<DD, SHARED, S>(a, gp, gc + (size_t)s0 * st, n, nm, t, s0, tid, z, active && L < live, t == a.T - 1, w, rd, lane);
        CB_LEARNED_DEGREES(CB_ROW)
#undef CB_ROW
        n = nn;
        nm = nmn;
        at += d;
        qe--;
      } while (qe >= 0 && !c.level_end[qe]);
      __syncthreads();
      if constexpr (SHARED) {
        for (int base = 0; q > qe; q--) {
          const int L = c.layer_order[q];
          const int s0 = c.layer_start[L], d = c.layer_start[L + 1] - s0;
          for (int i = tid; i < 2 * d; i += nt) {
            const float* rd = red + (size_t)buf * nw * RW + 2 * base + i;
            float s = 0.f;
            for (int k = 0; k < nw; k++) s += rd[k * RW];
            const size_t wi = (size_t)t * c.n_entries + s0 + (i < d ? i : i - d);
            atomicAdd(i < d ? &a.g_alpha[wi] : &a.g_beta[wi], i < d ? s : -s);
          }
          base += d;
        }
        buf ^= 1;
      }
      q = qe;
    }
  }
}

// Codeword bytes (bit 0 counts) to packed words, a warp per word and step.  The host loop over
// the bits took 10 ms for 1024 words of 2704 bits, this 0.01.
__global__ void __launch_bounds__(256) pack_codewords_kernel(const uint8_t* bytes, uint32_t* words, int64_t n_frames,
                                                             int n_bits) {
  const int wpc = (n_bits + 31) >> 5, lane = threadIdx.x & 31;
  const int64_t total = n_frames * wpc, step = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t w = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); w < total; w += step) {
    const int64_t f = w / wpc;
    const int v = (int)(w - f * wpc) * 32 + lane;
    const uint32_t word = __ballot_sync(kFull, v < n_bits && (bytes[f * n_bits + v] & 1));
    if (lane == 0) words[w] = word;
  }
}

// Adam (Kingma & Ba, 2015) on the scales and offsets
__global__ void adam_kernel(float* w, const float* g, float* m, float* v, int64_t n, float lr, float b1, float b2,
                            float eps, float c1, float c2) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    float gi = g[i];
    float mi = b1 * m[i] + (1.f - b1) * gi;
    float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  }
}

}  // namespace

cudaError_t launch_learned(const LearnedArgs& a, bool forward, cudaStream_t s) {
  if (forward && a.shared) {
    learned_live_kernel<<<1, 256, 0, s>>>(a);
    if (cudaError_t e = cudaGetLastError()) return e;
  }
  const int threads = ((a.code.z + 31) / 32) * 32;
  void* k;
  if (!forward && !a.shared) {
    k = (void*)learned_backward_kernel<false, 0>;
  } else if (forward) {
    k = a.shared ? (void*)learned_forward_kernel<true> : (void*)learned_forward_kernel<false>;
  } else {
    switch (learned_stride(a.code, a.shared)) {
      case 16: k = (void*)learned_backward_kernel<true, 16>; break;
      case 32: k = (void*)learned_backward_kernel<true, 32>; break;
      case 64: k = (void*)learned_backward_kernel<true, 64>; break;
      case 128: k = (void*)learned_backward_kernel<true, 128>; break;
      case 256: k = (void*)learned_backward_kernel<true, 256>; break;
      case 384: k = (void*)learned_backward_kernel<true, 384>; break;
      default: return cudaErrorInvalidValue;
    }
  }
  size_t smem = learned_post_bytes(a.code.n_full);
  if (a.shared)
    smem += forward ? 2 * sizeof(float2) * a.code.n_entries
                    : sizeof(float2) * a.code.n_entries + 2 * (size_t)(threads / 32) * 2 * kMaxLevelEdges * sizeof(float);
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  void* args[] = {(void*)&a};
  return cudaLaunchKernel(k, dim3((unsigned)a.n_frames), dim3(threads), args, smem, s);
}

cudaError_t launch_pack_codewords(const uint8_t* bytes, uint32_t* words, int64_t n_frames, int n_bits, cudaStream_t s) {
  const int64_t total = n_frames * ((n_bits + 31) / 32);
  pack_codewords_kernel<<<(int)std::min<int64_t>((total + 7) / 8, 8192), 256, 0, s>>>(bytes, words, n_frames, n_bits);
  return cudaGetLastError();
}

cudaError_t launch_adam(float* w, const float* g, float* m, float* v, int64_t n, float lr, int step,
                        cudaStream_t s) {
  const float b1 = 0.9f, b2 = 0.999f;
  float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
  int blocks = (int)std::min<int64_t>((n + 255) / 256, 4096);
  adam_kernel<<<blocks, 256, 0, s>>>(w, g, m, v, n, lr, b1, b2, 1e-8f, c1, c2);
  return cudaGetLastError();
}

}  // namespace cbk
