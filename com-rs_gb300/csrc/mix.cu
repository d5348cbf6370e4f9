// Mixed batches: codewords of different base graphs, lifting sizes, rates and
// modulations decoded by one persistent kernel, each with its own early exit.
//
// The batch's codewords are sorted by lifting size into classes.  The kernel walks the
// classes in order; for class k every CTA, one per SM, splits its threads into `slots` groups of
// `slot_threads` threads (a multiple of 32, synchronised by their own named barrier).  One
// CTA of 768 threads instead of two of 384: Z = 208 then has three slots of seven warps on an
// SM and not two, Z = 128 five of four warps and not four (the decode phase of 16384
// uneven codewords 9.0 -> 8.6 ms).
// Each slot pulls one codeword after another from the class's atomic queue (work
// stealing), decodes it with the layered min-sum of decode.cu (the same row updates,
// the same syndrome test, so every result equals the single-code path bit for bit) and
// takes the next codeword as soon as its own syndrome test passes.  A thread of a slot
// owns `rows_per_thread` lifted rows of each layer: the autotuner picks that number per
// class (more rows per thread = more slots in flight for small Z).
#include <cuda_runtime.h>

#include "decode_common.cuh"
#include "kernels.h"
#include "layered_nr.cuh"

namespace cbk {
namespace {

// a slot of one warp needs no barrier of the CTA's sixteen
__device__ __forceinline__ void slot_sync(int bar, int n) {
  if (n == 32) __syncwarp();
  else asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(n) : "memory");
}

// OR of `bad` over the slot's threads (flag starts at 0 and is left at 0)
__device__ __forceinline__ bool slot_any(int bad, int* flag, int bar, int n, int lt) {
  if (bad) atomicOr(flag, 1);
  slot_sync(bar, n);
  const int f = *(volatile int*)flag;
  slot_sync(bar, n);
  if (lt == 0) *flag = 0;
  return f != 0;
}

// Whether some check fails, for one slot: stage 1 on the rows of the first two
// layers, stage 2 on packed hard decisions (the test of decode.cu's some_check_fails).
// `own` forms the own columns of skipped rows before stage 2 reads them.
template <class Own>
__device__ bool slot_check_fails(const float* post, uint32_t* hd, const uint32_t* ent, const uint16_t* lstart,
                                 int rows_n, int ncol, int z, int lt, int nt, int bar, int* flag, const Own& own) {
  int bad = 0;
  for (int r = lt; r < z && !bad; r += nt)
    for (int L = 0; L < 2 && !bad; L++) {
      uint32_t par = 0;
      for (int t = lstart[L]; t < lstart[L + 1]; t++) {
        const uint32_t en = ent[t];
        int cc = r + (int)(en & 0xffffu);
        cc -= (cc >= z) ? z : 0;
        par ^= (uint32_t)(post[(int)(en >> 16) * z + cc] < 0.f);
      }
      bad = (int)par;
    }
  if (slot_any(bad, flag, bar, nt, lt)) return true;
  own();
  build_hard_decisions(post, hd, ncol, z, lt, nt);
  slot_sync(bar, nt);
  const int wz = (z + 31) >> 5, ws = wz + 1;
  for (int task = lt; task < rows_n * wz && !bad; task += nt) {
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
  return slot_any(bad, flag, bar, nt, lt);
}

// The rows of one iteration with the base graph's structure at compile time
// (layered_nr.cuh), the edge addresses from the slot's table.  Bound by issue: the degree and
// the entries' bounds are no longer read and branched on per row.  Used for slots of at
// least 128 threads; 16384 uneven codewords, generator and decoder: 9.32 ms, 9.99 with no
// slot on it, 9.41 from 256 threads, 9.52 from 64 and 9.70 with all slots on it.  The
// normalised rule only, the one a batch has.  (The table-driven rows keep the offset rule's
// branch, which nothing reaches: without it the compiler's registers fall out 1 % worse at 16384
// codewords and 20 % at 300.)
struct MixTable {
  const uint2* eaddr;  // {4 shift, 4 column Z} per entry
};
template <int BG, int Q>
__device__ __forceinline__ void mix_rows(unsigned char* post, const MixTable& tab, const StateSlot<float>& st, int lt,
                                         int z, bool first, float alpha, int live, int bar, int nt) {
  using G = cbn::Graph<BG>;
  if constexpr (Q < G::rows) {
    if constexpr (Q >= 4) {
      if constexpr (G::level_end[Q - 1] != 0) {
        if (live <= cbn::rest_min<BG>(Q)) return;
      }
    }
    constexpr int L = G::order[Q], S0 = G::start[L], D = G::start[L + 1] - S0;
    if (lt < z) {
      int r = lt;
      asm volatile("" : "+r"(r));  // (addresses formed where they are used, see nr_iteration)
      float a1 = 0.f, a2 = 0.f, n1, n2;
      uint32_t mt = 0u, nm;
      if (!first) st.load(L * z + r, a1, a2, mt);
      cbn::nr_row<BG, cbn::RuntimeLifting, S0, D, 1>(post, tab, r, 4 * r, 4 * z, a1, a2, mt, alpha, n1, n2, nm);
      st.store(L * z + r, n1, n2, nm);
    }
    if constexpr (G::level_end[Q] != 0) slot_sync(bar, nt);
    mix_rows<BG, Q + 1>(post, tab, st, lt, z, first, alpha, live, bar, nt);
  }
}

// Decode one codeword of the batch in a slot; RHO rows per thread (0: one, by mix_rows).
// flag[0] is slot_any's; flag[1] is set when the codeword runs every row (beyond_skipping).
// Returns whether the codeword has to be decoded again so.
template <int RHO>
__device__ bool decode_item(const MixDecodeArgs& a, const MixItem& it, unsigned char* sm, int ncol_max,
                            const StateSlot<float>& st, int lt, int nt, int bar, int* flag, unsigned int* err) {
  const cbd::DevCode& c = a.codes[it.code];
  const int z = c.z;
  const int ws = (z + 31) / 32 + 1;
  float* post = reinterpret_cast<float*>(sm);
  uint32_t* hd = reinterpret_cast<uint32_t*>(post + 68 * z);
  uint32_t* s_ent = hd + ncol_max * ws;
  uint2* s_addr = reinterpret_cast<uint2*>(s_ent + cbh::kMaxEntries);
  uint16_t* s_lstart = reinterpret_cast<uint16_t*>(s_addr + cbh::kMaxEntries);
  uint8_t* s_order = reinterpret_cast<uint8_t*>(s_lstart + cbh::kMaxLayers + 1);
  uint8_t* s_end = s_order + cbh::kMaxLayers;
  const int ncol = c.n_full / z;
  for (int i = lt; i < c.n_entries; i += nt) {
    const uint32_t en = c.entry[i];
    s_ent[i] = en;
    s_addr[i] = RHO ? c.eaddr[i] : make_uint2(4u * (en & 0xffffu), 4u * (en >> 16) * (uint32_t)z);
  }
  for (int i = lt; i <= c.rows_n; i += nt) s_lstart[i] = c.layer_start[i];
  for (int i = lt; i < c.rows_n; i += nt) {
    s_order[i] = c.layer_order[i];
    s_end[i] = c.level_end[i];
  }
  const float* llr = a.llr + it.llr_offset;
  const int rule = a.rule;
  const float alpha = a.alpha;
  const int rows_n = c.rows_n;
  volatile int* every = flag + 1;
  for (int v = lt; v < c.n_full; v += nt) post[v] = 0.f;
  slot_sync(bar, nt);
  // the batch's codes all use the plain rate matching 2Z + t
  Widest<float> widest;
  for (int t = lt; t < c.e; t += nt) {
    const float v = __fadd_rn(0.f, __ldcs(llr + t));
    widest.add(v);
    post[2 * z + t] = v;
  }
  if (widest.beyond()) *every = 1;
  slot_sync(bar, nt);
  const int rows_run = *every ? rows_n : c.rows_run, rows_live = *every ? rows_n : c.rows_live;
  for (int v = c.k_info + lt; v < c.k; v += nt) post[v] = cbd::kKnownBitLlr;
  slot_sync(bar, nt);
  int iters = 0;
  if (slot_check_fails(post, hd, s_ent, s_lstart, rows_n, ncol, z, lt, nt, bar, flag, [] {})) {
    iters = a.max_it;
    for (int iter = 1; iter <= a.max_it; iter++) {
      // the base rows by levels, as decode.cu runs them; each row's state is loaded where
      // it is used (loaded one row ahead: 17.56 against 17.40 ms per decode phase)
      if constexpr (RHO == 0) {
        unsigned char* pb = reinterpret_cast<unsigned char*>(post);
        if (c.bg == 1) mix_rows<1, 0>(pb, MixTable{s_addr}, st, lt, z, iter == 1, a.alpha, rows_live, bar, nt);
        else mix_rows<2, 0>(pb, MixTable{s_addr}, st, lt, z, iter == 1, a.alpha, rows_live, bar, nt);
      }
      for (int k = 0; RHO && k < rows_run; k++) {
        const int L = s_order[k];
        const int s0 = s_lstart[L], d = s_lstart[L + 1] - s0;
#pragma unroll
        for (int q = 0; q < RHO; q++) {
          const int r = lt + q * nt;
          if (r < z) {
            float a1 = 0.f, a2 = 0.f, n1, n2;
            uint32_t mt = 0u, nm;
            if (iter > 1) st.load(L * z + r, a1, a2, mt);
            if (a.rule == cbd::RULE_NMS)
              row_dispatch_lean<cbd::RULE_NMS>(d, post, EdgeAddrTable{s_addr + s0, r, 4 * r, 4 * z}, a1, a2, mt,
                                               a.alpha, n1, n2, nm);
            else
              row_dispatch_lean<cbd::RULE_OMS>(d, post, EdgeAddrTable{s_addr + s0, r, 4 * r, 4 * z}, a1, a2, mt,
                                               a.alpha, n1, n2, nm);
            st.store(L * z + r, n1, n2, nm);
          }
        }
        if (s_end[k]) slot_sync(bar, nt);
      }
      auto own = [&]() {
        if (rows_live == rows_n) return;
        unsent_rows(post, s_ent, s_lstart, rows_live, rows_n, z, lt, nt, [rule, alpha](int, int, float m) {
          return rule == cbd::RULE_NMS ? __fmul_rn(alpha, m) : fmaxf(__fsub_rn(m, alpha), 0.f);
        });
        slot_sync(bar, nt);
      };
      if (!slot_check_fails(post, hd, s_ent, s_lstart, rows_n, ncol, z, lt, nt, bar, flag, own)) {
        iters = iter;
        break;
      }
    }
    if (rows_live < rows_n) {
      int beyond = 0;
      for (int r = lt; r < z; r += nt) beyond |= (int)beyond_skipping(post, r, z, c.bg);
      if (slot_any(beyond, flag, bar, nt, lt)) {
        if (lt == 0) *every = 1;
        return true;
      }
    }
  }
  // counts against the sent info bits: the sent words, one per thread, loaded before the
  // ballots so that their latency overlaps them, against the decisions staged in hd (free
  // after the syndrome test)
  const int wpf = (c.k_info + 31) >> 5, lane = lt & 31, warp = lt >> 5, nw = nt >> 5;
  const uint32_t* ref = a.info + it.info_offset;
  const uint32_t ref_w = lt < wpf ? ref[lt] : 0u;
  for (int b0 = warp * 32; b0 < c.k_info; b0 += nw * 32) {
    int v = b0 + lane;
    uint32_t word = __ballot_sync(0xffffffffu, v < c.k_info && post[v] < 0.f);
    if (lane == 0) hd[b0 >> 5] = word;
  }
  slot_sync(bar, nt);
  unsigned int be = lt < wpf ? __popc(hd[lt] ^ ref_w) : 0u;
  for (int w = lt + nt; w < wpf; w += nt) be += __popc(hd[w] ^ ref[w]);
  if (be) atomicAdd(err, be);
  slot_sync(bar, nt);
  if (lt == 0) {
    cbd::FrameResult r;
    r.bit_errors = *err;
    r.frame_error = *err > 0;
    r.iterations = (uint8_t)iters;
    r.reserved = 0;
    a.results[it.index] = r;
    *err = 0;
    *every = 0;
  }
  return false;
}

__global__ void __launch_bounds__(kMixThreads, 1) mix_decode_kernel(const __grid_constant__ MixDecodeArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ long long s_item[kMixMaxSlots];
  __shared__ int s_flag[kMixMaxSlots][2];
  __shared__ unsigned int s_err[kMixMaxSlots];
  const int tid = threadIdx.x;
  if (tid < kMixMaxSlots) {
    s_flag[tid][0] = s_flag[tid][1] = 0;
    s_err[tid] = 0;
  }
  __syncthreads();
  for (int k = 0; k < a.n_classes; k++) {
    const MixClass cls = a.classes[k];
    const int slot = tid / cls.slot_threads;
    // A CTA opens at most twice its share of the class in slots: with all of them open, the
    // first CTAs take a small class whole and decode it on a few SMs (300 codewords,
    // generator and decoder: 0.97 against 0.81 ms).  One share leaves slots idle in the later
    // classes (2000 codewords 1.83 against 1.71 ms; three shares 1.76).
    const int share = (int)min((cls.count + gridDim.x - 1) / (long long)gridDim.x, (long long)kMixMaxSlots);
    if (slot < min(cls.slots, 2 * share)) {
      const int lt = tid - slot * cls.slot_threads, nt = cls.slot_threads, bar = slot + 1;
      unsigned char* sm = smem + (size_t)slot * cls.smem_per_slot;
      const StateSlot<float> st(a.state + (size_t)blockIdx.x * a.state_per_cta + (size_t)slot * cls.state_per_slot,
                                cbh::kMaxLayers * cls.z);
      for (;;) {
        if (lt == 0) s_item[slot] = (long long)atomicAdd(&a.counters[k], 1ull);
        slot_sync(bar, nt);
        const long long i = s_item[slot];
        slot_sync(bar, nt);
        if (i >= cls.count) break;
        const MixItem it = a.items[cls.first + i];
        bool again;
        do {
          if (cls.straight) again = decode_item<0>(a, it, sm, cls.max_ncol, st, lt, nt, bar, s_flag[slot], &s_err[slot]);
          else if (cls.rows_per_thread == 1) again = decode_item<1>(a, it, sm, cls.max_ncol, st, lt, nt, bar, s_flag[slot], &s_err[slot]);
          else again = decode_item<2>(a, it, sm, cls.max_ncol, st, lt, nt, bar, s_flag[slot], &s_err[slot]);
        } while (again);
      }
    }
    __syncthreads();
  }
}

}  // namespace

size_t mix_slot_smem_bytes(int z) {
  const int ws = (z + 31) / 32 + 1;
  size_t b = (size_t)68 * z * 4 + (size_t)68 * ws * 4 + (size_t)cbh::kMaxEntries * (4 + 8) +
             (size_t)(cbh::kMaxLayers + 1) * 2 + (size_t)cbh::kMaxLayers * 2;
  return (b + 15) & ~(size_t)15;
}

int mix_decode_grid(size_t smem, int device) {
  void* k = (void*)mix_decode_kernel;
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return 0;
  int per_sm = 0, sms = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kMixThreads, smem);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  return per_sm * sms;
}

cudaError_t launch_mix_decode(const MixDecodeArgs& a, int grid, size_t smem, cudaStream_t s) {
  if (a.rule != cbd::RULE_NMS) return cudaErrorInvalidValue;  // (mix_rows has no other)
  void* k = (void*)mix_decode_kernel;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  void* args[] = {(void*)&a};
  return cudaLaunchKernel(k, dim3(grid), dim3(kMixThreads), args, smem, s);
}

}  // namespace cbk
