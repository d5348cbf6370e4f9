// The NR encoder on packed columns, by the threads of one CTA: the frame generator's
// (gen.cu) and the block encoder's (encode.cu).
//
// LdpcCode::encode_block with Encoder::Core (crates/com-fec/src/ldpc.rs:774-786): the
// syndromes of the four core base rows, the core parity from the block-circulant inverse
// of the core (computed on the host), then every extension parity bit from its own row.
// Every column's Z bits are packed 32 to a word; the rows r0 .. r0 + 31 of an entry (j, s)
// read the Z-bit column j from bit (r0 + s) mod Z on (window32, wrapping at Z), and the XOR
// over a row's entries is then the parity of 32 rows at once.
#pragma once
#include "dev_math.cuh"
#include "device_common.cuh"

namespace cbk {
namespace {

// cwp: [n_full / Z][ceil(Z / 32) + 1] words, the systematic columns filled (each with a zero
// word at its end); synp: 4 such columns of scratch.  Fills the parity columns; ends with a
// barrier.
__device__ __forceinline__ void encode_packed_columns(const cbd::DevCode& c, uint32_t* cwp, uint32_t* synp, int tid,
                                                      int nt) {
  const int z = c.z, wz = (z + 31) >> 5, ws = wz + 1;
  // the 32-row window of a packed Z-bit column from row r0 with shift s (rows past Z read 0)
  auto window = [&](const uint32_t* col, int r0, int shift) -> uint32_t {
    int o = r0 + shift;
    o -= (o >= z) ? z : 0;
    uint32_t win = window32(col, o);
    const int nrows = min(32, z - r0);
    if (o + nrows > z) win |= window32(col, 0) << (z - o);
    return nrows == 32 ? win : (win & ((1u << nrows) - 1u));
  };
  // core syndromes over the systematic columns
  for (int task = tid; task < 4 * wz; task += nt) {
    const int L = task / wz, g = task - L * wz;
    uint32_t acc = 0;
    for (int t = c.layer_start[L]; t < c.layer_start[L + 1]; t++) {
      const uint32_t en = c.entry[t];
      const int j = (int)(en >> 16);
      if (j < c.cols_k) acc ^= window(cwp + j * ws, g * 32, (int)(en & 0xffffu));
    }
    synp[L * ws + g] = acc;
    if (g == wz - 1) synp[L * ws + wz] = 0u;
  }
  __syncthreads();
  // core parity: block-circulant inverse of the core
  for (int task = tid; task < 4 * wz; task += nt) {
    const int blk = task / wz, g = task - blk * wz;
    uint32_t acc = 0;
    for (int t = 0; t < c.n_core_terms; t++) {
      const uint32_t ct = c.core_term[t];
      if ((int)(ct >> 20) != blk) continue;
      acc ^= window(synp + (int)((ct >> 16) & 15u) * ws, g * 32, (int)(ct & 0xffffu));
    }
    uint32_t* col = cwp + (c.cols_k + blk) * ws;
    col[g] = acc;
    if (g == wz - 1) col[wz] = 0u;
  }
  __syncthreads();
  // extension parity: row L >= 4 closes on its own column cols_k + L (shift 0) and reads
  // only systematic and core parity columns
  for (int task = 4 * wz + tid; task < c.rows_n * wz; task += nt) {
    const int L = task / wz, g = task - L * wz;
    uint32_t acc = 0;
    for (int t = c.layer_start[L]; t < c.layer_start[L + 1]; t++) {
      const uint32_t en = c.entry[t];
      const int j = (int)(en >> 16);
      if (j != c.cols_k + L) acc ^= window(cwp + j * ws, g * 32, (int)(en & 0xffffu));
    }
    uint32_t* col = cwp + (c.cols_k + L) * ws;
    col[g] = acc;
    if (g == wz - 1) col[wz] = 0u;
  }
  __syncthreads();
}

}  // namespace
}  // namespace cbk
