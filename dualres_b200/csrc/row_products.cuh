// Kriging products on the CUDA cores: W mu_D and W^T rs for chain sets that do
// not use the tensor-core tiles.
//
// The matrix is cut into groups of R = 4 consecutive rows.  A group stores the
// union of its rows' columns once, each with 4 values (0 where a row does not
// have the column): a chain vector is fetched once for 4 rows, and an entry
// takes 18 bytes (columns are 16-bit offsets from a 32-bit base per batch of 32
// entries; a batch whose columns would span more is filled up with entries of
// value 0).  Neighbouring rows share most of their columns: on a 32^3 volume at
// 6.9 mm W^T stores 1.34 values per nonzero (6.1 bytes, 8 in CSR) and W, whose
// rows lie two voxels apart, 1.7 (7.8 bytes); a third and two fifths of the gathers.
//
// A warp takes S = 32 / CL entries at a time: CL lanes share an entry, each with
// V adjacent chains (one vector load) in NR rounds, 4 chains per lane from 5 chains;
// with 1, 2 or 4 chains every lane has its own entry.  U steps' loads are issued before any is used, and L2
// is asked for the next group's entries meanwhile.  SW warps share a group of
// W, whose groups are few and long; a group of W^T has a warp of its own.  The
// sums are reduced over the lanes by halving exchanges (the rows are divided
// among the lanes as it goes), then the epilogue writes rs = Ys - W mu_D
// (MultiResParameters.h:361-363, 505-507) or
// gD = sigma_h^-2 (Yh - mu_D) + sigma_s^-2 W^T rs (:357-364) and adds the squared
// residuals to the block's partials.
//
// What bounds it is latency: a group is a chain of its pointer, its entries (from
// memory on large volumes) and the chain vectors (L1 / L2).  Measured (W / W^T,
// us; before: CSR rows): 1 chain, 32^3 volume 5.8 / 5.7 (7.8 / 7.9); 2 chains,
// 80x80x64, 510 MB of entries 56 / 47, 4.9 TB/s (134 / 160); 12 chains, 43x23x17
// 9.0 / 10.1 (23 / 20); 16 chains, 64x64x48 29.5 / 29 launched back to back and 35 /
// 33 inside an iteration (tensor-core tiles 58 / 45, whose dense blob is 8 times the
// entries there).  Tried: groups of single rows
// (W 78 us on 80x80x64), entries streamed through a shared-memory ring by
// cp.async (88 / 71 us: the ring takes the L1 that the chain vectors hit).
#pragma once

#include "common.cuh"
#include "drb.h"
#include "tma.cuh"

namespace drb {

constexpr int ROWP_NT = 256;

// V floats at p (aligned to V * 4 bytes).
template <int V>
__device__ __forceinline__ void load_chains(const float* p, float* x) {
  if constexpr (V == 4) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    x[0] = t.x; x[1] = t.y; x[2] = t.z; x[3] = t.w;
  } else if constexpr (V == 2) {
    const float2 t = *reinterpret_cast<const float2*>(p);
    x[0] = t.x; x[1] = t.y;
  } else {
    x[0] = *p;
  }
}
// U and the blocks per SM that the registers are budgeted for, by chains per lane.  W: 4 steps at 5 blocks (80x80x64, 2
// chains: 60 us; 8 steps at 3 blocks 67); W^T: 8 steps at 3 blocks (47.8; 4 at 5 blocks 47.4, but 6.9 against 6.0 us on
// 32^3).  With 4 chains per lane 3 blocks (16 chains, 64x64x48: W 30.7 us with 4 steps, 2 unbudgeted blocks 38; W^T 30.5
// with 2 steps, 31.6 with 4).
template <int CV, bool WT> struct RowpCfg {
  static constexpr int U = CV <= 2 ? (WT ? 8 : 4) : (CV <= 4 ? (WT ? 2 : 4) : 2);
  static constexpr int MINB = CV <= 2 ? (WT ? 3 : 5) : (CV <= 4 ? 3 : 1);
};

template <int V, int CL, int NR, int SW, bool WT>
__global__ void __launch_bounds__(ROWP_NT, RowpCfg<V * NR, WT>::MINB)
    k_row_product(DevVolume v, DevRowGroups M, DevChains ch, int step, int sel, int chain_only) {
  constexpr int R = ROWP_R, S = 32 / CL, CV = V * NR, CW = CL * CV;  // entries per step; chains per lane, chains covered
  constexpr int U = RowpCfg<CV, WT>::U;
  constexpr int RO = R > S ? R / S : 1;                   // rows that a lane ends up with
  constexpr int GB = 8 / SW;                              // groups per block at a time
  __shared__ float part[SW > 1 ? 8 * R * CW : 1];
  // rows that add to a chain's squared residual: a warp's, or a thread's share of the shared groups
  constexpr int NRED = SW > 1 ? (ROWP_NT / CW < R * GB ? ROWP_NT / CW : R * GB) : 8;
  __shared__ double red[NRED * CW];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int slot = lane / CL, cl = lane % CL, sub = warp % SW;
  // the warp's first group: where its entries lie, and L2 is asked for them (the matrix is constant: this may run ahead
  // of the kernel that makes the chain vectors)
  const int stride = gridDim.x * GB;
  int g = blockIdx.x * GB + warp / SW;
  int p0 = 0, p1 = 0;
  auto fetch = [&](int gg, int& a, int& b) {
    a = gg < M.groups ? __ldg(M.ptr + gg) : 0;
    b = gg < M.groups ? __ldg(M.ptr + gg + 1) : 0;
  };
  auto prefetch = [&](int a, int b) {
    // whole 16-byte units around the entries; the arrays are padded to 64 entries
    if (M.stream && lane == 0 && sub == 0 && b > a) {
      const int a8 = a & ~7, n8 = ((b + 7) & ~7) - a8;
      bulk_prefetch_l2(M.val + (long long)a8 * R, n8 * R * 4);
      bulk_prefetch_l2(M.off + a8, n8 * 2);
    }
  };
  fetch(g, p0, p1);
  prefetch(p0, p1);
  grid_dep_wait();

  const int C = ch.C;
  const long long Cp = ch.Cp;
  const float* __restrict__ mu = ch.muD + (long long)sel * v.n_h * Cp;
  const float* __restrict__ X = WT ? ch.rs : mu;
  auto chain = [&](int n) { return (cl + CL * (n / V)) * V + n % V; };  // chain of this lane's value n
  auto active = [&](int c) { return c < C && (chain_only < 0 || c == chain_only) && (step < 0 || step <= ch.st[c].L_cur); };
  // the row (of its group's R) a lane ends up with first, and whether it is the one that writes it
  int first = 0;
  bool writer = true;
  {
    int rows = R;
#pragma unroll
    for (int o = 16; o >= CL; o >>= 1) {
      if (rows > 1) {
        rows >>= 1;
        if (lane & o) first += rows;
      } else if (lane & o) {
        writer = false;
      }
    }
  }
  // SW > 1: thread t finishes rows t / CW, + NT / CW, ... of chain t % CW
  const int tc = threadIdx.x % CW;
  bool act[CV];
  float sh[CV], ss[CV];
  double sq[CV];
#pragma unroll
  for (int n = 0; n < CV; n++) {
    const int c = SW > 1 ? tc : chain(n);
    act[n] = active(c);
    sq[n] = 0.0;
    sh[n] = ss[n] = 0.f;
    if (WT && act[n]) {
      sh[n] = ch.st[c].sh;
      ss[n] = ch.st[c].ss;
    }
  }
  // the rounds are the same for all warps of a block: they meet at barriers when they share groups
  const int rounds = (M.groups + stride - 1) / stride;
  for (int it = 0; it < rounds; it++, g += stride) {
    if (SW == 1 && g >= M.groups) break;
    // the next group's entries are on their way from memory while this one's are used
    int n0, n1;
    fetch(g + stride, n0, n1);
    // the epilogue's operands
    float y[RO], m[RO][CV];
    if constexpr (SW == 1) {
#pragma unroll
      for (int r = 0; r < RO; r++) {
        const int row = g * R + first + r;
        const bool on = writer && row < M.n_rows;
        y[r] = on ? __ldg((WT ? v.Yh : v.Ys) + row) : 0.f;
#pragma unroll
        for (int n = 0; n < CV; n++) m[r][n] = WT && on && act[n] ? mu[row * Cp + chain(n)] : 0.f;
      }
    }
    float acc[R][CV];
#pragma unroll
    for (int r = 0; r < R; r++)
#pragma unroll
      for (int n = 0; n < CV; n++) acc[r][n] = 0.f;
    bool asked = false;
    for (int kb = p0 + sub * S; kb < p1; kb += U * SW * S) {
      float a[U][R], x[U][CV];
      int col[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int k = kb + u * SW * S + slot;
        col[u] = 0;
#pragma unroll
        for (int r = 0; r < R; r++) a[u][r] = 0.f;
        if (k < p1) {
          const int cu = __ldg(M.base + (k >> 5)) + (int)__ldg(M.off + k);
          const float4 t = __ldg(reinterpret_cast<const float4*>(M.val) + k);
          if (in_bounds(cu, M.n_cols, ch.err)) {
            col[u] = cu;
            a[u][0] = t.x; a[u][1] = t.y; a[u][2] = t.z; a[u][3] = t.w;
          }
        }
      }
      if (!asked) {
        prefetch(n0, n1);
        asked = true;
      }
#pragma unroll
      for (int u = 0; u < U; u++)
#pragma unroll
        for (int n = 0; n < NR; n++) {
          if (CW == V || chain(n * V) < C) {
            load_chains<V>(X + col[u] * Cp + chain(n * V), x[u] + n * V);
          } else {
#pragma unroll
            for (int i = 0; i < V; i++) x[u][n * V + i] = 0.f;
          }
        }
      // a column that a row does not have takes no part in its sum (0 * inf would)
#pragma unroll
      for (int u = 0; u < U; u++)
#pragma unroll
        for (int r = 0; r < R; r++)
          if (a[u][r] != 0.f) {
#pragma unroll
            for (int n = 0; n < CV; n++) acc[r][n] = fmaf(a[u][r], x[u][n], acc[r][n]);
          }
    }
    {
      int rows = R;
#pragma unroll
      for (int o = 16; o >= CL; o >>= 1) {
        const bool up = (lane & o) != 0;
        if (rows > 1) {
          rows >>= 1;
#pragma unroll
          for (int r = 0; r < R / 2; r++) {
            if (r >= rows) break;
#pragma unroll
            for (int n = 0; n < CV; n++) {
              const float mine = up ? acc[rows + r][n] : acc[r][n], other = up ? acc[r][n] : acc[rows + r][n];
              acc[r][n] = mine + __shfl_xor_sync(0xffffffffu, other, o);
            }
          }
        } else {
#pragma unroll
          for (int n = 0; n < CV; n++) acc[0][n] += __shfl_xor_sync(0xffffffffu, acc[0][n], o);
        }
      }
    }
    auto finish = [&](int row, int c, float sum, float yy, float mm, float s_h, float s_s) -> double {
      const float res = WT ? yy - mm : yy - sum;
      if (WT) ch.gD[row * Cp + c] = s_h * res + s_s * sum;
      else ch.rs[row * Cp + c] = res;
      return (double)res * res;
    };
    if constexpr (SW == 1) {
      if (writer) {
#pragma unroll
        for (int r = 0; r < RO; r++) {
          const int row = g * R + first + r;
          if (row >= M.n_rows) break;
#pragma unroll
          for (int n = 0; n < CV; n++)
            if (act[n]) sq[n] += finish(row, chain(n), acc[r][n], y[r], m[r][n], sh[n], ss[n]);
        }
      }
    } else {
      const int row0 = (g - warp / SW) * R, r0 = threadIdx.x / CW;  // the block's first row, this thread's first of them
      const float y0 = r0 < R * GB && row0 + r0 < M.n_rows ? __ldg((WT ? v.Yh : v.Ys) + row0 + r0) : 0.f;
      if (writer) {
#pragma unroll
        for (int r = 0; r < RO; r++)
#pragma unroll
          for (int n = 0; n < CV; n++) part[(warp * R + first + r) * CW + chain(n)] = acc[r][n];
      }
      __syncthreads();
      for (int r = r0; r < R * GB; r += ROWP_NT / CW) {
        const int row = row0 + r;
        if (row >= M.n_rows || !act[0]) break;
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < SW; w++) s += part[((r / R * SW + w) * R + r % R) * CW + tc];
        sq[0] += finish(row, tc, s, r == r0 ? y0 : __ldg((WT ? v.Yh : v.Ys) + row), WT ? mu[row * Cp + tc] : 0.f, sh[0], ss[0]);
      }
      if (it + 1 < rounds) __syncthreads();
    }
    p0 = n0;
    p1 = n1;
  }
  if constexpr (SW == 1) {
#pragma unroll
    for (int n = 0; n < CV; n++) {
      double t = sq[n];
#pragma unroll
      for (int o = 16; o >= CL; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (slot == 0) red[warp * CW + chain(n)] = t;
    }
  } else {
    if ((int)threadIdx.x < NRED * CW) red[threadIdx.x] = sq[0];
  }
  __syncthreads();
  for (int c = threadIdx.x; c < CW; c += ROWP_NT) {
    if (!active(c)) continue;
    double t = 0.0;
    for (int w = 0; w < NRED; w++) t += red[w * CW + c];
    const int slot_l = WT ? SL_RHL : SL_RSL, slot_0 = WT ? SL_RH0 : SL_RS0;
    const int sl = step <= 0 ? slot_0 : (step == ch.st[c].L_cur ? slot_l : SL_SCRATCH);
    ch.part[((long long)c * NSLOT + sl) * ch.maxblk + blockIdx.x] = t;
  }
}

// Single-resolution volumes have no W: gD = sigma_h^-2 (Yh - mu_D), element by element (chains fastest), with the
// ||Yh - mu_D||^2 partials per block.  Thread t of a block of NT handles chain t % CW; CW >= C is a power of two.
__global__ void __launch_bounds__(ROWP_NT) k_data_gradient(DevVolume v, DevChains ch, int CW, int step, int sel,
                                                           int chain_only) {
  grid_dep_wait();
  __shared__ double red[ROWP_NT];
  const int c = threadIdx.x % CW, rpb = ROWP_NT / CW;
  const long long Cp = ch.Cp;
  const bool act = c < ch.C && (chain_only < 0 || c == chain_only) && (step < 0 || step <= ch.st[c].L_cur);
  double sq = 0.0;
  if (act) {
    const float sh = ch.st[c].sh;
    const float* mu = ch.muD + (long long)sel * v.n_h * Cp + c;
    for (int row = blockIdx.x * rpb + threadIdx.x / CW; row < v.n_h; row += gridDim.x * rpb) {
      const float res = v.Yh[row] - mu[row * Cp];
      ch.gD[row * Cp + c] = sh * res;
      sq += (double)res * res;
    }
  }
  red[threadIdx.x] = sq;
  __syncthreads();
  if ((int)threadIdx.x < CW && act) {
    double t = 0.0;
    for (int w = 0; w < rpb; w++) t += red[w * CW + c];
    const int sl = step <= 0 ? SL_RH0 : (step == ch.st[c].L_cur ? SL_RHL : SL_SCRATCH);
    ch.part[((long long)c * NSLOT + sl) * ch.maxblk + blockIdx.x] = t;
  }
}

}  // namespace drb
