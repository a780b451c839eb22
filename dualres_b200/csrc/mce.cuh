// Minimum-contrast summary of an image on the device
// (compute_mce_summary_data_impl, estimate_kernel_parameters.h:50-101).
//
// For every lattice offset p and every pair of voxels (x, x + p) inside the
// grid whose values are both non-zero and not NaN: the sums of x*y, x and y in
// double and the pair count.  That is 25,348 offsets times the image: FP64
// arithmetic, 3 FMAs per offset and voxel, is what bounds it.
//
// A task is 8 offsets that differ in x only (dx0 .. dx0 + 7 at one (dy, dz)); a lane
// has one task, and a warp walks the x rows of its slab together, four voxels
// at a time: the four x values (one load for the warp) meet a window of eleven y
// values that slides along the row in registers, so 96 FMAs take one 16-byte
// load of each row and eight conversions.  Masked values are zero and masks
// are factors 0 or 1, so that nothing branches; the counts come from bit rows by
// popcount.  Infinite voxels would meet those zeros (0 * inf is NaN), so the rows
// hold 0 in their place and k_mce_infinite adds their pairs; without any it only
// writes its zeros (2 us).  Rows are padded with zeros (dx0 is a multiple of 4: every load is
// aligned and none is tested), rows outside the grid are a row of zeros, and x
// rows without data are skipped.  Slabs interleave the rows, which balances
// them; a second kernel adds the slabs in order, so results do not depend on
// scheduling.  Measured on a 76x76x60 image, whole call: 3.0 ms (34.3 ms with one
// voxel pair per thread at a time, masks tested and rows divided out in the loop).
#pragma once

#include "common.cuh"

namespace drb {

constexpr int MCE_THREADS = 128;
constexpr int MCE_LAGS = 8;
constexpr int MCE_REACH = 25;  // largest |component| of an offset (perturbation_matrix.h:19-109)
constexpr int MCE_FRONT = 32, MCE_BACK = 40;  // zeros before and after a row: dx0 >= -20, dx0 + 7 <= 27

struct MceSums {
  double sxy, sx, sy;
  int n;
};
// 8 offsets (dx0 + l, dy, dz): out[l] is the offset's index, or -1 where it is none of the summary's.
struct MceTask {
  int dy, dz, dx0;
  int out[MCE_LAGS];
};
// Geometry of the padded rows: pitch floats a row and bw words of mask bits (bit 32 + i is voxel i); row ny * nz is zero.
struct MceRows {
  int nx, ny, nz, pitch, bw;
};

// any[r]: 0 without data, 2 with an infinite voxel (which also sets *infinite), else 1.
__global__ void k_mce_rows(const float* __restrict__ img, MceRows g, float* __restrict__ rows, uint32_t* __restrict__ bits,
                           int* __restrict__ any, int* __restrict__ infinite) {
  const int r = blockIdx.x, lane = threadIdx.x;  // one warp per row
  const bool real = r < g.ny * g.nz;
  float* row = rows + (long long)r * g.pitch;
  for (int i = lane; i < g.pitch; i += 32) {
    const int x = i - MCE_FRONT;
    float v = real && x >= 0 && x < g.nx ? img[(long long)r * g.nx + x] : 0.f;
    if (!isfinite(v)) v = 0.f;
    row[i] = v;
  }
  uint32_t some = 0, inf = 0;
  for (int q = 0; q < g.bw; q++) {
    const int x = 32 * (q - 1) + lane;
    const float v = real && x >= 0 && x < g.nx ? img[(long long)r * g.nx + x] : 0.f;
    const uint32_t b = __ballot_sync(0xffffffffu, !isnan(v) && v != 0.f);
    if (lane == 0) bits[(long long)r * g.bw + q] = b;
    some |= b;
    inf |= __ballot_sync(0xffffffffu, isinf(v));
  }
  if (lane == 0) {
    any[r] = inf != 0 ? 2 : some != 0;
    if (inf != 0) *infinite = 1;
  }
}

__global__ void __launch_bounds__(MCE_THREADS) k_mce_pairs(const float* __restrict__ rows, const uint32_t* __restrict__ bits,
                                                          const int* __restrict__ any, MceRows g,
                                                          const MceTask* __restrict__ tasks, int n_tasks, int n_off,
                                                          MceSums* __restrict__ part) {
  const int t = blockIdx.y * MCE_THREADS + threadIdx.x;
  const int nrows = g.ny * g.nz, n4 = (g.nx + 3) / 4, nw = (g.nx + 31) / 32;
  const MceTask* T = tasks + min(t, n_tasks - 1);
  const int dy = T->dy, dz = T->dz, dx0 = T->dx0;
  double sxy[MCE_LAGS], sx[MCE_LAGS], sy[MCE_LAGS];
  int n[MCE_LAGS];
#pragma unroll
  for (int l = 0; l < MCE_LAGS; l++) {
    sxy[l] = sx[l] = sy[l] = 0.0;
    n[l] = 0;
  }
  for (int r = blockIdx.x; r < nrows; r += gridDim.x) {
    if (!__ldg(any + r)) continue;  // the same row for the whole block
    const int j2 = r % g.ny + dy, k2 = r / g.ny + dz;
    const int r2 = j2 >= 0 && j2 < g.ny && k2 >= 0 && k2 < g.nz ? k2 * g.ny + j2 : nrows;
    const float4* X = reinterpret_cast<const float4*>(rows + (long long)r * g.pitch + MCE_FRONT);
    const float4* Y = reinterpret_cast<const float4*>(rows + (long long)r2 * g.pitch + MCE_FRONT + dx0);
    double w[12], m[12];  // y values and their masks at x .. x + 11 (+ dx0)
    auto put = [&](int at, float4 v) {
      const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int i = 0; i < 4; i++) {
        w[at + i] = (double)f[i];
        m[at + i] = f[i] != 0.f ? 1.0 : 0.0;
      }
    };
    put(0, __ldg(Y));
    put(4, __ldg(Y + 1));
    for (int i = 0; i < n4; i++) {
      const float4 xv = __ldg(X + i);
      put(8, __ldg(Y + i + 2));
      const float f[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const double x = (double)f[u], mx = f[u] != 0.f ? 1.0 : 0.0;
#pragma unroll
        for (int l = 0; l < MCE_LAGS; l++) {
          sxy[l] = fma(x, w[u + l], sxy[l]);
          sx[l] = fma(x, m[u + l], sx[l]);
          sy[l] = fma(mx, w[u + l], sy[l]);
        }
      }
#pragma unroll
      for (int l = 0; l < 8; l++) {
        w[l] = w[l + 4];
        m[l] = m[l + 4];
      }
    }
    const uint32_t* bx = bits + (long long)r * g.bw + 1;
    const uint32_t* by = bits + (long long)r2 * g.bw;
    for (int q = 0; q < nw; q++) {
      const uint32_t x = __ldg(bx + q);
#pragma unroll
      for (int l = 0; l < MCE_LAGS; l++) {
        const int p = 32 + 32 * q + dx0 + l;  // >= 12
        n[l] += __popc(x & __funnelshift_r(__ldg(by + (p >> 5)), __ldg(by + (p >> 5) + 1), p & 31));
      }
    }
  }
  if (t >= n_tasks) return;
#pragma unroll
  for (int l = 0; l < MCE_LAGS; l++) {
    const int o = T->out[l];
    if (o >= 0) part[(long long)blockIdx.x * n_off + o] = MceSums{sxy[l], sx[l], sy[l], n[l]};
  }
}

// The pairs of infinite voxels, as one more slab: a thread takes one offset p and, for each infinite voxel v in the image's order,
// the pairs (v, v + p) and, unless its other voxel is infinite too (and counts it), (v - p, v).  The counts are k_mce_pairs'.
__global__ void k_mce_infinite(const float* __restrict__ img, const int* __restrict__ any, const int* __restrict__ infinite,
                               MceRows g, const MceTask* __restrict__ tasks, int n_tasks, MceSums* __restrict__ part) {
  const int t = (blockIdx.x * blockDim.x + threadIdx.x) / MCE_LAGS, l = threadIdx.x % MCE_LAGS;
  if (t >= n_tasks || tasks[t].out[l] < 0) return;
  MceSums s{0.0, 0.0, 0.0, 0};
  if (*infinite) {
    const int p[3] = {tasks[t].dx0 + l, tasks[t].dy, tasks[t].dz};
    // the value at (x, y, z), 0 where it is masked or outside the grid
    auto value = [&](int x, int y, int z) {
      if (x < 0 || x >= g.nx || y < 0 || y >= g.ny || z < 0 || z >= g.nz) return 0.f;
      const float v = img[((long long)z * g.ny + y) * g.nx + x];
      return isnan(v) ? 0.f : v;
    };
    auto add = [&](float x, float y) {
      s.sxy += (double)x * (double)y;
      s.sx += (double)x;
      s.sy += (double)y;
    };
    for (int r = 0; r < g.ny * g.nz; r++) {
      if (any[r] != 2) continue;
      const int y = r % g.ny, z = r / g.ny;
      for (int x = 0; x < g.nx; x++) {
        const float v = img[(long long)r * g.nx + x];
        if (!isinf(v)) continue;
        const float b = value(x + p[0], y + p[1], z + p[2]), a = value(x - p[0], y - p[1], z - p[2]);
        if (b != 0.f) add(v, b);
        if (a != 0.f && !isinf(a)) add(a, v);
      }
    }
  }
  part[tasks[t].out[l]] = s;
}

// Slab sums in order; covariance (sum_xy - sum_x sum_y / n) / (n - 1) for n > 1, else 0.
__global__ void k_mce_finish(const MceSums* __restrict__ part, int n_slabs, int n_off, float* covariance,
                             int* npairs, double* sums) {
  const int o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= n_off) return;
  double sxy = 0.0, sx = 0.0, sy = 0.0;
  int n = 0;
  for (int s = 0; s < n_slabs; s++) {
    const MceSums& p = part[(long long)s * n_off + o];
    sxy += p.sxy;
    sx += p.sx;
    sy += p.sy;
    n += p.n;
  }
  npairs[o] = n;
  covariance[o] = n > 1 ? (float)((sxy - sx * sy / n) / (double)(n - 1)) : 0.0f;
  if (sums) {
    sums[3 * o] = sxy;
    sums[3 * o + 1] = sx;
    sums[3 * o + 2] = sy;
  }
}

}  // namespace drb
