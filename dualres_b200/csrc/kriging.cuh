// Kriging weights on the device (get_sparse_kriging_matrix_data,
// kriging_matrix.h:148-343): one weight vector per std-res voxel,
// w = K_AA^-1 k_A over the present neighbours A, normalised to sum 1.
//
// With S = K^-1 over the full neighbourhood F (computed once per volume) a row
// whose absent neighbours are B solves, by the identity
//   K_AA^-1 k_A = [S v]_A,   v_A = k_A,  v_B = -y,  S_BB y = [S v0]_B,  v0 = (k_A, 0),
// one system of size |B| instead of |A|; the host picks the cheaper route per
// row (kriging_schur_route).  Every system is symmetric positive definite and is
// factored in FP64 by a blocked Cholesky: the 32 x 32 diagonal block by one
// warp, its triangular inverse, the panel below it as a product with that
// inverse, then a 64 x 64-tiled rank-32 update of the trailing matrix.  One
// CTA solves one row at a time, taking rows from a shared counter in
// descending order of cost; its matrix lives in a private slot of global
// memory, the lower triangle packed by rows.  A row whose pivot is not
// positive is reported, and the caller solves that row by QR as the host
// builder does.
//
// What bounds it: the rows' diagonal blocks.  A row's factorisation is a chain of 32-column panels, each a chain of 32
// square roots, and one row is one CTA's (two CTAs of 512 threads per SM: one's products hide the other's chains).
// With that chain in registers (kr_factor_diag), the products on the FP64 matrix instruction (kr_tile64), four
// rows of K^-1 per warp in the dense passes and the weights rounded to float on the device, a 30x28x26 volume (1.56 M
// weights, systems up to 678) solves its rows in 9.4 ms with the download, 24.4 ms before, and forms K^-1 (1357) in
// 3.9 ms, 7.1 ms before.
#pragma once

namespace drb {

constexpr int KR_NT = 256;   // threads per CTA of the K^-1 kernels
constexpr int KR_RT = 512;   // threads per CTA of the row kernel
constexpr int KR_NB = 32;    // panel width
constexpr int KR_TILE = 64;  // trailing-update tile
constexpr int KR_LDT = KR_NB + 1;  // pitch of the diagonal blocks: a column's 32 entries lie in different pairs of banks
constexpr int KR_LDP = KR_NB + 4;  // pitch of the product operands: 4 rows x 4 columns do (kr_dmma's fragments)

enum : int { KR_ROUTE_SCHUR = 0, KR_ROUTE_DIRECT = 1 };
enum : int { KR_OK = 0, KR_DROP = 1, KR_NOT_SPD = 2 };

struct KrigArgs {
  int m;                      // neighbourhood size
  const double* K;            // m x m
  const double* S;            // m x m inverse (Schur route only)
  const int* row_start;       // per std-res row, into pid / kp
  const int* pid;             // offset id of each present neighbour
  const double* kp;           // covariance of each present neighbour with the std-res centre
  const int* task_row;        // rows to solve, in order of decreasing cost
  const int* task_route;
  int ntasks;
  int* counter;               // next task
  double* x;                  // scratch, indexed like pid: the row being solved
  float* w;                   // output weights, indexed like pid
  int* status;                // per row: KR_OK, KR_DROP (weight sum NaN), KR_NOT_SPD
  double* scratch;            // per CTA: nmax (nmax + 1) / 2 (packed matrix) + m (v) + nmax (t) doubles, then m ints
  size_t slot;                // doubles per CTA slot
  int nmax;
};

// Shared memory of one CTA (dynamic).
struct KrigSmem {
  double D[KR_NB][KR_LDT];      // diagonal block / its factor
  double Di[KR_NB][KR_LDT];     // inverse of the factor
  double PA[KR_TILE][KR_LDP];   // panel rows (tile I)
  double PB[KR_TILE][KR_LDP];   // panel rows (tile J)
  double red[KR_RT / 32];
  int flag;
  int task;
  int nb;
};

__device__ __forceinline__ double kr_block_sum(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
  for (int i = 0; i < KR_RT / 32; i++) s += red[i];  // fixed order: every thread gets the same sum
  __syncthreads();
  return s;
}

// Factor the kb x kb block D in place (lower) with warp 0 and write its inverse to Di (zero above the diagonal).
// Returns false (block-uniform) if a pivot is not positive.
//
// This is the serial part of every panel.  Lane i owns row i of the factor and column i of the inverse, eight columns
// (rows) of them in registers at a time: inside such a group a step is one reciprocal square root, one product and
// independent updates, with the pivot row passed by shuffles; terms of earlier groups come from shared memory, eight
// chains side by side.  The terms are taken in the order of plain substitution.
__device__ __noinline__ bool kr_factor_diag(double (*D)[KR_LDT], double (*Di)[KR_LDT], int& flag, int kb) {
  const int lane = threadIdx.x & 31;
  constexpr unsigned ALL = 0xffffffffu;
  if (threadIdx.x < 32) {
    int bad = 0;
    double rinv = 0.0;  // lane i: 1 / L[i][i]
#pragma unroll 1
    for (int g = 0; g < kb && !bad; g += 8) {
      double a[8];
#pragma unroll
      for (int q = 0; q < 8; q++) a[q] = D[lane][g + q];
#pragma unroll 1
      for (int l = 0; l < g; l++) {
        const double x = D[lane][l];
        double c[8];
#pragma unroll
        for (int q = 0; q < 8; q++) c[q] = D[g + q][l];
#pragma unroll
        for (int q = 0; q < 8; q++) a[q] = fma(-x, c[q], a[q]);
      }
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const double d = __shfl_sync(ALL, a[j], g + j);
        if (g + j < kb && !(d > 0.0)) bad = 1;  // the same in every lane
        const double inv = rsqrt(fmax(d, 1e-300));
        if (lane == g + j) {
          rinv = inv;
          a[j] = d * inv;
        } else {
          a[j] *= inv;
        }
#pragma unroll
        for (int l = j + 1; l < 8; l++) a[l] = fma(-a[j], __shfl_sync(ALL, a[j], g + l), a[l]);
      }
#pragma unroll
      for (int q = 0; q < 8; q++)
        if (lane >= g + q) D[lane][g + q] = a[q];
      __syncwarp();
    }
    if (!bad) {
#pragma unroll 1
      for (int g = 0; g < kb; g += 8) {
        double s[8];
#pragma unroll
        for (int q = 0; q < 8; q++) s[q] = lane == g + q ? 1.0 : 0.0;
#pragma unroll 1
        for (int l = 0; l < g; l++) {
          const double x = Di[l][lane];
          double c[8];
#pragma unroll
          for (int q = 0; q < 8; q++) c[q] = D[g + q][l];
#pragma unroll
          for (int q = 0; q < 8; q++) s[q] = fma(-c[q], x, s[q]);
        }
#pragma unroll
        for (int j = 0; j < 8; j++) {
          s[j] *= __shfl_sync(ALL, rinv, g + j);
#pragma unroll
          for (int l = j + 1; l < 8; l++) s[l] = fma(-D[g + l][g + j], s[j], s[l]);
        }
#pragma unroll
        for (int q = 0; q < 8; q++)
          if (g + q < kb) Di[g + q][lane] = s[q];
        __syncwarp();
      }
    }
    if (lane == 0) flag = bad;
  }
  __syncthreads();
  return !flag;
}
__device__ bool kr_factor_diag(KrigSmem& sm, int kb) { return kr_factor_diag(sm.D, sm.Di, sm.flag, kb); }

// Position of (i, j), j <= i, in a lower triangle packed by rows: row i starts at i (i + 1) / 2.
// 32 bits: a neighbourhood has at most 5000 voxels, its triangle 12.5 million entries.
__device__ __forceinline__ unsigned kr_at(int i, int j) { return (unsigned)i * (i + 1) / 2 + j; }

// c (8 x 8) += a (8 x 4) b (4 x 8) in FP64 by one warp: lane holds a[lane / 4][lane % 4], b[lane % 4][lane / 4] and
// c[lane / 4][2 (lane % 4) + {0, 1}].  The matrix instruction's rate is that of the scalar FP64 FMAs, but its operands
// are spread over the warp: 2 loads of shared memory feed 256 products, where a 2 x 4 register tile per thread takes
// 6 loads for as many and waits on them.
__device__ __forceinline__ void kr_dmma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// A warp's part (8 TA rows from row i, 8 TB columns from column j) of the 64 x 64 product PA PB^T over 32 columns.
template <int TA, int TB>
__device__ __forceinline__ void kr_tile64(const double (*PA)[KR_LDP], const double (*PB)[KR_LDP], int i, int j,
                                          double (&acc)[TA][TB][2]) {
  const int r = (threadIdx.x & 31) >> 2, k = threadIdx.x & 3;
#pragma unroll
  for (int a = 0; a < TA; a++)
#pragma unroll
    for (int b = 0; b < TB; b++) acc[a][b][0] = acc[a][b][1] = 0.0;
#pragma unroll 4
  for (int l = 0; l < KR_NB; l += 4) {
    double pa[TA], pb[TB];
#pragma unroll
    for (int a = 0; a < TA; a++) pa[a] = PA[i + 8 * a + r][l + k];
#pragma unroll
    for (int b = 0; b < TB; b++) pb[b] = PB[j + 8 * b + r][l + k];
#pragma unroll
    for (int a = 0; a < TA; a++)
#pragma unroll
      for (int b = 0; b < TB; b++) kr_dmma(acc[a][b], pa[a], pb[b]);
  }
}

// Panel rows times the inverse of the diagonal factor: out(i, j) = sum_{l <= j} PA[i][l] Di[j][l] for i < ch, j < kb.
// Lane j of a warp takes several rows i side by side (independent chains of terms).
template <int NT, class Out>
__device__ __forceinline__ void kr_panel64(const double (*PA)[KR_LDP], const double (*Di)[KR_LDT], int ch, int kb,
                                           Out&& out) {
  constexpr int NW = NT / 32, Q = KR_TILE / NW;
  const int j = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (j >= kb) return;
  double s[Q];
#pragma unroll
  for (int q = 0; q < Q; q++) s[q] = 0.0;
  for (int l = 0; l <= j; l++) {
    const double d = Di[j][l];
#pragma unroll
    for (int q = 0; q < Q; q++) s[q] = fma(PA[warp + NW * q][l], d, s[q]);
  }
#pragma unroll
  for (int q = 0; q < Q; q++)
    if (warp + NW * q < ch) out(warp + NW * q, j, s[q]);
}

// In-place Cholesky M = L L^T of the n x n matrix (lower triangle, packed by rows: kr_at).  The 32 x 32 diagonal
// blocks of the result hold the inverses of L's diagonal blocks, which is what the solves multiply by.
__device__ bool kr_cholesky(double* M, int n, KrigSmem& sm) {
  static_assert(KR_RT == 512, "the trailing update gives each of 16 warps a 16 x 16 part of a tile");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // rows i0..i0+64 (below n) of the panel at column k0
  auto load_panel = [&](double (*P)[KR_LDP], int i0, int k0, int kb) {
    constexpr int NW = KR_RT / 32;
    double t[KR_TILE / NW];
#pragma unroll
    for (int q = 0; q < KR_TILE / NW; q++) {
      const int i = i0 + warp + NW * q;
      t[q] = (i < n && lane < kb) ? M[kr_at(i, k0 + lane)] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < KR_TILE / NW; q++) P[warp + NW * q][lane] = t[q];
  };
  for (int k0 = 0; k0 < n; k0 += KR_NB) {
    const int kb = min(KR_NB, n - k0);
    for (int i = warp; i < kb; i += KR_RT / 32) sm.D[i][lane] = lane <= i ? M[kr_at(k0 + i, k0 + lane)] : 0.0;
    __syncthreads();
    if (!kr_factor_diag(sm, kb)) return false;
    for (int i = warp; i < kb; i += KR_RT / 32)
      if (lane <= i) M[kr_at(k0 + i, k0 + lane)] = sm.Di[i][lane];
    const int r0 = k0 + kb;
    // panel: L[i, k0:k0+kb] = A[i, k0:k0+kb] Di^T, in chunks of KR_TILE rows
    for (int c0 = r0; c0 < n; c0 += KR_TILE) {
      __syncthreads();
      load_panel(sm.PA, c0, k0, kb);
      __syncthreads();
      kr_panel64<KR_RT>(sm.PA, sm.Di, min(KR_TILE, n - c0), kb,
                 [&](int i, int j, double x) { M[kr_at(c0 + i, k0 + j)] = x; });
    }
    __syncthreads();
    // trailing update A[i, j] -= L[i, panel] . L[j, panel] for r0 <= j <= i < n, 64 x 64 tiles (kb = 32 where one is left)
    const int T = (n - r0 + KR_TILE - 1) / KR_TILE;
    for (int tI = 0; tI < T; tI++) {
      const int i0 = r0 + tI * KR_TILE;
      load_panel(sm.PA, i0, k0, kb);
      for (int tJ = 0; tJ <= tI; tJ++) {
        const int j0 = r0 + tJ * KR_TILE;
        __syncthreads();
        load_panel(sm.PB, j0, k0, kb);
        // a warp's 16 x 16 part; its old values are fetched before the product, which covers their latency
        const int wi = 16 * (warp >> 2), wj = 16 * (warp & 3);
        const int ti = i0 + wi + (lane >> 2), tj = j0 + wj + 2 * (lane & 3);
        const bool part = i0 + wi < n && j0 + wj <= i0 + wi + 15;  // not all outside the lower triangle
        double old[2][2][2], acc[2][2][2];
#pragma unroll
        for (int e = 0; e < 8; e++) {
          const int i = ti + 8 * (e >> 2), j = tj + 8 * ((e >> 1) & 1) + (e & 1);
          old[e >> 2][(e >> 1) & 1][e & 1] = (i < n && j <= i) ? M[kr_at(i, j)] : 0.0;
        }
        __syncthreads();
        if (part) {
          kr_tile64<2, 2>(sm.PA, sm.PB, wi, wj, acc);
#pragma unroll
          for (int e = 0; e < 8; e++) {
            const int i = ti + 8 * (e >> 2), j = tj + 8 * ((e >> 1) & 1) + (e & 1);
            if (i < n && j <= i) M[kr_at(i, j)] = old[e >> 2][(e >> 1) & 1][e & 1] - acc[e >> 2][(e >> 1) & 1][e & 1];
          }
        }
      }
      __syncthreads();
    }
  }
  __syncthreads();
  return true;
}

// Solves L L^T x = b in place (b: n doubles in global memory), L from kr_cholesky.
__device__ void kr_solve(const double* L, int n, double* b, KrigSmem& sm) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nblk = (n + KR_NB - 1) / KR_NB;
  auto load_inverse = [&](int k0, int kb) {
    __syncthreads();
    for (int i = warp; i < kb; i += KR_RT / 32) sm.Di[i][lane] = lane <= i ? L[kr_at(k0 + i, k0 + lane)] : 0.0;
    __syncthreads();
  };
  // forward: y_k = Di (b_k - sum_{l<k} L_kl y_l), right-looking updates
  for (int kbk = 0; kbk < nblk; kbk++) {
    const int k0 = kbk * KR_NB, kb = min(KR_NB, n - k0);
    load_inverse(k0, kb);
    if (tid < kb) {
      double s = 0.0;
      for (int l = 0; l <= tid; l++) s += sm.Di[tid][l] * b[k0 + l];
      sm.PA[0][tid] = s;
    }
    __syncthreads();
    if (tid < kb) b[k0 + tid] = sm.PA[0][tid];
    __syncthreads();
    for (int i = k0 + kb + tid; i < n; i += KR_RT) {
      const double* Li = L + kr_at(i, k0);
      double s = 0.0;
#pragma unroll 8
      for (int l = 0; l < kb; l++) s += Li[l] * sm.PA[0][l];
      b[i] -= s;
    }
  }
  // backward: x_k = Di^T (y_k - sum_{l>k} L_lk^T x_l)
  for (int kbk = nblk - 1; kbk >= 0; kbk--) {
    const int k0 = kbk * KR_NB, kb = min(KR_NB, n - k0);
    load_inverse(k0, kb);
    if (tid < kb) {
      double s = 0.0;
      for (int l = tid; l < kb; l++) s += sm.Di[l][tid] * b[k0 + l];
      sm.PA[0][tid] = s;
    }
    __syncthreads();
    if (tid < kb) b[k0 + tid] = sm.PA[0][tid];
    __syncthreads();
    for (int i = tid; i < k0; i += KR_RT) {
      double s = 0.0;
#pragma unroll 8
      for (int l = 0; l < kb; l++) s += L[kr_at(k0 + l, i)] * sm.PA[0][l];
      b[i] -= s;
    }
  }
  __syncthreads();
}

// Dense products out[r] = sum_j Mat[rows[r]][j] v[j] over the m offsets, four rows of a warp side by side: the rows are
// read from L2, and one at a time the warp waits a latency for every 256 B.
__device__ void kr_rows_dot(const double* Mat, int m, const int* rows, int nrows, const double* v, double* out) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int r0 = 4 * warp; r0 < nrows; r0 += 4 * (KR_RT / 32)) {
    const double* Mr[4];
    double s[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      Mr[q] = Mat + (size_t)rows[min(r0 + q, nrows - 1)] * m;
      s[q] = 0.0;
    }
#pragma unroll 2
    for (int j = lane; j < m; j += 32) {
      const double vj = v[j];
#pragma unroll
      for (int q = 0; q < 4; q++) s[q] += Mr[q][j] * vj;
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
      for (int o = 16; o > 0; o >>= 1) s[q] += __shfl_xor_sync(0xffffffffu, s[q], o);
      if (lane == 0 && r0 + q < nrows) out[r0 + q] = s[q];
    }
  }
}

// M = the lower triangle of Mat[rows][rows] (n rows), packed: one warp per row.
__device__ void kr_gather(double* M, const double* Mat, int m, const int* rows, int n) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = warp; i < n; i += KR_RT / 32) {
    const double* Mr = Mat + (size_t)rows[i] * m;
#pragma unroll 4
    for (int j = lane; j <= i; j += 32) M[kr_at(i, j)] = Mr[rows[j]];
  }
}

// ---------------------------------------------------------------- K^-1 over the whole GPU
// S = K^-1 of the neighbourhood covariance (m up to 5000), once per volume:
//   right-looking blocked Cholesky K = L L^T in panels of KR_NB columns: the diagonal block by one CTA
//   (k_chol_diag, which also keeps the inverse of the block's factor), the panel below it by one CTA per 64 rows
//   (k_chol_panel), the trailing update by one CTA per 64 x 64 tile of the lower triangle (k_chol_update);
//   X = L^-1 one block row at a time, X_ij = -Dinv_i sum_{j <= k < i} L_ik X_kj, one CTA per block column
//   (k_trinv_row);  S = X^T X, one CTA per 32 x 32 tile of the lower triangle, stored to both triangles so that S is
//   exactly symmetric (k_trinv_gram).
// A pivot that is not positive clears *ok and every later launch returns at once.

// The kb x kb diagonal block at k0: factored in place, its factor's inverse to Dinv[k0 / KR_NB] (32 x 32, zero
// outside kb x kb).
__global__ void __launch_bounds__(KR_NT) k_chol_diag(double* M, int n, int k0, double* Dinv, int* ok) {
  __shared__ double D[KR_NB][KR_LDT], Di[KR_NB][KR_LDT];
  __shared__ int flag;
  if (!*ok) return;
  const int kb = min(KR_NB, n - k0), tid = threadIdx.x;
  for (int e = tid; e < KR_NB * KR_NB; e += KR_NT) {
    const int i = e / KR_NB, j = e % KR_NB;
    D[i][j] = (i < kb && j <= i) ? M[(size_t)(k0 + i) * n + k0 + j] : 0.0;
    Di[i][j] = 0.0;
  }
  __syncthreads();
  const bool good = kr_factor_diag(D, Di, flag, kb);
  if (!good) {
    if (tid == 0) *ok = 0;
    return;
  }
  double* Dg = Dinv + (size_t)(k0 / KR_NB) * KR_NB * KR_NB;
  for (int e = tid; e < KR_NB * KR_NB; e += KR_NT) {
    const int i = e / KR_NB, j = e % KR_NB;
    if (i < kb && j <= i) M[(size_t)(k0 + i) * n + k0 + j] = D[i][j];
    Dg[e] = (i < kb && j < kb) ? Di[i][j] : 0.0;
  }
}

// L[i, k0:k0+kb] = A[i, k0:k0+kb] Dinv^T for the 64 rows i of this CTA below the diagonal block.
__global__ void __launch_bounds__(KR_NT) k_chol_panel(double* M, int n, int k0, const double* Dinv, const int* ok) {
  __shared__ double Di[KR_NB][KR_LDT], PA[KR_TILE][KR_LDP];
  if (!*ok) return;
  const int kb = min(KR_NB, n - k0), tid = threadIdx.x;
  const int c0 = k0 + kb + blockIdx.x * KR_TILE, ch = min(KR_TILE, n - c0);
  const double* Dg = Dinv + (size_t)(k0 / KR_NB) * KR_NB * KR_NB;
  for (int e = tid; e < KR_NB * KR_NB; e += KR_NT) Di[e / KR_NB][e % KR_NB] = Dg[e];
  for (int e = tid; e < KR_TILE * KR_NB; e += KR_NT) {
    const int i = e / KR_NB, l = e % KR_NB;
    PA[i][l] = (i < ch && l < kb) ? M[(size_t)(c0 + i) * n + k0 + l] : 0.0;
  }
  __syncthreads();
  kr_panel64<KR_NT>(PA, Di, ch, kb, [&](int i, int j, double x) { M[(size_t)(c0 + i) * n + k0 + j] = x; });
}

// Lower-triangle tile index b -> (tI, tJ), tJ <= tI.
__device__ __forceinline__ void kr_tri_tile(int b, int* tI, int* tJ) {
  int i = (int)((sqrt(8.0 * (double)b + 1.0) - 1.0) * 0.5);
  while (i * (i + 1) / 2 > b) i--;
  while ((i + 1) * (i + 2) / 2 <= b) i++;
  *tI = i;
  *tJ = b - i * (i + 1) / 2;
}

// A[i, j] -= L[i, panel] . L[j, panel] on one 64 x 64 tile of the trailing lower triangle.
__global__ void __launch_bounds__(KR_NT) k_chol_update(double* M, int n, int k0, const int* ok) {
  __shared__ double PA[KR_TILE][KR_LDP], PB[KR_TILE][KR_LDP];
  if (!*ok) return;
  const int kb = min(KR_NB, n - k0), r0 = k0 + kb, tid = threadIdx.x;
  int tI, tJ;
  kr_tri_tile(blockIdx.x, &tI, &tJ);
  const int i0 = r0 + tI * KR_TILE, j0 = r0 + tJ * KR_TILE;
  const int ni = min(KR_TILE, n - i0), nj = min(KR_TILE, n - j0);
  for (int e = tid; e < KR_TILE * KR_NB; e += KR_NT) {
    const int i = e / KR_NB, l = e % KR_NB;
    PA[i][l] = (i < ni && l < kb) ? M[(size_t)(i0 + i) * n + k0 + l] : 0.0;
    PB[i][l] = (i < nj && l < kb) ? M[(size_t)(j0 + i) * n + k0 + l] : 0.0;
  }
  __syncthreads();
  static_assert(KR_NT == 256, "each of 8 warps takes a 32 x 16 part");
  const int lane = tid & 31, wi = 32 * (tid >> 7), wj = 16 * ((tid >> 5) & 3);
  double acc[4][2][2];
  kr_tile64<4, 2>(PA, PB, wi, wj, acc);
#pragma unroll
  for (int e = 0; e < 16; e++) {
    const int i = i0 + wi + 8 * (e >> 2) + (lane >> 2), j = j0 + wj + 8 * ((e >> 1) & 1) + 2 * (lane & 3) + (e & 1);
    if (i < n && j <= i) M[(size_t)i * n + j] -= acc[e >> 2][(e >> 1) & 1][e & 1];
  }
}

// One 32 x 32 tile product acc += A^T? B over shared tiles: acc[p][q] += sum_r TA[p][r] TB[r][q] (TRANS = false) or
// sum_r TA[r][p] TB[r][q] (TRANS = true); each of the 8 warps owns 8 rows by 16 columns of it (kr_tile_at).
template <bool TRANS>
__device__ __forceinline__ void kr_tile_mac(const double (*TA)[KR_LDP], const double (*TB)[KR_LDP],
                                            double (&acc)[2][2]) {
  const int r = (threadIdx.x & 31) >> 2, k = threadIdx.x & 3;
  const int p = 8 * (threadIdx.x >> 6) + r, q = 16 * ((threadIdx.x >> 5) & 1) + r;
#pragma unroll
  for (int l = 0; l < KR_NB; l += 4) {
    const double a = TRANS ? TA[l + k][p] : TA[p][l + k];
    kr_dmma(acc[0], a, TB[l + k][q]);
    kr_dmma(acc[1], a, TB[l + k][q + 8]);
  }
}
// Row p and column q in the tile of acc[e / 2][e % 2].
__device__ __forceinline__ void kr_tile_at(int e, int* p, int* q) {
  *p = 8 * (threadIdx.x >> 6) + ((threadIdx.x & 31) >> 2);
  *q = 16 * ((threadIdx.x >> 5) & 1) + 8 * (e >> 1) + 2 * (threadIdx.x & 3) + (e & 1);
}

// Loads the 32 x 32 tile of the n x n row-major matrix at block (bi, bj), zero outside n x n.
__device__ __forceinline__ void kr_load_tile(double (*T)[KR_LDP], const double* A, int n, int bi, int bj) {
  for (int e = threadIdx.x; e < KR_NB * KR_NB; e += KR_NT) {
    const int i = e / KR_NB, j = e % KR_NB, gi = bi * KR_NB + i, gj = bj * KR_NB + j;
    T[i][j] = (gi < n && gj < n) ? A[(size_t)gi * n + gj] : 0.0;
  }
}

// Block row bi of X = L^-1: CTA bj < bi computes X[bi][bj] = -Dinv_bi sum_{bj <= k < bi} L[bi][k] X[k][bj];
// CTA bj = bi writes X[bi][bi] = Dinv_bi.
__global__ void __launch_bounds__(KR_NT) k_trinv_row(const double* L, int n, int bi, const double* Dinv, double* X,
                                                     const int* ok) {
  __shared__ double TA[KR_NB][KR_LDP], TB[KR_NB][KR_LDP];
  if (!*ok) return;
  const int bj = blockIdx.x;
  const double* Dg = Dinv + (size_t)bi * KR_NB * KR_NB;
  double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
  if (bj == bi) {
#pragma unroll
    for (int e = 0; e < 4; e++) {
      int p, q;
      kr_tile_at(e, &p, &q);
      acc[e >> 1][e & 1] = Dg[p * KR_NB + q];
    }
  } else {
    for (int k = bj; k < bi; k++) {
      __syncthreads();
      kr_load_tile(TA, L, n, bi, k);
      kr_load_tile(TB, X, n, k, bj);
      __syncthreads();
      kr_tile_mac<false>(TA, TB, acc);
    }
    // X[bi][bj] = -Dinv_bi acc (acc through shared memory)
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 4; e++) {
      int p, q;
      kr_tile_at(e, &p, &q);
      TB[p][q] = acc[e >> 1][e & 1];
    }
    for (int e = threadIdx.x; e < KR_NB * KR_NB; e += KR_NT) TA[e / KR_NB][e % KR_NB] = Dg[e];
    __syncthreads();
    double r[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
    kr_tile_mac<false>(TA, TB, r);
#pragma unroll
    for (int e = 0; e < 4; e++) acc[e >> 1][e & 1] = -r[e >> 1][e & 1];
  }
#pragma unroll
  for (int e = 0; e < 4; e++) {
    int p, q;
    kr_tile_at(e, &p, &q);
    const int gi = bi * KR_NB + p, gj = bj * KR_NB + q;
    if (gi < n && gj < n) X[(size_t)gi * n + gj] = acc[e >> 1][e & 1];
  }
}

// S[ba][bb] = sum_{k >= ba} X[k][ba]^T X[k][bb] for the tile (ba >= bb) of this CTA, stored with its transpose.
__global__ void __launch_bounds__(KR_NT) k_trinv_gram(const double* X, int n, double* S, const int* ok) {
  __shared__ double TA[KR_NB][KR_LDP], TB[KR_NB][KR_LDP];
  if (!*ok) return;
  int ba, bb;
  kr_tri_tile(blockIdx.x, &ba, &bb);
  const int nb = (n + KR_NB - 1) / KR_NB;
  double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
  for (int k = ba; k < nb; k++) {
    __syncthreads();
    kr_load_tile(TA, X, n, k, ba);
    kr_load_tile(TB, X, n, k, bb);
    __syncthreads();
    kr_tile_mac<true>(TA, TB, acc);
  }
#pragma unroll
  for (int e = 0; e < 4; e++) {
    int p, q;
    kr_tile_at(e, &p, &q);
    const int gi = ba * KR_NB + p, gj = bb * KR_NB + q;
    if (gi < n && gj < n) {
      S[(size_t)gi * n + gj] = acc[e >> 1][e & 1];
      S[(size_t)gj * n + gi] = acc[e >> 1][e & 1];
    }
  }
}

__global__ void __launch_bounds__(KR_RT, 2) k_kriging_rows(KrigArgs a) {
  extern __shared__ __align__(16) unsigned char kr_smraw[];
  KrigSmem& sm = *reinterpret_cast<KrigSmem*>(kr_smraw);
  const int tid = threadIdx.x;
  double* M = a.scratch + (size_t)blockIdx.x * a.slot;
  double* v = M + kr_at(a.nmax, 0);  // the packed lower triangle of an nmax x nmax matrix
  double* t = v + a.m;
  int* ids = reinterpret_cast<int*>(t + a.nmax);
  const int m = a.m;
  for (;;) {
    __syncthreads();
    if (tid == 0) sm.task = atomicAdd(a.counter, 1);
    __syncthreads();
    const int ti = sm.task;
    if (ti >= a.ntasks) break;
    const int row = a.task_row[ti], route = a.task_route[ti];
    const int r0 = a.row_start[row], cnt = a.row_start[row + 1] - r0;
    const int* pid = a.pid + r0;
    const double* k = a.kp + r0;
    double* x = a.x + r0;
    bool ok = true;
    if (route == KR_ROUTE_DIRECT) {
      const int n = cnt;
      kr_gather(M, a.K, m, pid, n);
      for (int i = tid; i < n; i += KR_RT) x[i] = k[i];
      __syncthreads();
      ok = kr_cholesky(M, n, sm);
      if (ok) kr_solve(M, n, x, sm);
    } else {
      // v0 = (k_A, 0) over the offsets; absent offsets B in ascending order
      for (int j = tid; j < m; j += KR_RT) {
        v[j] = 0.0;
        ids[j] = 1;
      }
      __syncthreads();
      for (int i = tid; i < cnt; i += KR_RT) {
        v[pid[i]] = k[i];
        ids[pid[i]] = 0;
      }
      __syncthreads();
      if (tid < 32) {  // compact the absent offsets (ascending) in place: a chunk is read before anything is written to it
        int nb = 0;
        for (int j0 = 0; j0 < m; j0 += 32) {
          const int j = j0 + tid;
          const bool absent = j < m && ids[j];
          const unsigned mask = __ballot_sync(0xffffffffu, absent);
          if (absent) ids[nb + __popc(mask & ((1u << tid) - 1))] = j;
          nb += __popc(mask);
          __syncwarp();
        }
        if (tid == 0) sm.nb = nb;
      }
      __syncthreads();
      const int nb = sm.nb;
      if (nb > 0) {
        kr_rows_dot(a.S, m, ids, nb, v, t);  // t = [S v0]_B
        kr_gather(M, a.S, m, ids, nb);
        __syncthreads();
        ok = kr_cholesky(M, nb, sm);
        if (ok) {
          kr_solve(M, nb, t, sm);
          for (int q = tid; q < nb; q += KR_RT) v[ids[q]] = -t[q];
          __syncthreads();
        }
      }
      if (ok) {
        kr_rows_dot(a.S, m, pid, cnt, v, x);
        __syncthreads();
      }
    }
    int st = KR_OK;
    if (!ok) {
      st = KR_NOT_SPD;
    } else {
      double s = 0.0;
      if (tid < KR_NT)  // the order of the sum does not depend on the size of the CTA
        for (int i = tid; i < cnt; i += KR_NT) s += x[i];
      double wsum = kr_block_sum(s, sm.red);
      if (isnan(wsum)) {
        st = KR_DROP;
      } else {
        if (wsum == 0.0) wsum = 1.0;  // kriging_matrix.h:318-319
        for (int i = tid; i < cnt; i += KR_RT) a.w[r0 + i] = (float)(x[i] / wsum);
      }
    }
    if (tid == 0) a.status[row] = st;
  }
}

}  // namespace drb
