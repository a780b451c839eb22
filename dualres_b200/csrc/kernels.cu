// Device kernels of the dual-resolution GP-HMC sampler.
//
// The sampler keeps every chain's state in the spectral domain of the
// circulant embedding: u = IFFT(mu) and q = IFFT(p) (unnormalised).  In that
// basis the reference's operators (include/dualres/MultiResParameters.h) become:
//   position update  mu* += FFT(IFFT(p) eps/(N lambda_m))  ->  u* += eps q / lambda_m
//   prior gradient   FFT(IFFT(mu)/(-N lambda))             ->  -u / lambda
//   log prior        -(1/2N) sum |IFFT(mu)|^2 / lambda       ->  -(1/2N) sum |u|^2 / lambda
//   kinetic energy   -(1/2N) sum |IFFT(p)|^2 / lambda_m      ->  -(1/2N) sum |q|^2 / lambda_m
// all element-wise, zeroed on S = {Re lambda <= 0} exactly as _low_rank_adjust
// does.  Only the data term needs real space: Re mu at the data voxels, and the
// scatter of the data gradient.  One gradient therefore costs one pruned
// forward transform (spectral -> real box) and one pruned inverse transform
// (real box -> spectral) instead of the reference's four full 3D FFTs.
//
// The state is split into the spectra of Re mu and Im mu, u = h + i g, each
// Hermitian (h(-k) = conj h(k)), so the planes kz = 0 .. E2/2 hold all of it:
// EZ = E2/2 + 1 planes, NH = EZ E1 E0 modes.  lambda is even in every axis, so
// the operators above act on h and g alike and never mix them.  Only h meets
// the data: the leapfrog steps carry h (half the modes through every kernel),
// and g, whose dynamics are element-wise and linear, is taken through all of an
// iteration's steps in registers by k_momentum.  Sums over all modes weight the
// planes 0 < kz < E2/2 by two (plane_weight).  Measured against the full complex
// state (64 chains on a 64^3 embedding): update 139 -> 73 us, forward / inverse z
// pass 20.4 / 18.1 -> 10.6 / 10.1 us, an iteration 6.1 -> 4.1 ms; 16 chains on
// 128^3: update 458 -> 252 us, z 38 / 34 -> 16 / 17 us (since then the plane kernels below:
// 68 and 177 us).
#include "common.cuh"
#include "drb.h"
#include "fft.cuh"
#include "tma.cuh"

namespace drb {

// e / d as __umulhi(e, box_div_magic(d)) for box positions (e < 2^15, 2 <= d <= 1024): the multiplier
// ceil(2^32 / d) gives the exact quotient there, without a division per element.
__device__ __forceinline__ uint32_t box_div_magic(int d) { return 0xFFFFFFFFu / (uint32_t)d + 1u; }

// Multiplicity of spectral plane z in a sum over all modes: its mirror image E2 - z is not stored.
__device__ __forceinline__ double plane_weight(int z, int E2) { return (z == 0 || 2 * z == E2) ? 1.0 : 2.0; }

// ----------------------------------------------------------------- twiddles
__device__ float2 g_tw_f[TW_TOTAL];
__device__ double2 g_tw_d[TW_TOTAL];

// ----------------------------------------------------------------- HMC parameters
// Device restatement of HMCParameters<float> (include/dualres/HMCParameters.h).
__device__ __forceinline__ float hmc_eps(const ChainState& h, double u01) {
  // :212-221  eps() = eps (warm-up) or max(eps * U(0.9, 1.1), eps0)
  if (h.warmup) return (float)h.eps;
  return (float)fmax(h.eps * (0.9 + 0.2 * u01), h.eps0);
}
__device__ __forceinline__ int hmc_steps(const ChainState& h) {  // :172-179
  return h.eps_start_found ? h.integrator_steps : 1;
}
__device__ __forceinline__ int hmc_save_iteration(const ChainState& h) {  // :158-161
  return (h.iteration > h.burnin) && ((h.iteration - h.burnin) % h.thin == 0);
}
// During the burn-in the step size follows the rate min(1, R): where log R lies a few units below zero, its rounding (1e-4 to
// 1e-3) becomes a difference of that size between the step sizes of two summation orders, and the chains part there.
__device__ void hmc_update(ChainState& h, float mh_rate_f) {  // :259-297
  const double mh_rate = (double)mh_rate_f;
  if (h.iteration == h.burnin) {
    h.warmup = 0;
    h.eps_start_found = 1;
    if (h.eps_bar > h.eps0) h.eps = h.eps_bar;
  }
  if (h.warmup) {
    if (!h.eps_start_found) {
      if (h.iteration == 0) h.A = 2 * (int)(mh_rate > 0.5) - 1;
      if (pow(mh_rate, h.A) > pow(2.0, -h.A)) {
        h.eps *= pow(2.0, h.A);
      } else {
        h.eps_start_found = 1;
        h.eps_target = log(10.0 * h.eps);
      }
    } else {
      const double it = (double)h.iteration;
      h.h_bar = (1 - 1 / (it + h.t0)) * h.h_bar + (h.mh_target - mh_rate) / (it + h.t0);
      h.eps = exp(h.eps_target - (double)sqrtf((float)h.iteration) * h.h_bar / h.gamma);
      h.eps = fmax(h.eps, h.eps0);
      const double pk = pow((double)(float)h.iteration, -h.kappa);
      h.eps_bar = exp(pk * log(h.eps) + (1 - pk) * log(h.eps_bar));
    }
  } else {
    h.mh_running_sum += mh_rate;
  }
  h.iteration++;
}

// Marsaglia & Tsang (2000), "A simple method for generating gamma variables",
// ACM TOMS 26(3); shape < 1 by Gamma(a) = Gamma(a + 1) U^(1/a).  Draws come
// from the counter stream (stream, chain, iteration, base + attempt).  The
// loop is bounded; a failure sets *err and returns the mean.
__device__ double gamma_draw(double shape, double scale, uint64_t seed, uint32_t stream, uint32_t chain,
                             uint32_t iter, uint32_t base, int* err) {
  double boost = 1.0;
  if (shape < 1.0) {
    const u32x4 r = philox(u32x4{base + 1000u, iter, chain, stream}, seed);
    boost = pow(u01d(r.x, r.y), 1.0 / shape);
    shape += 1.0;
  }
  const double d = shape - 1.0 / 3.0, c = 1.0 / sqrt(9.0 * d);
  for (uint32_t a = 0; a < 64; a++) {
    const u32x4 r1 = philox(u32x4{base + 2 * a, iter, chain, stream}, seed);
    const u32x4 r2 = philox(u32x4{base + 2 * a + 1, iter, chain, stream}, seed);
    const double x = box_muller_d(u01d(r1.x, r1.y), u01d(r1.z, r1.w)).x;
    double v = 1.0 + c * x;
    if (v <= 0.0) continue;
    v = v * v * v;
    const double u = u01d(r2.x, r2.y);
    if (log(u) < 0.5 * x * x + d - d * v + d * log(v)) return d * v * boost * scale;
  }
  *err += 1;
  return shape * scale;
}

// ----------------------------------------------------------------- pass kernel
// Batched 1D FFT along the middle axis of [A][n][B] arrays, one tile of 32
// lines (line = a * B + b) of one chain (blockIdx.y) per block: the y passes of
// the x-line path, the initial state and the unpruned 3D transforms.
template <int N> struct PassCfg {
  static constexpr int NT = 256;
};

template <int N, int DIR, class C>
__global__ void __launch_bounds__(PassCfg<N>::NT) k_pass(PassArgs a, DevChains ch, const C* __restrict__ tw) {
  grid_dep_wait();
  constexpr int TL = TILE_LINES, P = TILE_LINES + 1, NT = PassCfg<N>::NT;
  extern __shared__ __align__(16) unsigned char smraw[];
  C* sm = reinterpret_cast<C*>(smraw);
  __shared__ long long s_in0[TL], s_out0[TL];  // per tile line: index of its element 0 in the input / output
  const int c = blockIdx.y;
  if (a.step >= 0 && ch.st != nullptr && a.step > ch.st[c].L_cur) return;
  const long long lines = (long long)a.A * a.B;
  const long long l0 = (long long)blockIdx.x * TL;
  const int B = a.B, n_in = a.n_in, n_out = a.n_out;
  if (threadIdx.x < TL) {
    // line lam = a * B + b starts at (a * n) * B + b; computed once per line rather than per element
    const long long lam = l0 + threadIdx.x;
    const long long aa = lam / B, bb = lam - aa * B;
    s_in0[threadIdx.x] = aa * n_in * B + bb;
    s_out0[threadIdx.x] = aa * n_out * B + bb;
  }
  __syncthreads();
  const int nl = (int)min((long long)TL, lines - l0);
  // bounds of the indices (checked builds only): a chain's stride in the input / output (the whole array when there is
  // one field)
  const long long in_lim = a.in_cs > 0 ? a.in_cs : 0x7fffffffffffffffLL;
  const long long out_lim = a.out_cs > 0 ? a.out_cs : 0x7fffffffffffffffLL;
  const C* in = reinterpret_cast<const C*>(a.in) + (long long)c * a.in_cs;
  C* out = reinterpret_cast<C*>(a.out) + (long long)c * a.out_cs;
  auto load = [&](int l, int i) -> C {
    C val = mk((decltype(C().x))0, (decltype(C().x))0);
    if (l < nl && i < n_in) {
      const long long idx = s_in0[l] + (long long)i * B;
      if (in_bounds(idx, in_lim, ch.err)) val = in[idx];
    }
    return val;
  };
  // the loads of a thread are issued before its shared-memory stores, up to 16 at a time: PER independent loads in
  // flight per round (tiles of a whole number of block-widths)
  constexpr int PER = TL * N / NT;
  constexpr int CH = PER > 16 ? 16 : PER;
  if constexpr (PER >= 1 && PER * NT == TL * N && PER % CH == 0) {
#pragma unroll 1
    for (int k0 = 0; k0 < PER; k0 += CH) {
      C r[CH];
#pragma unroll
      for (int k = 0; k < CH; k++) {
        const int e = threadIdx.x + (k0 + k) * NT;
        r[k] = B == 1 ? load(e / N, e % N) : load(e % TL, e / TL);
      }
#pragma unroll
      for (int k = 0; k < CH; k++) {
        const int e = threadIdx.x + (k0 + k) * NT;
        if (B == 1) sm[(e % N) * P + e / N] = r[k];
        else sm[(e / TL) * P + e % TL] = r[k];
      }
    }
  } else if (B == 1) {
    for (int e = threadIdx.x; e < TL * N; e += NT) {
      const int l = e / N, i = e % N;
      sm[i * P + l] = load(l, i);
    }
  } else {
    for (int e = threadIdx.x; e < TL * N; e += NT) {
      const int i = e / TL, l = e % TL;
      sm[i * P + l] = load(l, i);
    }
  }
  __syncthreads();
  fft_smem<N, DIR, TL, NT, C>(sm, 1, P, TL, tw + tw_offset(N));

  auto store = [&](int l, int k) {
    if (l >= nl || k >= n_out) return;
    const long long idx = s_out0[l] + (long long)k * B;
    if (in_bounds(idx, out_lim, ch.err)) out[idx] = sm[k * P + l];
  };
  if (B == 1) {
    for (int e = threadIdx.x; e < TL * N; e += NT) store(e / N, e % N);
  } else {
    for (int e = threadIdx.x; e < TL * N; e += NT) store(e % TL, e / TL);
  }
}

// ----------------------------------------------------------------- z passes
// The z transforms between the real box and T2 (the planes 0 .. E2/2 of its
// half spectrum along z).  A tile line is a pair of x-adjacent real lines a, b
// carried as one complex line a + i b, so one transform of length E2 serves two
// lines and T2 moves as float4 (the pair's A(k), B(k)):
//   inverse  gD in the box -> Z, then A(k) = (Z(k) + conj Z(-k)) / 2 and
//            B(k) = (Z(k) - conj Z(-k)) / 2i for k = 0 .. E2/2;
//   forward  Z(k) = A(k) + i B(k), Z(-k) = conj A(k) + i conj B(k), whose
//            transform's real and imaginary parts are Re mu on the two lines
//            (in the planes k = 0 and E2/2, real for a real field, the real parts are taken).
// CPB = 1: TL pair lines of one chain (blockIdx.y): 32, or 8 when 32 would give
// fewer blocks than two per SM.  CPB = 8: 4 consecutive pair lines of 8 chains
// (chain group blockIdx.y): the chain-minor arrays mu_D, mu_O and gD are then
// touched 8 chains x 4 bytes contiguously, one 32-byte sector instead of one
// value per 256-byte row, and T2 in runs of 64 bytes.
template <int N, int TL> struct ZCfg {
  static constexpr int WANT = TL * N / 8;  // a thread holds 8 elements
  static constexpr int NT = WANT < 32 ? 32 : (WANT > 256 ? 256 : WANT);
  static constexpr int P = TL;             // element pitch: threads run along the lines, whole rows at a time
  static constexpr int SMEM = N * P * 8;
};

// Per chain of a tile: whether it takes part in this step.
template <int CPB>
__device__ __forceinline__ bool z_chain_active(const ZArgs& a, const DevChains& ch, int c) {
  if (CPB > 1 && c >= ch.C) return false;
  return a.step < 0 || ch.st == nullptr || a.step <= ch.st[c].L_cur;
}

template <int N, int TL, int CPB, int PLAN>
__global__ void __launch_bounds__(ZCfg<N, TL>::NT) k_zinv(ZArgs a, DevVolume v, DevChains ch, const float2* __restrict__ tw) {
  grid_dep_wait();
  constexpr int NT = ZCfg<N, TL>::NT, P = ZCfg<N, TL>::P, LPC = TL / CPB, H = N / 2;
  extern __shared__ __align__(16) unsigned char smraw[];
  float2* sm = reinterpret_cast<float2*>(smraw);
  const int l = threadIdx.x % TL;          // NT is a multiple of TL: a thread keeps its line
  constexpr int KS = NT / TL;              // elements between a thread's consecutive ones
  const int c = blockIdx.y * CPB + l / LPC;
  const int lp = blockIdx.x * LPC + l % LPC;
  const bool act = z_chain_active<CPB>(a, ch, c);
  if (CPB == 1 && !act) return;
  const int plane = v.by * v.bx;
  const bool on = act && 2 * lp < plane;
  const long long box = (long long)plane * v.bz;
  constexpr int PER = (N + KS - 1) / KS, CH = PER > 8 ? 8 : PER;
  const int k0 = threadIdx.x / TL;
#pragma unroll 1
  for (int q0 = 0; q0 < PER; q0 += CH) {
    int2 j[CH];
#pragma unroll
    for (int q = 0; q < CH; q++) {
      const int z = k0 + (q0 + q) * KS;
      const long long idx = (long long)z * plane + 2 * lp;
      j[q] = make_int2(-1, -1);
      if (on && z < v.bz && in_bounds(idx + 1, box, ch.err)) j[q] = __ldg(reinterpret_cast<const int2*>(v.box_to_d + idx));
    }
    float2 r[CH];
#pragma unroll
    for (int q = 0; q < CH; q++) {
      r[q] = make_float2(0.f, 0.f);
      if (j[q].x >= 0 && in_bounds(j[q].x, v.n_h, ch.err)) r[q].x = ch.gD[(long long)j[q].x * ch.Cp + c];
      if (j[q].y >= 0 && in_bounds(j[q].y, v.n_h, ch.err)) r[q].y = ch.gD[(long long)j[q].y * ch.Cp + c];
    }
#pragma unroll
    for (int q = 0; q < CH; q++)
      if (N % KS == 0 || k0 + (q0 + q) * KS < N) sm[(k0 + (q0 + q) * KS) * P + l] = r[q];
  }
  __syncthreads();
  fft_smem<N, +1, TL, NT, float2, PLAN>(sm, 1, P, TL, tw + tw_offset(N));
  if (!on) return;
  float2* T = ch.T2 + (long long)c * ch.t2_stride + 2 * lp;
  for (int k = k0; k <= H; k += KS) {
    const float2 zk = sm[k * P + l], zm = sm[((N - k) % N) * P + l];
    if (in_bounds((long long)k * plane + 2 * lp + 1, ch.t2_stride, ch.err))
      *reinterpret_cast<float4*>(T + (long long)k * plane) =
          make_float4(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y), 0.5f * (zk.y + zm.y), 0.5f * (zm.x - zk.x));
  }
}

template <int N, int TL, int CPB, int PLAN>
__global__ void __launch_bounds__(ZCfg<N, TL>::NT) k_zfwd(ZArgs a, DevVolume v, DevChains ch, const float2* __restrict__ tw) {
  grid_dep_wait();
  constexpr int NT = ZCfg<N, TL>::NT, P = ZCfg<N, TL>::P, LPC = TL / CPB, H = N / 2;
  extern __shared__ __align__(16) unsigned char smraw[];
  float2* sm = reinterpret_cast<float2*>(smraw);
  const int l = threadIdx.x % TL;
  constexpr int KS = NT / TL;
  const int c = blockIdx.y * CPB + l / LPC;
  const int lp = blockIdx.x * LPC + l % LPC;
  const bool act = z_chain_active<CPB>(a, ch, c);
  if (CPB == 1 && !act) return;
  const int plane = v.by * v.bx;
  const bool on = act && 2 * lp < plane;
  const float2* T = ch.T2 + (long long)c * ch.t2_stride + 2 * lp;
  const int k0 = threadIdx.x / TL;
  // T2 is read for the last time before the next inverse z pass: streaming loads, evicted first
  auto load = [&](int k) {
    if (on && k <= H && in_bounds((long long)k * plane + 2 * lp + 1, ch.t2_stride, ch.err))
      return __ldcs(reinterpret_cast<const float4*>(T + (long long)k * plane));
    return make_float4(0.f, 0.f, 0.f, 0.f);
  };
  // k = 0 .. H-1 over the threads, and the threads of k = 0 also take k = H
  constexpr int PER = (H + KS - 1) / KS, CH = PER > 4 ? 4 : PER;
  float4 rh = make_float4(0.f, 0.f, 0.f, 0.f);
  if (k0 == 0) rh = load(H);
#pragma unroll 1
  for (int q0 = 0; q0 < PER; q0 += CH) {
    float4 r[CH];
#pragma unroll
    for (int q = 0; q < CH; q++) r[q] = load(k0 + (q0 + q) * KS);
#pragma unroll
    for (int q = 0; q < CH; q++) {
      const int k = k0 + (q0 + q) * KS;
      if (k == 0) {
        sm[l] = make_float2(r[q].x, r[q].z);
      } else if (k < H) {
        sm[k * P + l] = make_float2(r[q].x - r[q].w, r[q].y + r[q].z);
        sm[(N - k) * P + l] = make_float2(r[q].x + r[q].w, r[q].z - r[q].y);
      }
    }
  }
  if (k0 == 0) sm[H * P + l] = make_float2(rh.x, rh.z);
  __syncthreads();
  fft_smem<N, -1, TL, NT, float2, PLAN>(sm, 1, P, TL, tw + tw_offset(N));
  if (!on) return;
  // whether mu_O is written
  const bool wo = a.write_o == 1 || (a.write_o == 2 && ch.st != nullptr && a.step == ch.st[c].L_cur);
  float* mD = ch.muD + (long long)a.sel * v.n_h * ch.Cp + c;
  float* mO = ch.muO + (long long)a.sel * v.n_o * ch.Cp + c;
  const long long box = (long long)plane * v.bz;
  for (int z = k0; z < v.bz; z += KS) {
    const long long idx = (long long)z * plane + 2 * lp;
    if (!in_bounds(idx + 1, box, ch.err)) continue;
    const float2 m = cscale(sm[z * P + l], a.scale);
    const int2 j = __ldg(reinterpret_cast<const int2*>(v.box_to_d + idx));
    if (j.x >= 0 && in_bounds(j.x, v.n_h, ch.err)) mD[(long long)j.x * ch.Cp] = m.x;
    if (j.y >= 0 && in_bounds(j.y, v.n_h, ch.err)) mD[(long long)j.y * ch.Cp] = m.y;
    if (wo) {
      const int2 o = __ldg(reinterpret_cast<const int2*>(v.box_to_o + idx));
      if (o.x >= 0 && in_bounds(o.x, v.n_o, ch.err)) mO[(long long)o.x * ch.Cp] = m.x;
      if (o.y >= 0 && in_bounds(o.y, v.n_o, ch.err)) mO[(long long)o.y * ch.Cp] = m.y;
    }
  }
}

// ----------------------------------------------------------------- momentum and Im mu
// One launch per iteration, before its leapfrog steps, over the rows (z, y) of
// the half spectrum.  It draws the momentum (MultiResParameters.h:784-815),
// q = sqrt(N lambda_m) w with w(k) ~ CN(0, 2) iid over all N modes, as in the
// full spectrum (one Philox call per pair of x-adjacent modes), and splits it:
//   h part  sqrt(N lambda_m) (w(k) + conj w(-k)) / 2  -> Q, for the leapfrog kernels;
//   g part  sqrt(N lambda_m) (w(k) - conj w(-k)) / 2i, kept here.
// The g part of the state (Im mu) feels only the prior, so its whole trajectory
//   q -= (eps / 2) u / lambda;  L times { u += eps q / lambda_m;  q -= eps u / lambda (the last one halved) }
// is element-wise: it runs here in registers, 4 FMA per component and step, and
// reads and writes g once per iteration instead of once per step.  Energies of
// the g part and sum |w|^2 go to partial-sum entries nb_x + block (the leapfrog
// kernels' entries are 0 .. nb_x - 1).
// FIXED: the g part of a given momentum is read from Gq and left there (the h
// part is in Q), and SL_E0 receives sum |q|^2 / lambda_m; one chain at a time.
constexpr int MOM_ITEMS = 512;  // modes of a row group: 512 / E0 rows
constexpr int MOM_NT = 256;

template <bool FIXED>
__global__ void __launch_bounds__(MOM_NT) k_momentum(DevVolume v, DevChains ch) {
  grid_dep_wait();
  __shared__ float2 wa[FIXED ? 1 : MOM_ITEMS], wb[FIXED ? 1 : MOM_ITEMS];
  __shared__ double red[MOM_NT / 32];
  const int c = blockIdx.y;
  ChainState& st = ch.st[c];
  int L = st.L_cur;
  float eps = st.eps_cur;
  if constexpr (!FIXED) {
    // the arguments of MultiResParameters::update: eps() and integrator_steps() (gaussian_process_model.h:135); every
    // thread forms them, the first leaves them for the kernels that follow
    const u32x4 r = philox(u32x4{0u, (uint32_t)st.iteration, (uint32_t)(ch.chain0 + c), RNG_SCALAR}, ch.seed);
    eps = hmc_eps(st, u01d(r.x, r.y));
    L = st.done ? -1 : hmc_steps(st);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      if (L >= 0) st.eps_cur = eps;
      st.L_cur = L;
    }
  }
  if (L < 0) return;
  const int E0 = v.E0, E1 = v.E1, E2 = v.E2, acc = st.acc;
  const long long NH = v.NH;
  const float sh = st.sh, Nf = (float)v.N;
  const float2* Gs = ch.G + ((long long)c * 2 + acc) * NH;
  float2* Gd = ch.G + ((long long)c * 2 + (acc ^ 1)) * NH;
  float2* Qc = ch.Q + (long long)c * NH;
  double e0 = 0.0, lp0 = 0.0, lpl = 0.0, kl = 0.0;
  const int rows = v.EZ * E1, rpg = MOM_ITEMS / E0;  // E0 is a power of two <= 256
  for (int r0 = blockIdx.x * rpg; r0 < rows; r0 += gridDim.x * rpg) {
    const int nr = min(rpg, rows - r0), items = nr * E0;
    if constexpr (!FIXED) {
      __syncthreads();
      for (int p = threadIdx.x; p < items; p += MOM_NT) {
        // pairs of modes: the rows themselves, then their mirror images
        const int which = 2 * p >= items, i = 2 * p - which * items, row = r0 + i / E0, x = i % E0;
        int z = row / E1, y = row % E1;
        if (which) {
          z = z == 0 ? 0 : E2 - z;
          y = y == 0 ? 0 : E1 - y;
        }
        const long long gi = ((long long)z * E1 + y) * E0 + x;
        const u32x4 r = philox(u32x4{(uint32_t)(gi >> 1), (uint32_t)st.iteration, (uint32_t)(ch.chain0 + c),
                                     RNG_MOMENTUM}, ch.seed);
        float2* w = which ? wb : wa;
        w[i] = box_muller(u01f(r.x), u01f(r.y));
        w[i + 1] = box_muller(u01f(r.z), u01f(r.w));
      }
      __syncthreads();
    }
    for (int i = threadIdx.x; i < items; i += MOM_NT) {
      const int row = r0 + i / E0;
      const long long gi = (long long)r0 * E0 + i;
      const double wt = plane_weight(row / E1, E2);
      float2 u = __ldcs(Gs + gi);
      const float s = v.sinv[gi];
      const bool live = s > 0.0f;
      const float lm = s + sh;  // lambda_m = 1/lambda + sigma_h^-2 (MultiResParameters.h:735-738)
      float2 q;
      if constexpr (FIXED) {
        q = ch.Gq[gi];
        if (live) e0 += wt * ((double)(q.x * q.x + q.y * q.y) / (double)lm);
      } else {
        const int x = i % E0;
        const float2 w = wa[i], m = wb[i - x + (x == 0 ? 0 : E0 - x)];
        const float a = live ? 0.5f * sqrtf(Nf * lm) : 0.0f;
        // sum |w|^2 over all modes: each mode of the mirror plane is some m of this plane
        e0 += (double)(w.x * w.x + w.y * w.y);
        if (wt > 1.0) e0 += (double)(m.x * m.x + m.y * m.y);
        Qc[gi] = make_float2(a * (w.x + m.x), a * (w.y - m.y));
        q = make_float2(a * (w.y + m.y), a * (m.x - w.x));
      }
      if (live) {
        lp0 += wt * ((double)(u.x * u.x + u.y * u.y) * (double)s);
        const float kick = eps * s, half = 0.5f * kick, drift = eps / lm;
        q.x = fmaf(-half, u.x, q.x);
        q.y = fmaf(-half, u.y, q.y);
#pragma unroll 4
        for (int t = 1; t < L; t++) {
          u.x = fmaf(drift, q.x, u.x);
          u.y = fmaf(drift, q.y, u.y);
          q.x = fmaf(-kick, u.x, q.x);
          q.y = fmaf(-kick, u.y, q.y);
        }
        if (L > 0) {
          u.x = fmaf(drift, q.x, u.x);
          u.y = fmaf(drift, q.y, u.y);
          q.x = fmaf(-half, u.x, q.x);
          q.y = fmaf(-half, u.y, q.y);
        }
        lpl += wt * ((double)(u.x * u.x + u.y * u.y) * (double)s);
        kl += wt * ((double)(q.x * q.x + q.y * q.y) / (double)lm);
      }
      if (L > 0) __stcs(Gd + gi, u);  // an evaluation (L = 0) leaves the state as it is
      if constexpr (FIXED) ch.Gq[gi] = q;
    }
  }
  const double sums[4] = {e0, lp0, lpl, kl};
  const int slots[4] = {SL_E0, SL_LP0, SL_LPL, SL_KL};
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const double t = block_sum(sums[k], red);
    if (threadIdx.x == 0) ch.part[((long long)c * NSLOT + slots[k]) * ch.maxblk + ch.nb_x + blockIdx.x] = t;
  }
}

// u = h + i g on all N modes <-> the half spectra.  A mode k of a plane z > E2/2 is conj of -k.
__global__ void k_merge(DevVolume v, const float2* __restrict__ h, const float2* __restrict__ g, float2* __restrict__ u) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= v.N) return;
  const int x = (int)(i % v.E0), y = (int)((i / v.E0) % v.E1), z = (int)(i / ((long long)v.E0 * v.E1));
  long long j = i;
  float sg = 1.0f;
  if (z >= v.EZ) {
    j = ((long long)(v.E2 - z) * v.E1 + (y == 0 ? 0 : v.E1 - y)) * v.E0 + (x == 0 ? 0 : v.E0 - x);
    sg = -1.0f;
  }
  const float2 a = h[j], b = g[j];
  u[i] = make_float2(a.x - sg * b.y, sg * a.y + b.x);
}
__global__ void k_split(DevVolume v, const float2* __restrict__ u, float2* __restrict__ h, float2* __restrict__ g) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= v.NH) return;
  const int x = (int)(i % v.E0), y = (int)((i / v.E0) % v.E1), z = (int)(i / ((long long)v.E0 * v.E1));
  const long long j = ((long long)(z == 0 ? 0 : v.E2 - z) * v.E1 + (y == 0 ? 0 : v.E1 - y)) * v.E0 + (x == 0 ? 0 : v.E0 - x);
  const float2 a = u[i], m = u[j];
  h[i] = make_float2(0.5f * (a.x + m.x), 0.5f * (a.y - m.y));
  g[i] = make_float2(0.5f * (a.y + m.y), 0.5f * (m.x - a.x));
}

// ----------------------------------------------------------------- x-line kernel
// The hot kernel of one leapfrog step, for 32 x-lines of one chain:
//   inverse x-FFT of the data gradient (spectral except along x),
//   kick  q += k eps (IFFT(data grad) - u / lambda)          (MultiResParameters.h:690, 699)
//   drift u* += eps q / lambda_m                              (:693-698)
//   forward x-FFT of u* for the next gradient.
// Step 0 starts from the momentum that k_momentum drew and adds the initial
// energies; the last step only kicks and accumulates the final energies (:702-705).
template <int E0> struct XCfg {
  static constexpr int NT = 256;
  // blocks per SM the register budget targets: at E0 = 256 the 67.6 KB tile allows three (85 registers, no
  // spills; two at the unconstrained 126 registers), at E0 <= 128 four
  static constexpr int MINB = E0 == 256 ? 3 : 4;
};

template <int E0, int PLAN = 0>
__global__ void __launch_bounds__(XCfg<E0>::NT, XCfg<E0>::MINB) k_xline(DevVolume v, DevChains ch, int step, int flags,
                                                        const float2* __restrict__ tw) {
  grid_dep_wait();
  constexpr int TL = TILE_LINES, P = TILE_LINES + 1, NT = XCfg<E0>::NT;
  extern __shared__ __align__(16) unsigned char smraw[];
  float2* sm = reinterpret_cast<float2*>(smraw);
  __shared__ double red[NT / 32];
  const int c = blockIdx.y;
  const ChainState& st = ch.st[c];
  const int Lc = st.L_cur;
  if (step > Lc) return;
  const bool first = step == 0, last = step == Lc;
  const float eps = st.eps_cur, sh = st.sh;
  const int acc = st.acc;
  const long long NH = v.NH;
  const long long lines = (long long)v.E1 * v.EZ;
  const long long lam0 = (long long)blockIdx.x * TL;
  // the block's lines of the state and of T1 lie in their arrays (checked builds)
  if (!in_bounds(min(lam0 + TL, lines) * E0 - 1, NH, ch.err) ||
      !in_bounds(min(lam0 + TL, lines) * v.bx - 1, ch.t1_stride, ch.err))
    return;
  const int nl = (int)min((long long)TL, lines - lam0);
  float2* Ub = ch.U + (long long)c * 2 * NH;
  const float2* Usrc = Ub + (long long)(first ? acc : (acc ^ 1)) * NH;
  float2* Udst = Ub + (long long)(acc ^ 1) * NH;
  float2* Qc = ch.Q + (long long)c * NH;
  float2* T1 = ch.T1 + (long long)c * ch.t1_stride;
  const int bx = v.bx;
  if ((flags & XF_L2_PREFETCH) && threadIdx.x == 0 && E0 >= 4) {
    bulk_prefetch_l2(Usrc + lam0 * E0, (uint32_t)nl * E0 * 8);
    bulk_prefetch_l2(Qc + lam0 * E0, (uint32_t)nl * E0 * 8);
    bulk_prefetch_l2(v.sinv + lam0 * E0, (uint32_t)nl * E0 * 4);
  }

  for (int e = threadIdx.x; e < TL * E0; e += NT) {
    const int l = e / E0, x = e % E0;
    float2 val = make_float2(0.f, 0.f);
    if (l < nl && x < bx) val = T1[(lam0 + l) * bx + x];
    sm[x * P + l] = val;
  }
  __syncthreads();
  fft_smem<E0, +1, TL, NT, float2, PLAN>(sm, 1, P, TL, tw + tw_offset(E0));

  const bool fixed = (flags & XF_FIXED_MOMENTUM) != 0;
  const bool write_q = !last || (flags & XF_WRITE_Q_LAST);
  const float keps = ((first || last) ? 0.5f : 1.0f) * eps;
  double pa = 0.0, pb = 0.0;
  for (int e = threadIdx.x; e < TL * (E0 / 2); e += NT) {
    const int l = e / (E0 / 2), x = 2 * (e % (E0 / 2));
    if (l >= nl) continue;
    const long long gi = (lam0 + l) * E0 + x;
    const float4 u4 = __ldcs(reinterpret_cast<const float4*>(Usrc + gi));
    const float2 s2 = *reinterpret_cast<const float2*>(v.sinv + gi);
    const float4 q4 = __ldcs(reinterpret_cast<const float4*>(Qc + gi));
    const double wt = (first || last) ? plane_weight((int)((lam0 + l) / v.E1), v.E2) : 0.0;
    float2 uo[2], qo[2];
#pragma unroll
    for (int m = 0; m < 2; m++) {
      const float2 u = m == 0 ? make_float2(u4.x, u4.y) : make_float2(u4.z, u4.w);
      const float s = m == 0 ? s2.x : s2.y;
      const bool live = s > 0.0f;
      const float lm = s + sh;  // lambda_m = 1/lambda + sigma_h^-2 (MultiResParameters.h:735-738)
      float2 q = m == 0 ? make_float2(q4.x, q4.y) : make_float2(q4.z, q4.w);
      if (first && live) {  // the kinetic energy of a drawn momentum is k_momentum's sum |w|^2
        if (fixed) pa += wt * ((double)(q.x * q.x + q.y * q.y) / (double)lm);
        pb += wt * ((double)(u.x * u.x + u.y * u.y) * (double)s);
      }
      const float2 g = sm[(x + m) * P + l];
      float2 gt = g;
      if (live) {
        gt.x = fmaf(-u.x, s, g.x);
        gt.y = fmaf(-u.y, s, g.y);
      }
      q.x = fmaf(keps, gt.x, q.x);
      q.y = fmaf(keps, gt.y, q.y);
      float2 un = u;
      if (last) {
        // the final energies; a step that is both first and last only evaluates (a gradient / log posterior
        // call) and keeps the energies at mu
        if (live && !first) {
          pa += wt * ((double)(u.x * u.x + u.y * u.y) * (double)s);
          pb += wt * ((double)(q.x * q.x + q.y * q.y) / (double)lm);
        }
      } else if (live) {
        const float f = eps / lm;
        un.x = fmaf(f, q.x, u.x);
        un.y = fmaf(f, q.y, u.y);
      }
      uo[m] = un;
      qo[m] = q;
      sm[(x + m) * P + l] = un;
    }
    // streaming loads and stores of the state, as in the plane kernel: it is not read again before the next step
    if (write_q) __stcs(reinterpret_cast<float4*>(Qc + gi), make_float4(qo[0].x, qo[0].y, qo[1].x, qo[1].y));
    if (!last) __stcs(reinterpret_cast<float4*>(Udst + gi), make_float4(uo[0].x, uo[0].y, uo[1].x, uo[1].y));
  }
  // per-block partial sums -> accept step
  if (first || last) {
    const double ta = block_sum(pa, red);
    if (threadIdx.x == 0) ch.part[((long long)c * NSLOT + (first ? SL_E0 : SL_LPL)) * ch.maxblk + blockIdx.x] = ta;
    const double tb = block_sum(pb, red);
    if (threadIdx.x == 0) ch.part[((long long)c * NSLOT + (first ? SL_LP0 : SL_KL)) * ch.maxblk + blockIdx.x] = tb;
  }
  if (last) return;
  __syncthreads();
  fft_smem<E0, -1, TL, NT, float2, PLAN>(sm, 1, P, TL, tw + tw_offset(E0));
  const uint32_t mb = box_div_magic(bx);
  for (int e = threadIdx.x; e < TL * bx; e += NT) {
    const int l = (int)__umulhi((uint32_t)e, mb), x = e - l * bx;
    if (l < nl) T1[(lam0 + l) * bx + x] = sm[x * P + l];
  }
}

// ----------------------------------------------------------------- square plane kernel
// The leapfrog update fused with the y and x transforms of one z-plane of one
// chain (E0 == E1 == E), one block per (z-plane, chain):
//   T2[c][z][y < by][x < bx] --inverse y (columns x < bx), inverse x (rows)-->
//   spectral plane; kick / drift as in k_xline; forward x, forward y --> T2.
// For E = 64 the plane uses the padded layout of PaddedPlane (bank-conflict free
// radix stages); smaller planes an odd row pitch.  Square planes up to 64 only: the
// whole plane is in shared memory, four blocks to an SM at E = 64.
template <int E>
struct PlaneGeom {
  static constexpr bool PADDED = E == 64;
  static constexpr int R1 = 8, R2 = 8;
  static constexpr int P = E + 1;  // odd pitch of the unpadded layout
  static constexpr int SIZE = PADDED ? PaddedPlane<E>::SIZE : E * (E + 1);
  __device__ __forceinline__ static int at(int y, int x) {
    if constexpr (PADDED) return PaddedPlane<E>::phys(y, x);
    else return y * P + x;
  }
};

// 256 threads, four blocks per SM at 64 registers for E = 64 (64 chains on a 64^3 embedding: 68.3 us, 72.4 with three
// blocks at 80 registers, 79.9 with two blocks of 512 threads).
// WIDE: 512 threads with all the registers, for chain sets of at most a plane per SM (one chain on 64^3: 7.5 us, 9.0 with
// the narrow blocks).
template <bool WIDE> struct SquareCfg {
  static constexpr int NT = WIDE ? 512 : 256, MINB = WIDE ? 1 : 4;
};

// The padded planes prune both transforms to the box (ncols x nrows of T2): the inverse transforms read only the
// box (everything else is zero and is never stored), and the forward transforms write only what lands in it.
template <int E>
__device__ __forceinline__ void plane_fft(float2* sm, int ncols, int nrows, int dir, const float2* tw) {
  using G = PlaneGeom<E>;
  if constexpr (G::PADDED) {
    if (dir > 0) {
      plane_cols_padded<E, G::R1, G::R2, +1>(sm, ncols, tw, nrows, E);
      plane_rows_padded<E, G::R1, G::R2, +1>(sm, tw, ncols, E);
    } else {
      plane_rows_padded<E, G::R1, G::R2, -1>(sm, tw, E, ncols);
      plane_cols_padded<E, G::R1, G::R2, -1>(sm, ncols, tw, E, nrows);
    }
  } else {
    if (dir > 0) {
      fft_smem_warp<E, +1>(sm, 1, G::P, ncols, tw);
      fft_smem_warp<E, +1>(sm, G::P, 1, E, tw);
    } else {
      fft_smem_warp<E, -1>(sm, G::P, 1, E, tw);
      fft_smem_warp<E, -1>(sm, 1, G::P, ncols, tw);
    }
  }
}

// One plane of one chain after its inverse transforms, in two parts.  plane_update: the kick and the drift; the
// energies' per-thread partials go to pa / pb.  The state is read and written with streaming accesses (ld / st.global.cs):
// a plane's state is not read again before the next leapfrog step, by which time it has left L2 anyway, and evicting it
// first keeps T2 and the smaller arrays of the following kernels in L2.  plane_finish: the energies' block partials, then
// the forward transforms and the T2 store.
template <int E, int NT>
__device__ __forceinline__ void plane_update(float2* sm, const DevVolume& v, const ChainState& st, int z, bool first, bool last, int flags,
                                             const float2* srcU, const float2* srcQ, const float* srcS,
                                             float2* Udst, float2* Qc, double& pa_out, double& pb_out) {
  using G = PlaneGeom<E>;
  const int tid = threadIdx.x;
  const float eps = st.eps_cur, sh = st.sh;
  const bool write_q = !last || (flags & XF_WRITE_Q_LAST);
  const float keps = ((first || last) ? 0.5f : 1.0f) * eps;
  const bool fixed = (flags & XF_FIXED_MOMENTUM) != 0;
  double pa = 0.0, pb = 0.0;
  // Pairs of x-adjacent points: element pair e sits at li = 2e of the plane (x = 2 (e mod E/2), y = e / (E/2)),
  // so U, q and 1/lambda are read as float4 / float4 / float2 at index e: one pair at a time, the block's state being
  // prefetched into L2 at entry.  A thread reads and writes only its own elements, which is why the in-place state
  // buffers may be marked non-aliasing.
  constexpr int TOTAL = E * (E / 2);
  const float4* __restrict__ gU = reinterpret_cast<const float4*>(srcU);
  const float4* __restrict__ gQ = reinterpret_cast<const float4*>(srcQ);
  const float2* __restrict__ gS = reinterpret_cast<const float2*>(srcS);
  float4* __restrict__ oQ = reinterpret_cast<float4*>(Qc);
  float4* __restrict__ oU = reinterpret_cast<float4*>(Udst);
  for (int e = tid; e < TOTAL; e += NT) {
    const float4 u4 = __ldcs(gU + e);
    const float4 q4 = __ldcs(gQ + e);
    const float2 s2 = gS[e];
    const int y = e / (E / 2), x = 2 * (e % (E / 2));
    const int pi0 = G::at(y, x), pi1 = pi0 + 1;  // x is even: x + 1 is the next slot in either layout
    float2 uo[2], qo[2];
#pragma unroll
    for (int m = 0; m < 2; m++) {
      const float2 u = m == 0 ? make_float2(u4.x, u4.y) : make_float2(u4.z, u4.w);
      const float s = m == 0 ? s2.x : s2.y;
      const bool live = s > 0.0f;
      const float lm = s + sh;
      float2 q = m == 0 ? make_float2(q4.x, q4.y) : make_float2(q4.z, q4.w);
      if (first && live) {  // the kinetic energy of a drawn momentum is k_momentum's sum |w|^2
        if (fixed) pa += (double)(q.x * q.x + q.y * q.y) / (double)lm;
        pb += (double)(u.x * u.x + u.y * u.y) * (double)s;
      }
      const int pi = m == 0 ? pi0 : pi1;
      const float2 g = sm[pi];
      float2 gt = g;
      if (live) {
        gt.x = fmaf(-u.x, s, g.x);
        gt.y = fmaf(-u.y, s, g.y);
      }
      q.x = fmaf(keps, gt.x, q.x);
      q.y = fmaf(keps, gt.y, q.y);
      float2 un = u;
      if (last) {
        if (live && !first) {  // first and last: an evaluation step, energies at mu only
          pa += (double)(u.x * u.x + u.y * u.y) * (double)s;
          pb += (double)(q.x * q.x + q.y * q.y) / (double)lm;
        }
      } else if (live) {
        const float f = eps / lm;
        un.x = fmaf(f, q.x, u.x);
        un.y = fmaf(f, q.y, u.y);
      }
      uo[m] = un;
      qo[m] = q;
      sm[pi] = un;
    }
    if (write_q) __stcs(oQ + e, make_float4(qo[0].x, qo[0].y, qo[1].x, qo[1].y));
    if (!last) __stcs(oU + e, make_float4(uo[0].x, uo[0].y, uo[1].x, uo[1].y));
  }
  const double wt = plane_weight(z, v.E2);
  pa_out = wt * pa;
  pb_out = wt * pb;
}

template <int E, int NT>
__device__ __forceinline__ void plane_finish(float2* sm, const DevChains& ch, int c, int z, bool first, bool last,
                                             double pa, double pb, float2* T, int bx, int by, const float2* twE,
                                             double* red) {
  using G = PlaneGeom<E>;
  const int tid = threadIdx.x;
  if (first || last) {
    const double ta = block_sum(pa, red);
    if (tid == 0) ch.part[((long long)c * NSLOT + (first ? SL_E0 : SL_LPL)) * ch.maxblk + z] = ta;
    const double tb = block_sum(pb, red);
    if (tid == 0) ch.part[((long long)c * NSLOT + (first ? SL_LP0 : SL_KL)) * ch.maxblk + z] = tb;
  }
  if (last) return;
  __syncthreads();
  plane_fft<E>(sm, bx, by, -1, twE);
  const uint32_t mb = box_div_magic(bx);
  for (int e = tid; e < by * bx; e += NT) {
    const int y = (int)__umulhi((uint32_t)e, mb), x = e - y * bx;
    T[y * bx + x] = sm[G::at(y, x)];
  }
}

// Loads the T2 box of one plane into the plane buffer (for the padded layout only the box: the pruned inverse
// transforms read nothing outside it).
template <int E, int NT>
__device__ __forceinline__ void plane_load_box(float2* sm, const float2* __restrict__ T, int bx, int by) {
  using G = PlaneGeom<E>;
  const int tid = threadIdx.x;
  if constexpr (G::PADDED) {
    const uint32_t mb = box_div_magic(bx);
    for (int e = tid; e < by * bx; e += NT) {
      const int y = (int)__umulhi((uint32_t)e, mb), x = e - y * bx;
      sm[G::at(y, x)] = __ldcs(T + e);  // the last read of this T2 plane before the next inverse z pass
    }
  } else {
    for (int e = tid; e < E * E; e += NT) {
      const int y = e / E, x = e % E;
      sm[G::at(y, x)] = (y < by && x < bx) ? T[y * bx + x] : make_float2(0.f, 0.f);
    }
  }
}

template <int E, bool WIDE>
__global__ void __launch_bounds__(SquareCfg<WIDE>::NT, SquareCfg<WIDE>::MINB) k_plane_square(DevVolume v, DevChains ch, int step, int flags,
                                                              const float2* __restrict__ tw) {
  grid_dep_wait();
  constexpr int NT = SquareCfg<WIDE>::NT;
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ double red[NT / 32];
  float2* sm = reinterpret_cast<float2*>(smraw);
  const int c = blockIdx.y, z = blockIdx.x;
  const ChainState& st = ch.st[c];
  const int Lc = st.L_cur;
  if (step > Lc) return;
  // the block's plane of the state and of T2 lie in their arrays (checked builds)
  if (!in_bounds((long long)(z + 1) * E * E - 1, v.NH, ch.err) ||
      !in_bounds((long long)(z + 1) * v.by * v.bx - 1, ch.t2_stride, ch.err))
    return;
  const bool first = step == 0, last = step == Lc;
  const int acc = st.acc;
  const long long NH = v.NH;
  const int bx = v.bx, by = v.by;
  const int tid = threadIdx.x;
  float2* Ub = ch.U + (long long)c * 2 * NH;
  const float2* Usrc = Ub + (long long)(first ? acc : (acc ^ 1)) * NH + (long long)z * E * E;
  float2* Udst = Ub + (long long)(acc ^ 1) * NH + (long long)z * E * E;
  float2* Qc = ch.Q + (long long)c * NH + (long long)z * E * E;
  const float* Sg = v.sinv + (long long)z * E * E;
  float2* T = ch.T2 + (long long)c * ch.t2_stride + (long long)z * by * bx;
  // the twiddles of length E in shared memory: the row and column stages load a lane's twiddles again for every
  // line, and as global loads (L1 hits) they were most of the kernel's load instructions (4 % of its time on the full
  // spectrum)
  __shared__ float2 twE[E];
  for (int i = tid; i < E; i += NT) twE[i] = tw[tw_offset(E) + i];
  if ((flags & XF_L2_PREFETCH) && tid == 0) {
    bulk_prefetch_l2(Usrc, E * E * 8);
    bulk_prefetch_l2(Qc, E * E * 8);
    bulk_prefetch_l2(Sg, E * E * 4);
  }
  plane_load_box<E, NT>(sm, T, bx, by);
  __syncthreads();
  plane_fft<E>(sm, bx, by, +1, twE);
  double pa, pb;
  plane_update<E, NT>(sm, v, st, z, first, last, flags, Usrc, Qc, Sg, Udst, Qc, pa, pb);
  plane_finish<E, NT>(sm, ch, c, z, first, last, pa, pb, T, bx, by, twE, red);
}

// ----------------------------------------------------------------- xy-plane kernel
// The leapfrog update fused with the y and x transforms of one z-plane of one
// chain (E0, E1 <= 128), one block per (z-plane, chain):
//   T2[c][z][y < by][x < bx] --inverse y (columns x < bx)--> T[y < E1][x < bx];
//   per row y: inverse x, kick / drift as in k_xline, forward x --> T[y][x < bx];
//   --forward y (y < by)--> T2.
// Only the box's columns of the plane are ever held (E1 x bx); a row's E0 points
// are in registers between its transforms (row_inverse, row_forward), and a warp
// takes its rows through all three steps without a block barrier, so that one
// warp's state is on its way while another transforms (L2 is asked for all of the
// block's state at entry).  Used for planes with an axis of 128, where a whole plane
// would leave room for one block on an SM, and for planes that are not square,
// which otherwise go through separate y passes; the tuner tries it on the others.
// Measured: 16 chains on 128^3 177 us (whole plane in shared memory, 512
// threads: 246; x-line kernel with its y passes 190 + 61); 12 chains on 128x64x32 18.7 us
// (x-line 17.5 + 8.2); 64 chains on 64^3 87 us (k_plane_square 68). It is bound
// by latency: its registers leave 16 warps to an SM, which wait on the state (L1 pipe
// 48 %, DRAM 39 %, 3.2 TB/s).  Loading a row's whole state before its inverse transform was slower
// (128^3: 222 us: it spills at 128 registers).
// WIDE: 512 threads with all the registers, for chain sets of at most a plane per SM (4 chains on 128x128x64: 21.4 us,
// 27.9 with the narrow blocks).
template <int E0, int E1, bool WIDE>
struct PlaneCfg {
  static constexpr int NT = WIDE ? 512 : 256;
  static constexpr int MINB = WIDE ? 1 : ((E0 > 64 || E1 > 64) ? 2 : 3);  // blocks per SM the register budget targets
  static constexpr int ROW_ELEMS = (NT / 32) * RowPlan<E0>::ROWS * RowPlan<E0>::RP;
};
// Shared memory of a block (complex elements): the T array, then the warps' row buffers.
template <int E0, int E1>
__host__ __device__ constexpr int plane_box_elems(int bx) { return (E1 * row_pitch<E0>(bx) + 1) / 2 * 2; }

template <int E0, int E1, bool WIDE>
__global__ void __launch_bounds__(PlaneCfg<E0, E1, WIDE>::NT, PlaneCfg<E0, E1, WIDE>::MINB)
    k_xyplane(DevVolume v, DevChains ch, int step, int flags, const float2* __restrict__ tw) {
  grid_dep_wait();
  using Cfg = PlaneCfg<E0, E1, WIDE>;
  using PX = RowPlan<E0>;
  constexpr int NT = Cfg::NT, RP = PX::RP, RA = PX::RA, RB = PX::RB, ROWS = PX::ROWS;
  constexpr int PAIRS = RA / 2, UB = PAIRS <= 4 || WIDE ? 4 : 2;  // pairs of the state asked for together
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ double red[NT / 32];
  // the twiddles in shared memory: the stages load a lane's twiddles again for every line, and as global loads (L1
  // hits) they were most of the kernel's load instructions
  __shared__ float2 tw0[E0], tw1[E1];
  const int c = blockIdx.y, z = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const ChainState& st = ch.st[c];
  const int Lc = st.L_cur;
  if (step > Lc) return;
  constexpr int PLANE = E0 * E1;
  const int bx = v.bx, by = v.by;
  // the block's plane of the state and of T2 lie in their arrays (checked builds)
  if (!in_bounds((long long)(z + 1) * PLANE - 1, v.NH, ch.err) || !in_bounds((long long)(z + 1) * by * bx - 1, ch.t2_stride, ch.err))
    return;
  const bool first = step == 0, last = step == Lc, fixed = (flags & XF_FIXED_MOMENTUM) != 0;
  const bool write_q = !last || (flags & XF_WRITE_Q_LAST);
  const float eps = st.eps_cur, sh = st.sh, keps = ((first || last) ? 0.5f : 1.0f) * eps;
  const int acc = st.acc;
  const long long NH = v.NH, at_z = (long long)z * PLANE;
  const float2* Usrc = ch.U + ((long long)c * 2 + (first ? acc : (acc ^ 1))) * NH + at_z;
  float2* Udst = ch.U + ((long long)c * 2 + (acc ^ 1)) * NH + at_z;
  float2* Qc = ch.Q + (long long)c * NH + at_z;
  const float* Sg = v.sinv + at_z;
  float2* T = ch.T2 + (long long)c * ch.t2_stride + (long long)z * by * bx;
  if ((flags & XF_L2_PREFETCH) && tid == 0) {
    bulk_prefetch_l2(Usrc, PLANE * 8);
    bulk_prefetch_l2(Qc, PLANE * 8);
    bulk_prefetch_l2(Sg, PLANE * 4);
  }
  for (int i = tid; i < E0; i += NT) tw0[i] = tw[tw_offset(E0) + i];
  for (int i = tid; i < E1; i += NT) tw1[i] = tw[tw_offset(E1) + i];
  const int pitch = row_pitch<E0>(bx);
  float2* box = reinterpret_cast<float2*>(smraw);
  // the box in pairs of x-adjacent points (bx is even); the last read of this T2 plane before the next inverse z pass
  const int hx = bx / 2;
  const uint32_t mb = box_div_magic(hx);
  for (int e = tid; e < by * hx; e += NT) {
    const int y = hx == 1 ? e : (int)__umulhi((uint32_t)e, mb), x = 2 * (e - y * hx);
    const float4 t = __ldcs(reinterpret_cast<const float4*>(T) + e);
    float2* d = box + y * pitch + x;
    d[0] = make_float2(t.x, t.y);
    d[1] = make_float2(t.z, t.w);
  }
  __syncthreads();
  plane_cols<E1, +1>(box, pitch, bx, tw1, by, E1);
  __syncthreads();

  const int r = lane / PX::LN, b = lane % PX::LN;
  float2* row = box + plane_box_elems<E0, E1>(bx) + (warp * ROWS + r) * RP;
  double pa = 0.0, pb = 0.0;
#pragma unroll 1
  for (int y0 = warp * ROWS; y0 < E1; y0 += (NT / 32) * ROWS) {  // E1 is a multiple of ROWS
    const int y = y0 + r;
    // the lane's pairs of points, UB at a time: pair i = (mm, k) is points p(2 mm) + RA k and the next
    auto pair_at = [&](int i) { return (y * E0 + PX::butterfly(b, 2 * (i / RB)) + RA * (i % RB)) / 2; };
    float4 u4v[UB], q4v[UB];
    float2 s2v[UB];
    float2 e[PX::NBF][RB];
    row_inverse<E0>(box + y * pitch, bx, row, b, tw0, e);
#pragma unroll
    for (int i0 = 0; i0 < PAIRS; i0 += UB) {
#pragma unroll
      for (int i = 0; i < UB; i++) {
        const int at = pair_at(i0 + i);
        u4v[i] = __ldcs(reinterpret_cast<const float4*>(Usrc) + at);
        q4v[i] = __ldcs(reinterpret_cast<const float4*>(Qc) + at);
        s2v[i] = __ldg(reinterpret_cast<const float2*>(Sg) + at);
      }
#pragma unroll
      for (int i = 0; i < UB; i++) {
        const int at = pair_at(i0 + i), mm = (i0 + i) / RB, k = (i0 + i) % RB;
        float2 uo[2], qo[2];
#pragma unroll
        for (int m = 0; m < 2; m++) {
          const float2 u = m == 0 ? make_float2(u4v[i].x, u4v[i].y) : make_float2(u4v[i].z, u4v[i].w);
          const float s = m == 0 ? s2v[i].x : s2v[i].y;
          const bool live = s > 0.0f;
          const float lm = s + sh;  // lambda_m = 1/lambda + sigma_h^-2 (MultiResParameters.h:735-738)
          float2 q = m == 0 ? make_float2(q4v[i].x, q4v[i].y) : make_float2(q4v[i].z, q4v[i].w);
          if (first && live) {  // the kinetic energy of a drawn momentum is k_momentum's sum |w|^2
            if (fixed) pa += (double)(q.x * q.x + q.y * q.y) / (double)lm;
            pb += (double)(u.x * u.x + u.y * u.y) * (double)s;
          }
          const float2 g = e[2 * mm + m][k];
          float2 gt = g;
          if (live) {
            gt.x = fmaf(-u.x, s, g.x);
            gt.y = fmaf(-u.y, s, g.y);
          }
          q.x = fmaf(keps, gt.x, q.x);
          q.y = fmaf(keps, gt.y, q.y);
          float2 un = u;
          if (last) {
            if (live && !first) {  // first and last: an evaluation step, energies at mu only
              pa += (double)(u.x * u.x + u.y * u.y) * (double)s;
              pb += (double)(q.x * q.x + q.y * q.y) / (double)lm;
            }
          } else if (live) {
            const float f = eps / lm;
            un.x = fmaf(f, q.x, u.x);
            un.y = fmaf(f, q.y, u.y);
          }
          uo[m] = un;
          qo[m] = q;
          e[2 * mm + m][k] = un;
        }
        // streaming loads and stores of the state: it is not read again before the next leapfrog step, by which time
        // it has left L2 on large chain sets; evicting it first keeps T2 and the following kernels' arrays there
        if (write_q) __stcs(reinterpret_cast<float4*>(Qc) + at, make_float4(qo[0].x, qo[0].y, qo[1].x, qo[1].y));
        if (!last) __stcs(reinterpret_cast<float4*>(Udst) + at, make_float4(uo[0].x, uo[0].y, uo[1].x, uo[1].y));
      }
    }
    if (!last) row_forward<E0>(e, row, b, tw0, box + y * pitch, bx);
  }
  if (first || last) {
    const double wt = plane_weight(z, v.E2);
    const double ta = block_sum(wt * pa, red);
    if (tid == 0) ch.part[((long long)c * NSLOT + (first ? SL_E0 : SL_LPL)) * ch.maxblk + z] = ta;
    const double tb = block_sum(wt * pb, red);
    if (tid == 0) ch.part[((long long)c * NSLOT + (first ? SL_LP0 : SL_KL)) * ch.maxblk + z] = tb;
  }
  if (last) return;
  __syncthreads();
  plane_cols<E1, -1>(box, pitch, bx, tw1, E1, by);
  __syncthreads();
  for (int e = tid; e < by * hx; e += NT) {
    const int y = hx == 1 ? e : (int)__umulhi((uint32_t)e, mb), x = 2 * (e - y * hx);
    const float2* d = box + y * pitch + x;
    reinterpret_cast<float4*>(T)[e] = make_float4(d[0].x, d[0].y, d[1].x, d[1].y);
  }
}

// ----------------------------------------------------------------- per-iteration scalars
// Metropolis accept (MultiResParameters.h:702-726), Gibbs sigma draws
// (:821-838) and HMCParameters::update (HMCParameters.h:259-297).  The
// Hamiltonian difference is formed in FP64.  One block per chain: each warp sums
// one of the eight partial-sum slots, and two threads draw the two sigmas side by
// side (12.6 us for one chain with block-wide sums in turn and the draws one after the other).
__global__ void __launch_bounds__(256) k_accept(DevVolume v, DevChains ch) {
  __shared__ double sums[8];
  __shared__ float s_ss;
  __shared__ int s_err;
  const int c = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  ChainState& st = ch.st[c];
  if (st.L_cur < 0) return;
  {
    const bool residual_s = warp == SL_RS0 || warp == SL_RSL, residual_h = warp == SL_RH0 || warp == SL_RHL;
    const int nb = residual_s ? (v.n_s > 0 ? ch.nb_w : 0) : (residual_h ? ch.nb_wt : ch.nb_x + ch.nb_g);
    const double* p = ch.part + ((long long)c * NSLOT + warp) * ch.maxblk;
    double t = 0.0;
#pragma unroll 4
    for (int i = lane; i < nb; i += 32) t += p[i];
    t = warp_sum(t);
    if (lane == 0) sums[warp] = t;
  }
  __syncthreads();
  const double N = (double)v.N;
  const double sh = st.sh, ss = st.ss;
  const double lp0 = -0.5 * sums[SL_LP0] / N;
  const double ll0 = -0.5 * (sh * sums[SL_RH0] + (v.n_s > 0 ? ss * sums[SL_RS0] : 0.0));
  const double E0 = -0.5 * sums[SL_E0] + lp0 + ll0;
  const double lpL = -0.5 * sums[SL_LPL] / N;
  const double llL = -0.5 * (sh * sums[SL_RHL] + (v.n_s > 0 ? ss * sums[SL_RSL] : 0.0));
  const double KL = -0.5 * sums[SL_KL] / N;
  const double logR = (lpL + llL + KL) - E0;
  double R = exp(logR);
  if (isnan(R)) R = 0.0;
  const u32x4 r = philox(u32x4{0u, (uint32_t)st.iteration, (uint32_t)(ch.chain0 + c), RNG_SCALAR}, ch.seed);
  const double u = u01d(r.z, r.w);
  const bool moved = u < R;
  const double Rh = moved ? sums[SL_RHL] : sums[SL_RH0], Rs = moved ? sums[SL_RSL] : sums[SL_RS0];
  // Gibbs: shape n/2 + 1, rate ||residual||^2 / 2 (float arithmetic as in the reference); the first warp draws
  // sigma_h, the second sigma_s
  int err = 0;
  const int n = warp == 0 ? v.n_h : v.n_s;
  float draw = (float)ss;
  if (lane == 0 && (warp == 0 || (warp == 1 && n > 0))) {
    const float shape = 0.5f * (float)n + 1.0f, rate = 0.5f * (float)(warp == 0 ? Rh : Rs);
    draw = (float)gamma_draw(shape, 1.0 / (double)rate, ch.seed, RNG_SCALAR, ch.chain0 + c, st.iteration,
                             warp == 0 ? 16u : 4096u, &err);
  }
  if (lane == 0 && warp == 1) {
    s_ss = draw;
    s_err = err;
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  ch.moved[c] = moved;
  if (moved) {
    st.acc ^= 1;
    st.accepted += 1;
  }
  st.Rh_acc = Rh;
  st.Rs_acc = Rs;
  st.err += err + s_err;
  st.sh = draw;
  st.ss = s_ss;
  st.grad_evals += st.L_cur + 1;
  st.last_log_ratio = logR;
  st.last_E0 = E0;
  st.last_Ep = lpL + llL + KL;
  hmc_update(st, (float)fmin(1.0, R));
  st.save_now = 0;
  if (hmc_save_iteration(st)) {
    st.save_now = 1;
    st.saved += 1;
    const double ll = -0.5 * ((double)st.sh * Rh + (v.n_s > 0 ? (double)st.ss * Rs : 0.0));
    st.ll_sum += ll;
    st.sigh_sum += sqrt(1.0 / (double)st.sh);
    st.sigs_sum += v.n_s > 0 ? sqrt(1.0 / (double)st.ss) : 0.0;
    if (ch.save_rec != nullptr && st.saved <= st.n_save) {
      // MultiResParameters::sigma (MultiResParameters.h:613-619) is sqrt(1 / sigma^-2) in float
      double* r = ch.save_rec + ((long long)(st.saved - 1) * ch.C + c) * 3;
      r[0] = (double)sqrtf(1.0f / st.sh);
      r[1] = v.n_s > 0 ? (double)sqrtf(1.0f / st.ss) : 0.0;
      r[2] = ll;
    }
    if (st.saved >= st.n_save) st.done = 1;
  }
}

// mcmc_summary::update (gaussian_process_model.h:209-229): max |mu| per chain, then moments.  The accepted state's
// mu is still in the proposal half of an accepted move (ch.moved) here; k_summary_acc brings it over.
__global__ void __launch_bounds__(256) k_summary_max(DevVolume v, DevChains ch) {
  __shared__ float red[8];
  const int c = blockIdx.x;
  ChainState& st = ch.st[c];
  if (!st.save_now || st.L_cur < 0) return;
  const float* mo = ch.muO + (long long)ch.moved[c] * v.n_o * ch.Cp + c;
  float m = 0.f;
  for (int o = threadIdx.x; o < v.n_o; o += blockDim.x) m = fmaxf(m, fabsf(mo[(long long)o * ch.Cp]));
  for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < (int)(blockDim.x >> 5); i++) m = fmaxf(m, red[i]);
    m = fmaxf(m, red[0]);
    st.maxabs = m;
  }
}

// The end of an iteration over the elements of mu_D and mu_O: an accepted proposal's mu (half 1) becomes the accepted
// half 0 -- so that a product kernel finds every chain's vector in one half, contiguous over chains -- and on save
// iterations the summary sums take the accepted mu_O.  The copy costs one pass over mu_D per iteration; the halves by
// chain cost every step more (64 chains on a 64^3 embedding: forward z pass 10.6 -> 9.0 us, W 25.8 -> 23.7 us with one
// TMA gather per chunk instead of thread loads from both halves, an iteration 4.08 -> 3.93 ms).
__global__ void k_summary_acc(DevVolume v, DevChains ch) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int c = (int)(e % ch.Cp);
  if (c >= ch.C) return;
  const ChainState& st = ch.st[c];
  if (st.L_cur < 0) return;
  const bool moved = ch.moved[c] != 0;
  const long long nd = (long long)v.n_h * ch.Cp, total = (long long)v.n_o * ch.Cp;
  if (moved && e < nd) ch.muD[e] = ch.muD[nd + e];
  if (e >= total) return;
  if (!moved && !st.save_now) return;
  const float val = ch.muO[moved ? total + e : e];
  if (moved) ch.muO[e] = val;
  if (!st.save_now) return;
  ch.s1[e] += val;
  ch.s2[e] += (double)val * val;
  ch.sa[e] += fabs((double)val) / fmax((double)st.maxabs, 1e-6);
  if (ch.samples != nullptr) ch.samples[(long long)(st.saved - 1) * total + e] = val;
}

// Checkpoints written before mu_D / mu_O kept the accepted state in half 0 (it was in half acc): half 1 -> half 0 of
// the chains whose acc is 1.
__global__ void k_adopt_halves(DevVolume v, DevChains ch) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int c = (int)(e % ch.Cp);
  if (c >= ch.C || ch.st[c].acc == 0) return;
  const long long nd = (long long)v.n_h * ch.Cp, no = (long long)v.n_o * ch.Cp;
  if (e < nd) ch.muD[e] = ch.muD[nd + e];
  if (e < no) ch.muO[e] = ch.muO[no + e];
}

// ----------------------------------------------------------------- initialisation
// _initialize_sigma (MultiResParameters.h:764-778): sigma_h^-2 ~ Gamma(v, 1),
// sigma_s^-2 = sigma_h^-2 / U(0, 1).
__global__ void k_init_sigma(DevChains ch, float shape, int n_datasets) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ch.C) return;
  ChainState& st = ch.st[c];
  st.sh = (float)gamma_draw((double)shape, 1.0, ch.seed, RNG_INIT_SIGMA, ch.chain0 + c, 0u, 16u, &st.err);
  const u32x4 r = philox(u32x4{0u, 0u, (uint32_t)(ch.chain0 + c), RNG_INIT_SIGMA}, ch.seed);
  st.ss = n_datasets == 2 ? st.sh / u01f(r.x) : 1.0f;
}

// gD <- Yh for all chains (the data part of the initial state, add_data_to_mu).
__global__ void k_fill_gD(DevVolume v, DevChains ch) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (long long)v.n_h * ch.Cp) return;
  ch.gD[e] = v.Yh[e / ch.Cp];
}

// _initialize_mu (MultiResParameters.h:744-759) in the spectral basis:
// u0 += sqrt(N lambda) w / 10 on live modes, w ~ CN(0, 2) over all N modes, split into h and g as in k_momentum.
__global__ void k_init_prior(DevVolume v, DevChains ch) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int c = blockIdx.y;
  if (i >= v.NH) return;
  const int x = (int)(i % v.E0), y = (int)((i / v.E0) % v.E1), z = (int)(i / ((long long)v.E0 * v.E1));
  const long long j = ((long long)(z == 0 ? 0 : v.E2 - z) * v.E1 + (y == 0 ? 0 : v.E1 - y)) * v.E0 + (x == 0 ? 0 : v.E0 - x);
  const long long half = ((long long)c * 2 + ch.st[c].acc) * v.NH;
  auto draw = [&](long long k) {
    const u32x4 r = philox(u32x4{(uint32_t)(k >> 1), 0u, (uint32_t)(ch.chain0 + c), RNG_INIT_MU}, ch.seed);
    return (k & 1) ? box_muller(u01f(r.z), u01f(r.w)) : box_muller(u01f(r.x), u01f(r.y));
  };
  const float s = v.sinv[i];
  float2 g = make_float2(0.f, 0.f);
  if (s > 0.0f) {
    const float a = 0.5f * (sqrtf((float)v.N / s) * 0.1f);
    const float2 w = draw(i), m = draw(j);
    float2& h = ch.U[half + i];
    h.x += a * (w.x + m.x);
    h.y += a * (w.y - m.y);
    g = make_float2(a * (w.y + m.y), a * (m.x - w.x));
  }
  ch.G[half + i] = g;
}

// ----------------------------------------------------------------- spectrum (FP64, one-time)
// circulant_base_3d (circulant_base.inl:30-89): wrapped offsets, float norm of
// Q (o, 0), covariance evaluated in FP64.
__global__ void k_base(double2* base, int E0, int E1, int E2, float q00, float q01, float q02, float q10, float q11,
                       float q12, float q20, float q21, float q22, double th0, double th1, double th2, int covfun) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long N = (long long)E0 * E1 * E2;
  if (i >= N) return;
  const int l = (int)(i % E0), m = (int)((i / E0) % E1), n = (int)(i / ((long long)E0 * E1));
  const float o0 = (float)(l <= E0 / 2 ? l : E0 - l), o1 = (float)(m <= E1 / 2 ? m : E1 - m),
              o2 = (float)(n <= E2 / 2 ? n : E2 - n);
  // float arithmetic in source order with every product and sum rounded (no fused multiply-add), so the
  // distances equal a plain float evaluation of the same expression on the host
  const float a = __fadd_rn(__fadd_rn(__fmul_rn(q00, o0), __fmul_rn(q01, o1)), __fmul_rn(q02, o2));
  const float b = __fadd_rn(__fadd_rn(__fmul_rn(q10, o0), __fmul_rn(q11, o1)), __fmul_rn(q12, o2));
  const float cc = __fadd_rn(__fadd_rn(__fmul_rn(q20, o0), __fmul_rn(q21, o1)), __fmul_rn(q22, o2));
  const double d = (double)__fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(a, a), __fmul_rn(b, b)), __fmul_rn(cc, cc)));
  double val;
  if (covfun == 0)
    val = th0 * exp(-th1 * pow(fabs(d), th2));
  else
    val = th0 * pow(1.0 + th1 / th2 * d * d, -th2);
  base[i] = make_double2(val, 0.0);
}

// S = {Re lambda <= 0} (MultiResParameters.h:258-262); sinv = 1/Re lambda on live modes.  The base is even in every
// axis, so lambda(k) and lambda(-k) are the same number; the transform leaves them a rounding apart.  S and sinv are
// formed from their mean, which both get bit for bit: a Hermitian field stays Hermitian under the sampler's element-wise
// steps, and n_S counts the modes that are masked.  (lam_re reports the transform's own values.)
__global__ void k_spectrum(const double2* lam, float* sinv, double* lam_re, int E0, int E1, int E2, int* n_S) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long long)E0 * E1 * E2) return;
  const int x = (int)(i % E0), y = (int)((i / E0) % E1), z = (int)(i / ((long long)E0 * E1));
  const long long j = ((long long)(z == 0 ? 0 : E2 - z) * E1 + (y == 0 ? 0 : E1 - y)) * E0 + (x == 0 ? 0 : E0 - x);
  const double re = lam[i].x, sym = 0.5 * (re + lam[j].x);
  lam_re[i] = re;
  if (sym <= 0.0) atomicAdd(n_S, 1);
  sinv[i] = sym > 0.0 ? (float)(1.0 / sym) : -1.0f;
}

// ----------------------------------------------------------------- evaluation helpers
// Re field[idx[j]] for j < n; N bounds the indices (checked builds, failures to err).
__global__ void k_gather_re(const float2* field, const int* idx, int n, float* out, int pitch, int col, long long N,
                            int* err) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < n && in_bounds(idx[j], N, err)) out[(long long)j * pitch + col] = field[idx[j]].x;
}

// Block partials of sum_live |u|^2 * sinv  (mode 0) or sum_live |u|^2 / (sinv + sh)  (mode 1).
__global__ void __launch_bounds__(256) k_spectral_energy(const float2* u, const float* sinv, long long N, float sh,
                                                         int mode, double* part) {
  __shared__ double red[8];
  double acc = 0.0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
    const float s = sinv[i];
    if (s > 0.f) {
      const double m2 = (double)u[i].x * u[i].x + (double)u[i].y * u[i].y;
      acc += mode == 0 ? m2 * s : m2 / (double)(s + sh);
    }
  }
  const double t = block_sum(acc, red);
  if (threadIdx.x == 0) part[blockIdx.x] = t;
}

__global__ void k_scale(float2* u, long long N, float f) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < N) u[i] = make_float2(u[i].x * f, u[i].y * f);
}

// Device restatement of HMCParameters::update over a given MH-rate sequence (diagnostics).
// A wait that runs out: an mbarrier that nothing arrives on, waited for with a limit of limit_ms (the bounded-wait
// path every pipeline in this library takes when a copy or an MMA does not complete).
__global__ void k_debug_bounded_wait(uint64_t limit_ns, int* gave_up, unsigned long long* waited_ns) {
  __shared__ uint64_t bar;
  if (threadIdx.x != 0) return;
  mbar_init(&bar, 1);
  mbar_fence_init();
  const uint64_t t0 = globaltimer_ns();
  const bool ok = mbar_wait_bounded(&bar, 0, limit_ns);
  *waited_ns = globaltimer_ns() - t0;
  *gave_up = ok ? 0 : 1;
}

__global__ void k_debug_dual_averaging(ChainState st, int n, const float* rates, double* eps_out, int* steps_out) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  for (int i = 0; i < n; i++) {
    hmc_update(st, rates[i]);
    eps_out[i] = st.eps;
    steps_out[i] = hmc_steps(st);
  }
}

}  // namespace drb
