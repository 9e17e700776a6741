// fg_kernels.cuh -- device kernels of one feram MD step on B200.
//
// Device layout (chosen for the GPU, converted at the C-ABI boundary):
//   real fields  u, p, F, work : [comp][z][y][x]            (x contiguous)
//   spectra      spec          : [comp][z][ky_slot][kx_slot], row pitch KXP
//   k tables     dtab, ckmod   : [ky_slot][kz_slot][kx_slot][entries]
// Slots are the digit-reversed positions left by the in-place DIF FFT
// stages (fft_smem.cuh); rev{x,y,z} give the true wavenumber of a slot.
//
// One force evaluation (mirror_force_mirror.F:6-89) is four passes:
//   k_xy_fwd     per (z-plane, component): r2c along x + DIF along y of
//                u and u (x) u (dipoFFT.F:19-44) -> spec
//   k_z_lane (k_z_kspace for the lengths and options it does not take)
//                per (kx tile, ky): DIF along z, every k-space operation
//                (dipole-dipole multiply, inhomogeneous strain solve,
//                energies), DIT along z
//   k_xy_inv     per (z-plane, component): DIT along y + c2r along x
//   k_assemble   per site: dipole-dipole + anharmonic + field + homogeneous
//                and inhomogeneous strain coupling forces
#pragma once
#include "fft_lane.cuh"

#include <type_traits>

namespace fg {

// energy slots, fg_energy member order (energy_module.F:7-23)
enum {
  E_ACOU = 0, E_DIPO, E_SHORT, E_LONG, E_DIPE, E_UNH, E_HS, E_HC, E_IS, E_IC, E_IM, E_TOT, E_HNP, E_COUNT
};
constexpr int NQ_K = 5;   // k-space partial sums per block
constexpr int NQ_R = 2;   // real-space partial sums per block
constexpr int RED_THREADS = 256;

struct Geom {
  int Lx, Ly, Lz, m, NKX, KXP;
  long long plane_r;  // Lx*Ly
  long long plane_c;  // Ly*KXP
  long long nsite;    // Lx*Ly*Lz
  long long ncplx;    // Lz*Ly*KXP
  long long nkpos;    // Ly*Lz*KXP
  // Mixed path: sums of u and u u, [didi_rows][9], one row per warp of a
  // plane's block, written by the forward x-y pass and summed by
  // homo_strain_tail (null: FP64 path, whose spectra have them).  The products
  // are FP32; the two-stage kernels add the values of one butterfly (up to 64,
  // cv_sum) in FP32, the general kernels the two of a pair, and every sum from
  // there on is FP64.  The homogeneous strain and the k = 0 part of the dipole
  // energies follow these nine numbers; the rounding of the FP32 spectrum they
  // replace (4e-8 of its k = 0 value) moved the energies by 1e-3 eV from step to
  // step at 64^3, the largest part of the thermostat's error.  k0_exact: the k-space pass
  // leaves k = 0 out of the dipole energies and the tail adds it.
  int k0_exact, didi_rows;
  double* didi;
};

// Constants of the Hamiltonian and integrators, resident on the device.
struct Phys {
  double N, Ninv;
  double j[7], kap2x2;                       // short range (dipole-dipole-short-range.F)
  double P_alpha, P_gamma, P_k1, P_k2, P_k3, P_k4;
  double fa2g, tg, sk, tk2, fk;              // dVddi-unharmonic.F:28-32
  double B11, B12, B44;
  double HC2[6][6];                          // homogeneous_coupling_2 (elastic.F:60-75)
  double H[6][6], HG[6][6], HG_inv[6];       // homogeneous, Cholesky (elastic.F:26-52)
  double pNa03[3], epi_strain;
  int bulk_or_film;
  double Zstar;
  double dt, dt_2, Q, nf_kT, threeN_kT;
  double Qinv;       // 1 / Q
  double ke_scale;   // N / (2 n_sum_p): kinetic energy per masked sum p^2/m
  double target_ke;  // target_kinetic_energy (param_module.F:468), velocity scaling
  // per-species on-site constants for .relaxor runs (dVddi-unharmonic.F:
  // 28-32,40,73): force combinations, energy coefficients, kappa2(s)-kappa2(1)
  struct Species {
    double fa2g, tg, sk, tk2, fk, k4x8, Pa, Pg, P1, P2, P3, P4, dk2;
  } sp[3];
  double n_sum_p;
  int E_on;
  int modulation_on;
  // per-step field of molecular-dynamics.F:66-76 evaluated on the device
  // (fg_set_wave): wave(E_wave_type, i_step, n_thermalize, n_E_wave_period,
  // external_E_field) of wave_module.F:8-67
  int wave_type, wave_n_thermalize, wave_period, wave_pad;
  double wave_amp[3];
};

struct DevScalars {
  double s, pi, H0, s_old;
  double kick_coef;   // p <- p - kick_coef * F
  double drift_coef;  // u <- u + drift_coef * p * m^-1
  double lf_dt, lf_dt_2;
  double e[E_COUNT];
  double strain[6];
  double w_hom[6];    // sum_i strain_i * HC2(i, j)
  double didiK0[6];   // Re didiK(k = 0)
  double D0[6];       // the dipole table at k = 0 (Geom::k0_exact)
  double E[3];        // uniform external field
  double ke_sum;      // last masked sum p^2/m
  // Nose-Poincare half step (35a), (38), (35c) of the next step, prepared by
  // the closing tail of the previous one (or by np_prepare) and committed by
  // block 0 of the next closing kick: masked sum p^2/m and KE at the half
  // step, pi_{n+1/2}, s_{n+1}, the drift coefficient and the (35f) kick
  // coefficient dt/2 s_{n+1}.
  double pend_ke_sum, pend_ke, pend_pi, pend_s, pend_drift, pend_kick_f;
  double vs_scale;       // velocity scaling factor of the last vs step
  double vs_scale_acou;  // the same for the acoustic momenta
  long long i_step;      // step counter of the device-side field schedule
  int status;
  int pad;
};

// Per-replica buffers of a grouped launch: replicas of one supercell size,
// precision and material (the points of a sweep) stepped by one launch per
// kernel, the replica index being the grid's last dimension.  Each kernel
// that takes a RepArgs table replaces its per-replica pointer arguments by
// its replica's entry; null = a launch for one context.
struct RepArgs {
  void* u;
  void* p;
  void* F;
  void* spec;
  void* rwork;
  const void* dtab;
  const Phys* ph;
  DevScalars* sc;
  double* part_k;
  double* part_r;
  double* part_ke;
  unsigned int* done_as;  // k_assemble's last-block ticket
  const double* layer_minv;
  const unsigned char* layer_sump;
  double* didi;           // Geom::didi of the replica
};

// ---------------------------------------------------------------- reductions
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// v of lane `lane`, the whole warp converged
#ifndef FG_HOST_EMU
__device__ __forceinline__ double lane_value(double v, int lane) { return __shfl_sync(0xffffffffu, v, lane); }
#else
inline double lane_value(double v, int) { return v; }  // the emulated launches run no scalar tails
#endif

// Block-wide sum of NQ values; thread q < NQ writes part[blockid*NQ + q].
// Fixed reduction order, so results are reproducible run to run.
template <int NQ>
__device__ void block_partials(double* v, double* part, long long blockid) {
  __shared__ double red[32][NQ];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    double s = warp_sum(v[q]);
    if (lane == 0) red[wid][q] = s;
  }
  __syncthreads();
  if (threadIdx.x < NQ) {
    const int q = threadIdx.x, nw = (blockDim.x + 31) >> 5;
    double s = 0.0;
    for (int w = 0; w < nw; ++w) s += red[w][q];
    part[blockid * NQ + q] = s;
  }
  __syncthreads();
}

// The same for two sets of sums with arrays of their own, in one pass.
template <int NA, int NB>
__device__ void block_partials2(const double* va, const double* vb, double* pa, double* pb, long long blockid) {
  __shared__ double red[32][NA + NB];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int q = 0; q < NA + NB; ++q) {
    const double s = warp_sum(q < NA ? va[q < NA ? q : 0] : vb[q < NA ? 0 : q - NA]);
    if (lane == 0) red[wid][q] = s;
  }
  __syncthreads();
  if (threadIdx.x < NA + NB) {
    const int q = threadIdx.x;
    double s = 0.0;
    for (int w = 0; w < nw; ++w) s += red[w][q];
    (q < NA ? pa[blockid * NA + q] : pb[blockid * NB + q - NA]) = s;
  }
  __syncthreads();
}

// Sum of part[b*NQ + q] over b in fixed order by one RED_THREADS block.
__device__ double reduce_partials(const double* part, int nblk, int NQ, int q) {
  __shared__ double red[RED_THREADS];
  double s = 0.0;
  for (int b = threadIdx.x; b < nblk; b += blockDim.x) s += __ldcg(&part[(long long)b * NQ + q]);
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  double r = red[0];
  __syncthreads();
  return r;
}

// Scalar work of a tail: thread 0 runs body on shared-memory copies of the
// constants and scalars, loaded and stored back by the whole block in one
// round trip each (instead of a chain of dependent global loads and stores
// by one thread).
static_assert(sizeof(DevScalars) % 8 == 0, "DevScalars is copied as doubles");
static_assert(sizeof(Phys) % 8 == 0, "Phys is copied as doubles");
// The reduction of one or two sets of block partials (columns 0 .. NA-1 from
// the nblk rows of pa, then NB from the nblk_b rows of pb) and the scalar work
// on the totals v[NA + NB]: the loads of the constants and scalars are in
// flight with those of the partials, so a tail costs one round trip to the
// L2, not two.  Lane l of a warp takes column l % PA (PB) of the rows its
// thread index selects: 3 to 7 shuffles a warp, where every thread taking whole
// rows needs 5 per column (14 columns: 140 instructions a warp, all in one
// SM's shuffle unit).  The loads are batched by hand: left to the compiler
// they went out one by one (28 us for 64^3's plane sums, 14 batched).  body
// runs on the first LANES threads.  host (may be null): the host's copy of the
// scalars, in pinned memory, for the calls that return a step's energies: 0.6
// kB of posted writes instead of a copy of its own after the last kernel.
// Step of 16^3, mixed: 22.5 -> 21.5 us with this and the nine plane sums that
// cost 1.7 us before it.
template <int N>
struct PadCols {
  static constexpr int value = N <= 1 ? 1 : N <= 2 ? 2 : N <= 4 ? 4 : N <= 8 ? 8 : 16;
};
// The thread's sums of both sets, 8 loads of each in flight.
template <int NA, int NB>
__device__ __forceinline__ void column_sums(const double* __restrict__ pa, int na, const double* __restrict__ pb, int nb,
                                            double* sa, double* sb) {
  constexpr int PA = PadCols<NA>::value, PB = PadCols<NB>::value, U = 8;
  const int ca = threadIdx.x % PA, ra = blockDim.x / PA;
  const int cb = threadIdx.x % PB, rb = blockDim.x / PB;
  int ia = threadIdx.x / PA, ib = threadIdx.x / PB;
  if (ca >= NA) ia = na;
  if (NB == 0 || cb >= NB) ib = nb;
  *sa = *sb = 0.0;
  while (ia < na || ib < nb) {
    double a[U], b[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const int i = ia + k * ra, j = ib + k * rb;
      a[k] = i < na ? __ldcg(&pa[(long long)i * NA + ca]) : 0.0;
      b[k] = NB > 0 && j < nb ? __ldcg(&pb[(long long)j * NB + cb]) : 0.0;
    }
#pragma unroll
    for (int k = 0; k < U; ++k) {
      *sa += a[k];
      *sb += b[k];
    }
    ia += U * ra;
    ib += U * rb;
  }
}
template <int N>
__device__ __forceinline__ double column_warp_sum(double s) {
#pragma unroll
  for (int o = 16; o >= PadCols<N>::value; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  return s;
}
template <int NA, int NB, int LANES = 1, class F>
__device__ __forceinline__ void reduced_tail(const Phys* __restrict__ ph, DevScalars* sc, const double* __restrict__ pa,
                                             const double* __restrict__ pb, int nblk, int nblk_b, F&& body,
                                             DevScalars* host = nullptr) {
  constexpr int NQ = NA + NB;
  __shared__ Phys sph;
  __shared__ DevScalars ssc;
  __shared__ double red[NQ][32];
  __shared__ double tot[NQ];
  constexpr int NP = (int)(sizeof(Phys) / 8), NS = (int)(sizeof(DevScalars) / 8);
  for (int i = threadIdx.x; i < NP; i += blockDim.x)
    reinterpret_cast<double*>(&sph)[i] = __ldg(reinterpret_cast<const double*>(ph) + i);
  for (int i = threadIdx.x; i < NS; i += blockDim.x)
    reinterpret_cast<double*>(&ssc)[i] = __ldcg(reinterpret_cast<const double*>(sc) + i);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  double sa, sb;
  column_sums<NA, NB>(pa, nblk, pb, nblk_b, &sa, &sb);
  const double ta = column_warp_sum<NA>(sa);
  if (lane < NA) red[lane][wid] = ta;
  if constexpr (NB > 0) {
    const double tb = column_warp_sum<NB>(sb);
    if (lane < NB) red[NA + lane][wid] = tb;
  }
  __syncthreads();
  if (threadIdx.x < NQ) {
    double t = 0.0;
    for (int w = 0; w < nw; ++w) t += red[threadIdx.x][w];
    tot[threadIdx.x] = t;
  }
  __syncthreads();
  if (threadIdx.x < LANES) body(static_cast<const Phys*>(&sph), &ssc, tot);
  __syncthreads();
  for (int i = threadIdx.x; i < NS; i += blockDim.x) {
    const double v = reinterpret_cast<const double*>(&ssc)[i];
    reinterpret_cast<double*>(sc)[i] = v;
    if (host) reinterpret_cast<double*>(host)[i] = v;
  }
}

// Last-block-done: thread 0 of every block fences the block's partials and
// takes a ticket; the block drawing the last ticket sees all of them and
// finishes the grid-wide work (classic threadfence reduction, no waiting).
// The counter is reset for the next launch by that block.  Only thread 0
// fences, after the barrier that puts the partials' stores by the block's
// first warp before it: the tails read nothing but those partials (and values
// whose writers fence themselves).
__device__ __forceinline__ bool is_last_block(unsigned int* counter, unsigned nblocks) {
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned t = atomicAdd(counter, 1u);
    last = (t == nblocks - 1);
    if (last) *counter = 0u;
  }
  __syncthreads();
  if (last) __threadfence();
  return last;
}

__device__ __forceinline__ bool is_last_block(unsigned int* counter) { return is_last_block(counter, gridDim.x); }

// ------------------------------------------------------- analytic short range
// S(k) of the 27-point stencil of dipole-dipole-short-range.F:35-83 (2 kappa2
// on site, j1..j7 on the first three neighbour shells), evaluated from the
// cosines and sines of theta_a = 2 pi k_a / L_a.  Valid for L_a >= 3.
// Order: xx, yy, zz, yz, zx, xy.
__host__ __device__ inline void short_range_k(const double* j, double kap2x2, const double c[3], const double s[3],
                                              double S[6]) {
  for (int a = 0; a < 3; ++a) {
    const int b = (a + 1) % 3, g = (a + 2) % 3;
    S[a] = kap2x2 + 2 * j[1] * c[a] + 2 * j[0] * (c[b] + c[g]) + 4 * j[3] * c[b] * c[g] +
           4 * j[2] * c[a] * (c[b] + c[g]) + 8 * j[5] * c[0] * c[1] * c[2];
  }
  // off-diagonal (a, b) with third axis g: -4 j5 s_a s_b - 8 j7 s_a s_b c_g
  S[3] = -4 * j[4] * s[1] * s[2] - 8 * j[6] * s[1] * s[2] * c[0];  // yz
  S[4] = -4 * j[4] * s[2] * s[0] - 8 * j[6] * s[2] * s[0] * c[1];  // zx
  S[5] = -4 * j[4] * s[0] * s[1] - 8 * j[6] * s[0] * s[1] * c[2];  // xy
}

__device__ __noinline__ void homo_strain_tail(const Phys* __restrict__ ph, DevScalars* sc,
                                              const double* __restrict__ part_k, int nblk,
                                              const double* __restrict__ didi, const Geom g);

// ------------------------------------------------------------------ k_xy_fwd
enum { SRC_U9 = 0, SRC_FIELD = 1 };

// Per (z-plane, component): load a real plane, DIF along x on Lx/2 complex
// pairs, unpack to the Lx/2+1 bins of the real transform, DIF along y.
// SRC_U9: component c of (u_x, u_y, u_z, u_x^2, u_y^2, u_z^2, u_y u_z,
// u_z u_x, u_x u_y) from u (dipoFFT.F:19-44); components 9..11 are src
// components 3..5 (the acoustic displacement stored after u); with a per-site
// Z* (zstar != null) components zu0..zu0+2 are Z*(R) u (Z_u_R, dipoFFT.F:
// 36-44).  SRC_FIELD: component c of src.
// MC, LYC > 0 select the compile-time transforms for m = Lx/2 = MC and
// Ly = LYC (xy_fwd_ct / xy_inv_ct, launched with XyCT::NT threads); 0 =
// runtime plans (512 threads).  The compile-time kernels run the y transforms
// on MC columns, not MC + 1: the kx = 0 and kx = Lx/2 columns are real before
// the y pass (transforms of real rows), so X(0) + i X(Lx/2) travels as one
// complex column and is split by Hermitian symmetry after the pass (y_split);
// the inverse joins them the same way before its y pass (y_join).  posm + m
// and posm + m + Ly hold the y slot maps (slot -> ky, ky -> slot) that pair
// ky with -ky.
constexpr int kXYThreads = 512;

// Column kx = 0 after the forward y pass holds C = Y0 + i Ym, Y0 and Ym the
// y spectra of the real kx = 0 and kx = Lx/2 columns: Y0(k) = (C(k) +
// conj C(-k)) / 2, Ym(k) = (C(k) - conj C(-k)) / 2i.  a = C(k), b = C(-k).
template <typename C>
__device__ __forceinline__ void y_split(C a, C b, C& y0, C& ym) {
  using R = decltype(a.x);
  y0 = mk<C>((R)0.5 * (a.x + b.x), (R)0.5 * (a.y - b.y));
  ym = mk<C>((R)0.5 * (a.y + b.y), (R)0.5 * (b.x - a.x));
}
// Inverse: C(k) = H0(k) + i Hm(k) with H(k) = (Y(k) + conj Y(-k)) / 2, the
// Hermitian part, whose inverse transform is the real part of Y's (the
// imaginary parts of the kx = 0 and kx = Lx/2 bins are dropped, as FFTW's
// c2r does).  a0 = Y0(k), b0 = Y0(-k), am = Ym(k), bm = Ym(-k).
template <typename C>
__device__ __forceinline__ C y_join(C a0, C b0, C am, C bm) {
  using R = decltype(a0.x);
  const R h0x = (R)0.5 * (a0.x + b0.x), h0y = (R)0.5 * (a0.y - b0.y);
  const R hmx = (R)0.5 * (am.x + bm.x), hmy = (R)0.5 * (am.y - bm.y);
  return mk<C>(h0x - hmy, h0y + hmx);
}

// Shapes of the compile-time x-y transforms of a plane, on elements of W
// transforms (fft_lane.cuh).
//   x: rows q + NQ (2 l + h) of the plane (l < W, h < 2) form one group: rows
//      h = 0 and 1 are the real and imaginary part of one complex transform of
//      length Lx, and the W pairs its lanes.  R1 x R2 stages; the second stage
//      takes the butterflies of k and -k in one thread (R1/2 tasks per group),
//      which separates the two rows' half spectra in registers: no pass of its
//      own for the real transform, no twiddles for it.
//   y: W neighbouring x slots form one element; RY1 x RY2 stages.
// A plane thus takes three round trips through shared memory.  Groups are
// stored [q][x] with a row of Lx + 1 elements, columns [j][y] with Ly + 1:
// every stage's 8 neighbouring lanes touch 8 different 16-byte banks, and all
// element offsets of a thread are compile-time constants.  NT threads hold
// one second-stage task each (at most 16 elements = 64 registers of data);
// 512 threads of them fill an SM's registers.
template <typename T, int MC, int LYC>
struct XyCT {
  static constexpr int W = kLanes<T>;
  static constexpr int LX = 2 * MC, R1 = ct_radix(MC, 0), R2 = LX / R1;
  static constexpr int RY1 = ct_radix(LYC, 0), RY2 = LYC / RY1;
  static constexpr int NQ = LYC / (2 * W), NJ = MC / W;
  static constexpr int QS = LX + 1, JS = LYC + 1;
  // First x stage (and last inverse one): the butterfly of offset b reads
  // x = b + R2 s.  Group q takes the same butterfly from offset
  // bg = b + R2 (q % G) on, wrapping around the row (the transform of a
  // rotated sequence, whose twiddles are those of offset bg), so that the
  // lanes of a warp, R2 offsets of 32 / R2 rows, are spread over a row's
  // 128-byte lines instead of hitting one 32-byte bank group in each row.
  static constexpr int G = 32 / R2 < R1 ? 32 / R2 : R1;
  static constexpr int NB = R2 * G;
  static constexpr int T2 = (R1 / 2) * NQ;  // tasks of the second x stage
  static constexpr int NT = (T2 + 31) / 32 * 32;
  static __device__ __forceinline__ int wrap(int x) { return x < LX ? x : x - LX; }
  static_assert(R1 % 2 == 0 && (R2 / 2) % W == 0 && 32 % R2 == 0 && LYC % (2 * W) == 0 && ct_nst(MC) == 2 && ct_nst(LYC) == 2, "");
};
template <typename T, int MC, int LYC>
constexpr int xy_threads() {
  if constexpr (MC > 0) return XyCT<T, MC, LYC>::NT;
  else return kXYThreads;
}
template <typename T, int MC, int LYC>
constexpr int xy_min_blocks() {
  if constexpr (MC > 0) return 512 / XyCT<T, MC, LYC>::NT;
  else return sizeof(T) == 4 ? 2 : 1;
}

// Real fields of a plane as the lanes and parts of a group (row offsets in
// elements of T from the group's first row).
template <typename T, int NQ, int LX>
__device__ __forceinline__ CV<T> group_ld(const T* p) {
  return CV<T>{vpack(p[0], sizeof(T) == 4 ? p[2 * NQ * LX] : (T)0),
               vpack(p[NQ * LX], sizeof(T) == 4 ? p[3 * NQ * LX] : (T)0)};
}
template <int L, int NQ, int LX, typename T>
__device__ __forceinline__ void group_st(T* p, const CV<T>& v) {
  p[2 * L * NQ * LX] = vget<L>(v.re);
  p[(2 * L + 1) * NQ * LX] = vget<L>(v.im);
}

// The second x stage pairs class a (k = a + R1 t) with class R1 - a; class 0
// and class R1/2 pair with themselves and share a task.  For that task this
// moves the partners to where the other tasks have them: the upper half of
// v1 becomes the partners of class 0's lower half (with Z(Lx/2) in the last
// place, opposite Z(0)), the upper half of v0 those of class R1/2.
template <typename T, int R2>
__device__ __forceinline__ void self_partners(CV<T>* v0, CV<T>* v1) {
  const CV<T> nyq = v0[R2 / 2];
#pragma unroll
  for (int s = R2 / 2; s < R2; ++s) {
    const CV<T> p = s + 1 < R2 ? v0[s + 1 < R2 ? s + 1 : 0] : nyq;
    v0[s] = v1[s];
    v1[s] = p;
  }
}
template <typename T, int R2>
__device__ __forceinline__ void self_partners_undo(CV<T>* v0, CV<T>* v1) {
  CV<T> up[R2 / 2];
#pragma unroll
  for (int s = R2 / 2; s < R2; ++s) up[s - R2 / 2] = v1[s];
#pragma unroll
  for (int s = R2 / 2; s < R2; ++s) v1[s] = v0[s];
#pragma unroll
  for (int s = R2 / 2; s + 1 < R2; ++s) v0[s + 1] = up[s - R2 / 2];
  v0[R2 / 2] = up[R2 / 2 - 1];
}

// Lane L of group q: the columns t and t+1 (one W-wide element; W = 1: column
// t) of rows h = 0, 1 from Z(k) = A and Z(-k) = B, already halved:
// X0 = Z(k) + conj Z(-k), X1 = -i (Z(k) - conj Z(-k)).  dc: A, B hold Z(0) and
// Z(Lx/2); the column is X(0) + i X(Lx/2).
template <int L, typename T>
__device__ __forceinline__ void unpack_rows(const CV<T>& A, const CV<T>& B, bool dc, T* x0, T* x1) {
  const T ar = vget<L>(A.re), ai = vget<L>(A.im), br = vget<L>(B.re), bi = vget<L>(B.im);
  if (dc) {
    x0[0] = ar + ar;
    x0[1] = br + br;
    x1[0] = ai + ai;
    x1[1] = bi + bi;
  } else {
    x0[0] = ar + br;
    x0[1] = ai - bi;
    x1[0] = ai + bi;
    x1[1] = br - ar;
  }
}
// and back: Z(k) = X0 + i X1, Z(-k) = conj X0 + i conj X1.
template <typename T>
__device__ __forceinline__ void pack_rows(const T* x0, const T* x1, bool dc, T* z, T* zm) {
  if (dc) {
    z[0] = x0[0];
    z[1] = x1[0];
    zm[0] = x0[1];
    zm[1] = x1[1];
  } else {
    z[0] = x0[0] - x1[1];
    z[1] = x0[1] + x1[0];
    zm[0] = x0[0] + x1[1];
    zm[1] = x1[0] - x0[1];
  }
}

// Stores / loads of the columns of one class (R2/2 columns from slot0) of
// group q in the [j][y] layout.
template <typename T, int MC, int LYC, int L>
__device__ __forceinline__ void class_to_columns(CV<T>* buf, const CV<T>* lo, const CV<T>* up, int slot0, int q, bool dc0) {
  using C = XyCT<T, MC, LYC>;
  constexpr int H = C::R2 / 2, W = C::W;
#pragma unroll
  for (int t = 0; t < H; t += W) {
    T a0[2], a1[2], b0[2], b1[2];
    unpack_rows<L>(lo[t], up[C::R2 - 1 - t], dc0 && t == 0, a0, a1);
    if (W == 2) unpack_rows<L>(lo[t + W - 1], up[C::R2 - t - W], false, b0, b1);
    CV<T>* d = buf + (slot0 + t) / W * C::JS + q + 2 * L * C::NQ;
    cv_st(d, CV<T>{vpack(a0[0], W == 2 ? b0[0] : (T)0), vpack(a0[1], W == 2 ? b0[1] : (T)0)});
    cv_st(d + C::NQ, CV<T>{vpack(a1[0], W == 2 ? b1[0] : (T)0), vpack(a1[1], W == 2 ? b1[1] : (T)0)});
  }
}
template <typename T, int MC, int LYC>
__device__ __forceinline__ void columns_to_class(const CV<T>* buf, CV<T>* lo, CV<T>* up, int slot0, int q, bool dc0) {
  using C = XyCT<T, MC, LYC>;
  constexpr int H = C::R2 / 2, W = C::W;
#pragma unroll
  for (int t = 0; t < H; t += W) {
    const CV<T>* d = buf + (slot0 + t) / W * C::JS + q;
    CV<T> x[2 * W];  // rows h + 2 l
#pragma unroll
    for (int r = 0; r < 2 * W; ++r) x[r] = cv_ld(d + r * C::NQ);
    T z[W][W][2], zm[W][W][2];  // [column][lane]
#pragma unroll
    for (int l = 0; l < W; ++l) {
      {
        const T x0[2] = {vget<0>(x[2 * l].re), vget<0>(x[2 * l].im)}, x1[2] = {vget<0>(x[2 * l + 1].re), vget<0>(x[2 * l + 1].im)};
        pack_rows(x0, x1, dc0 && t == 0, z[0][l], zm[0][l]);
      }
      if (W == 2) {
        const T x0[2] = {vget<1>(x[2 * l].re), vget<1>(x[2 * l].im)}, x1[2] = {vget<1>(x[2 * l + 1].re), vget<1>(x[2 * l + 1].im)};
        pack_rows(x0, x1, false, z[W - 1][l], zm[W - 1][l]);
      }
    }
#pragma unroll
    for (int k = 0; k < W; ++k) {
      lo[t + k] = CV<T>{vpack(z[k][0][0], z[k][W - 1][0]), vpack(z[k][0][1], z[k][W - 1][1])};
      up[C::R2 - 1 - t - k] = CV<T>{vpack(zm[k][0][0], zm[k][W - 1][0]), vpack(zm[k][0][1], zm[k][W - 1][1])};
    }
  }
}

// Sum of the values of n elements, in FP32 (the mixed path's plane sums): two
// chains of n over the pairs of lanes, then those.
__device__ __forceinline__ float cv_sum(const CV<float>* v, int n) {
  F2 a = v[0].re, b = v[0].im;
#pragma unroll
  for (int s = 1; s < n; ++s) {
    a = vadd(a, v[s].re);
    b = vadd(b, v[s].im);
  }
  a = vadd(a, b);
  return vget<0>(a) + vget<1>(a);
}
__device__ __forceinline__ double cv_sum(const CV<double>*, int) { return 0.0; }
// Geom::didi entry of component c of plane z's first warp, null where there
// is none; every warp writes its own row.
template <typename T, int MODE>
__device__ __forceinline__ double* plane_didi(const Geom& g, const RepArgs* grp, int c, int z) {
  if (MODE != 0 || sizeof(T) != 4 || g.didi == nullptr || c > 8) return nullptr;
  return (grp ? grp[blockIdx.z].didi : g.didi) + (long long)z * (blockDim.x / 32) * 9 + c;
}
__device__ __forceinline__ void plane_sum(double s, double* didi) {
  s = warp_sum(s);
  if (threadIdx.x % 32 == 0) didi[threadIdx.x / 32 * 9] = s;
}

// Forward transform of one plane: pa (and, for products, pb) the real rows,
// dst the plane's spectrum rows.  128^2 FP32: 256 threads, 2 CTAs per SM.
enum { PLANE_PLAIN = 0, PLANE_SQUARE = 1, PLANE_PRODUCT = 2 };
template <typename T, int MC, int LYC>
__device__ __forceinline__ void xy_fwd_ct(const T* __restrict__ pa, const T* __restrict__ pb, int kind,
                                          cplx<T>* __restrict__ dst, int kxp, unsigned char* smem,
                                          const cplx<T>* __restrict__ twx, const cplx<T>* __restrict__ twy,
                                          const int* __restrict__ posm, double* __restrict__ didi) {
  using C = XyCT<T, MC, LYC>;
  constexpr int NT = C::NT, R1 = C::R1, R2 = C::R2, RY1 = C::RY1, RY2 = C::RY2, W = C::W;
  CV<T>* buf = reinterpret_cast<CV<T>*>(smem);
  __shared__ cplx<T> tabx[R1 * C::NB], taby[LYC], col0[LYC];
  double sum = 0.0;
  stage_twiddles<T, C::LX, R1, C::NB>(tabx, twx, (T)0.5);  // halved: see unpack_rows
  stage_twiddles<T, LYC, RY1, RY2>(taby, twy, (T)1);
  __syncthreads();
  pdl_wait();
  // first x stage, from the real rows
  lane_tasks<C::NQ * R2, NT>((int)threadIdx.x, [&](int t) {
    const int b = t % R2, q = t / R2, bg = b + R2 * (q % C::G);
    const T* r = pa + q * C::LX;
    CV<T> v[R1];
#pragma unroll
    for (int s = 0; s < R1; ++s) v[s] = group_ld<T, C::NQ, C::LX>(r + C::wrap(bg + s * R2));
    if (kind == PLANE_PRODUCT) {
      const T* r2 = pb + q * C::LX;
#pragma unroll
      for (int s = 0; s < R1; ++s) {
        const CV<T> w = group_ld<T, C::NQ, C::LX>(r2 + C::wrap(bg + s * R2));
        v[s] = CV<T>{vmul(v[s].re, w.re), vmul(v[s].im, w.im)};
      }
    } else if (kind == PLANE_SQUARE) {
#pragma unroll
      for (int s = 0; s < R1; ++s) v[s] = CV<T>{vmul(v[s].re, v[s].re), vmul(v[s].im, v[s].im)};
    }
    if (didi) sum += (double)cv_sum(v, R1);
    DftV<T, R1, false>::run(v);
    CV<T>* d = buf + q * C::QS + b;
    const lane_t<T> half = vall((T)0.5);
    cv_st(d, CV<T>{vmul(v[0].re, half), vmul(v[0].im, half)});
#pragma unroll
    for (int s = 1; s < R1; ++s) cv_st(d + s * R2, cvtw<T, false>(v[s], tabx[s * C::NB + bg]));
  });
  if (didi) plane_sum(sum, didi);
  __syncthreads();
  // second x stage with the separation of the rows
  {
    const bool on = threadIdx.x < C::T2;
    const int q = threadIdx.x % C::NQ, al = on ? threadIdx.x / C::NQ : 0;
    const int a1 = al == 0 ? R1 / 2 : R1 - al;
    CV<T> v0[R2], v1[R2];
    if (on) {
      const CV<T>* r = buf + q * C::QS;
#pragma unroll
      for (int t = 0; t < R2; ++t) v0[t] = cv_ld(r + al * R2 + t);
#pragma unroll
      for (int t = 0; t < R2; ++t) v1[t] = cv_ld(r + a1 * R2 + t);
      DftV<T, R2, false>::run(v0);
      DftV<T, R2, false>::run(v1);
      if (al == 0) self_partners<T, R2>(v0, v1);
    }
    __syncthreads();
    if (on) {
      class_to_columns<T, MC, LYC, 0>(buf, v0, v1, al * (R2 / 2), q, al == 0);
      class_to_columns<T, MC, LYC, 0>(buf, v1, v0, a1 * (R2 / 2), q, false);
      if constexpr (W == 2) {
        class_to_columns<T, MC, LYC, 1>(buf, v0, v1, al * (R2 / 2), q, al == 0);
        class_to_columns<T, MC, LYC, 1>(buf, v1, v0, a1 * (R2 / 2), q, false);
      }
    }
  }
  __syncthreads();
  // first y stage
  lane_tasks<C::NJ * RY2, NT>((int)threadIdx.x, [&](int t) {
    const int j = t % C::NJ, b = t / C::NJ;
    CV<T>* d = buf + j * C::JS + b;
    CV<T> v[RY1];
#pragma unroll
    for (int s = 0; s < RY1; ++s) v[s] = cv_ld(d + s * RY2);
    DftV<T, RY1, false>::run(v);
    cv_st(d, v[0]);
#pragma unroll
    for (int s = 1; s < RY1; ++s) cv_st(d + s * RY2, cvtw<T, false>(v[s], taby[s * RY2 + b]));
  });
  __syncthreads();
  pdl_launch();
  // second y stage, to the spectrum rows; column 0 to shared memory first
  lane_tasks<C::NJ * RY1, NT>((int)threadIdx.x, [&](int t) {
    const int j = t % C::NJ, a = t / C::NJ;
    const CV<T>* d = buf + j * C::JS + a * RY2;
    CV<T> v[RY2];
#pragma unroll
    for (int s = 0; s < RY2; ++s) v[s] = cv_ld(d + s);
    DftV<T, RY2, false>::run(v);
    cplx<T>* o = dst + (long long)(a * RY2) * kxp + W * j;
    if (j == 0) {
#pragma unroll
      for (int s = 0; s < RY2; ++s) {
        col0[a * RY2 + s] = mk<cplx<T>>(vget<0>(v[s].re), vget<0>(v[s].im));
        if constexpr (W == 2) o[(long long)s * kxp + 1] = mk<cplx<T>>(vget<1>(v[s].re), vget<1>(v[s].im));
      }
    } else {
#pragma unroll
      for (int s = 0; s < RY2; ++s) cv_row(reinterpret_cast<rowvec<T>*>(o + (long long)s * kxp), v[s]);
    }
  });
  __syncthreads();
  const int *revy = posm + MC, *posy = posm + MC + LYC;
  for (int sl = threadIdx.x; sl < LYC; sl += NT) {
    const int sp = __ldg(&posy[(LYC - __ldg(&revy[sl])) % LYC]);
    cplx<T> y0, ym;
    y_split(col0[sl], col0[sp], y0, ym);
    dst[(long long)sl * kxp] = y0;
    dst[(long long)sl * kxp + MC] = ym;
  }
}

// Inverse transform of one plane: src its spectrum rows (consumed: evict
// first), out its real rows.
template <typename T, int MC, int LYC>
__device__ __forceinline__ void xy_inv_ct(const cplx<T>* __restrict__ src, T* __restrict__ out, int kxp,
                                          unsigned char* smem, const cplx<T>* __restrict__ twx,
                                          const cplx<T>* __restrict__ twy, const int* __restrict__ posm) {
  using C = XyCT<T, MC, LYC>;
  constexpr int NT = C::NT, R1 = C::R1, R2 = C::R2, RY1 = C::RY1, RY2 = C::RY2, W = C::W;
  CV<T>* buf = reinterpret_cast<CV<T>*>(smem);
  __shared__ cplx<T> tabx[R1 * C::NB], taby[LYC], col0[LYC];
  const unsigned long long pol = l2_evict_first();
  auto ldc = [&](const cplx<T>* a) {
    if constexpr (sizeof(T) == 4 || FG_L2_HINT_FP64) return ld_first(a, pol);
    else return *a;
  };
  // columns 0 and Lx/2 joined (y_join)
  const int *revy = posm + MC, *posy = posm + MC + LYC;
  for (int sl = threadIdx.x; sl < LYC; sl += NT) {
    const int sp = __ldg(&posy[(LYC - __ldg(&revy[sl])) % LYC]);
    const cplx<T>*r = src + (long long)sl * kxp, *rm = src + (long long)sp * kxp;
    col0[sl] = y_join(ldc(r), ldc(rm), ldc(r + MC), ldc(rm + MC));
  }
  stage_twiddles<T, C::LX, R1, C::NB>(tabx, twx, (T)1);
  stage_twiddles<T, LYC, RY1, RY2>(taby, twy, (T)1);
  __syncthreads();
  // y: the last forward stage (no twiddles) from the spectrum rows
  lane_tasks<C::NJ * RY1, NT>((int)threadIdx.x, [&](int t) {
    const int j = t % C::NJ, a = t / C::NJ;
    const cplx<T>* r = src + (long long)(a * RY2) * kxp + W * j;
    CV<T> v[RY2];
#pragma unroll
    for (int s = 0; s < RY2; ++s) {
      if constexpr (sizeof(T) == 4) v[s] = cv_of(ld_first(reinterpret_cast<const float4*>(r + (long long)s * kxp), pol));
      else v[s] = cv_of(ldc(r + (long long)s * kxp));
    }
    if (j == 0) {
#pragma unroll
      for (int s = 0; s < RY2; ++s) {
        const cplx<T> c = col0[a * RY2 + s];
        if constexpr (W == 2) v[s] = CV<T>{vpack(c.x, vget<1>(v[s].re)), vpack(c.y, vget<1>(v[s].im))};
        else v[s] = CV<T>{vpack(c.x, c.x), vpack(c.y, c.y)};
      }
    }
    DftV<T, RY2, true>::run(v);
    CV<T>* d = buf + j * C::JS + a * RY2;
#pragma unroll
    for (int s = 0; s < RY2; ++s) cv_st(d + s, v[s]);
  });
  __syncthreads();
  lane_tasks<C::NJ * RY2, NT>((int)threadIdx.x, [&](int t) {
    const int j = t % C::NJ, b = t / C::NJ;
    CV<T>* d = buf + j * C::JS + b;
    CV<T> v[RY1];
    v[0] = cv_ld(d);
#pragma unroll
    for (int s = 1; s < RY1; ++s) v[s] = cvtw<T, true>(cv_ld(d + s * RY2), taby[s * RY2 + b]);
    DftV<T, RY1, true>::run(v);
#pragma unroll
    for (int s = 0; s < RY1; ++s) cv_st(d + s * RY2, v[s]);
  });
  __syncthreads();
  // x: rows joined in pairs, the last forward stage
  {
    const bool on = threadIdx.x < C::T2;
    const int q = threadIdx.x % C::NQ, al = on ? threadIdx.x / C::NQ : 0;
    const int a1 = al == 0 ? R1 / 2 : R1 - al;
    CV<T> v0[R2], v1[R2];
    if (on) {
      columns_to_class<T, MC, LYC>(buf, v0, v1, al * (R2 / 2), q, al == 0);
      columns_to_class<T, MC, LYC>(buf, v1, v0, a1 * (R2 / 2), q, false);
      if (al == 0) self_partners_undo<T, R2>(v0, v1);
      DftV<T, R2, true>::run(v0);
      DftV<T, R2, true>::run(v1);
    }
    __syncthreads();
    if (on) {
      CV<T>* r = buf + q * C::QS;
#pragma unroll
      for (int t = 0; t < R2; ++t) cv_st(r + al * R2 + t, v0[t]);
#pragma unroll
      for (int t = 0; t < R2; ++t) cv_st(r + a1 * R2 + t, v1[t]);
    }
  }
  __syncthreads();
  pdl_launch();
  lane_tasks<C::NQ * R2, NT>((int)threadIdx.x, [&](int t) {
    const int b = t % R2, q = t / R2, bg = b + R2 * (q % C::G);
    const CV<T>* d = buf + q * C::QS + b;
    CV<T> v[R1];
    v[0] = cv_ld(d);
#pragma unroll
    for (int s = 1; s < R1; ++s) v[s] = cvtw<T, true>(cv_ld(d + s * R2), tabx[s * C::NB + bg]);
    DftV<T, R1, true>::run(v);
    T* r = out + q * C::LX;
#pragma unroll
    for (int s = 0; s < R1; ++s) {
      const int x = C::wrap(bg + s * R2);
      group_st<0, C::NQ, C::LX>(r + x, v[s]);
      if constexpr (W == 2) group_st<1, C::NQ, C::LX>(r + x, v[s]);
    }
  });
}

template <typename T, int MODE, int MC = 0, int LYC = 0>
__global__ void __launch_bounds__(xy_threads<T, MC, LYC>(), xy_min_blocks<T, MC, LYC>())
    k_xy_fwd(const T* __restrict__ src, cplx<T>* __restrict__ spec, Geom g, FftPlan px, FftPlan py,
             const cplx<T>* __restrict__ twx, const cplx<T>* __restrict__ twm, const cplx<T>* __restrict__ twy,
             const int* __restrict__ posm, int out_comp0, const T* __restrict__ zstar = nullptr, int zu0 = 0,
             const RepArgs* __restrict__ grp = nullptr) {
  if (grp) {
    src = (const T*)grp[blockIdx.z].u;
    spec = (cplx<T>*)grp[blockIdx.z].spec;
  }
  FG_DYN_SMEM(smem_raw);
  using T2 = typename RT2<T>::type;
  const int z = blockIdx.x, c = blockIdx.y;
  const long long plane_off = (long long)z * g.plane_r;
  // what component c is: Z*(R) u_(c - zu0), a plain field, or u_ca u_cb
  const bool zu = MODE == SRC_U9 && zstar != nullptr && c >= zu0;
  const bool plain = !zu && (MODE == SRC_FIELD || c < 3 || c >= 9);
  const int ca = zu ? c - zu0
                    : plain ? (c >= 9 && MODE == SRC_U9 ? c - 6 : c) : (c == 3 || c == 8) ? 0 : (c == 4 || c == 6) ? 1 : 2;
  const int cb = (c == 3) ? 0 : (c == 4) ? 1 : (c == 5) ? 2 : (c == 6) ? 2 : (c == 7) ? 0 : 1;
  const T* pa = src + (long long)ca * g.nsite + plane_off;
  const T* pb = zu ? zstar + plane_off : src + (long long)cb * g.nsite + plane_off;
  cplx<T>* dst = spec + (long long)(out_comp0 + c) * g.ncplx + (long long)z * g.plane_c;
  if constexpr (MC > 0) {
    const int kind = plain ? PLANE_PLAIN : (!zu && c < 6) ? PLANE_SQUARE : PLANE_PRODUCT;
    xy_fwd_ct<T, MC, LYC>(pa, pb, kind, dst, g.KXP, smem_raw, twx, twy, posm, plane_didi<T, MODE>(g, grp, c, z));
  } else {
    pdl_wait();
    cplx<T>* buf = reinterpret_cast<cplx<T>*>(smem_raw);
    const int m = g.m, Ly = g.Ly, RS = m + 1, Lx = 2 * m;
    const int buf_len = Ly * RS;
    const int total = Ly * m;
    double* const didi = plane_didi<T, MODE>(g, grp, c, z);
    double sum = 0.0;
    if (plain) {
      // asynchronous copies of packed (x even, x odd) pairs
      for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
        const int y = idx / m, jx = idx - y * m;
        cp_async<(int)sizeof(cplx<T>)>(&buf[y * RS + jx], pa + (long long)y * Lx + 2 * jx);
      }
      cp_async_wait();
      if (didi)  // this thread's own copies
        for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
          const int y = idx / m;
          const cplx<T> v = buf[y * RS + idx - y * m];
          sum += (double)(v.x + v.y);
        }
    } else {
      // products: kLB independent loads in flight per thread, then compute
      constexpr int kLB = 4;
      for (int base = threadIdx.x; base < total; base += kLB * blockDim.x) {
        T2 va[kLB], vb[kLB];
#pragma unroll
        for (int r = 0; r < kLB; ++r) {
          const int idx = base + r * blockDim.x;
          if (idx < total) {
            const int y = idx / m, jx = idx - y * m;
            const long long o = (long long)y * Lx + 2 * jx;
            va[r] = *reinterpret_cast<const T2*>(pa + o);
            vb[r] = *reinterpret_cast<const T2*>(pb + o);
          }
        }
#pragma unroll
        for (int r = 0; r < kLB; ++r) {
          const int idx = base + r * blockDim.x;
          if (idx < total) {
            const int y = idx / m, jx = idx - y * m;
            const cplx<T> v = mk<cplx<T>>(va[r].x * vb[r].x, va[r].y * vb[r].y);
            if (didi) sum += (double)(v.x + v.y);
            buf[y * RS + jx] = v;
          }
        }
      }
    }
    if (didi) plane_sum(sum, didi);
    // X pass; row stride RS = m+1 keeps the row-interleaved mapping bank-conflict free
    __syncthreads();
    Batch B{Ly, 1, 0, RS, 1, true};
    fft_forward<T>(buf, B, px, twm, buf_len);
    // unpack: slot posm[k] holds Z(k) of the packed row; X(k) = E(k) + w^k O(k)
    const int half = m / 2 + 1;
    // lanes run along y (same k): conflict-free rows, uniform posm and twiddle
    for (int idx = threadIdx.x; idx < Ly * half; idx += blockDim.x) {
      const int k = idx / Ly, y = idx - k * Ly;
      cplx<T>* row = buf + y * RS;
      if (k == 0) {
        const cplx<T> z0 = row[0];
        row[0] = mk<cplx<T>>(z0.x + z0.y, (T)0);
        row[m] = mk<cplx<T>>(z0.x - z0.y, (T)0);
      } else {
        const int k2 = m - k;
        const int s1 = __ldg(&posm[k]), s2 = __ldg(&posm[k2]);
        const cplx<T> a = row[s1], b = row[s2];
        const cplx<T> w1 = twx[k], w2 = twx[k2];
        // X(k) = 1/2 (a + conj b) - i/2 w1 (a - conj b)
        const cplx<T> e1 = mk<cplx<T>>(a.x + b.x, a.y - b.y), d1 = mk<cplx<T>>(a.x - b.x, a.y + b.y);
        const cplx<T> wd1 = cmul(w1, d1);
        const cplx<T> X1 = mk<cplx<T>>((T)0.5 * (e1.x + wd1.y), (T)0.5 * (e1.y - wd1.x));
        const cplx<T> e2 = mk<cplx<T>>(b.x + a.x, b.y - a.y), d2 = mk<cplx<T>>(b.x - a.x, b.y + a.y);
        const cplx<T> wd2 = cmul(w2, d2);
        const cplx<T> X2 = mk<cplx<T>>((T)0.5 * (e2.x + wd2.y), (T)0.5 * (e2.y - wd2.x));
        row[s1] = X1;
        if (s2 != s1) row[s2] = X2;
      }
    }
    __syncthreads();
    Batch By{RS, RS, 1, 0, RS, true};
    fft_forward<T>(buf, By, py, twy, buf_len);
    pdl_launch();
    for (int idx = threadIdx.x; idx < Ly * RS; idx += blockDim.x) {
      const int y = idx / RS, col = idx - y * RS;
      dst[(long long)y * g.KXP + col] = buf[idx];
    }
  }
}

// ------------------------------------------------------------------ k_xy_inv
// Per (z-plane, component): DIT along y, repack the Lx/2+1 bins into Lx/2
// complex pairs (imaginary parts of the kx = 0 and kx = Lx/2 bins dropped,
// the half-complex convention of the reference's c2r), DIT along x, store
// the real plane.  Output is unnormalised (Lx*Ly*Lz times the IDFT).
template <typename T, int MC = 0, int LYC = 0>
__global__ void __launch_bounds__(xy_threads<T, MC, LYC>(), xy_min_blocks<T, MC, LYC>())
    k_xy_inv(const cplx<T>* __restrict__ spec, T* __restrict__ out, Geom g, FftPlan px, FftPlan py,
             const cplx<T>* __restrict__ twx, const cplx<T>* __restrict__ twm, const cplx<T>* __restrict__ twy,
             const int* __restrict__ posm, int in_comp0, const Phys* __restrict__ ph, DevScalars* sc,
             const double* __restrict__ part_k, int nblk_k, const RepArgs* __restrict__ grp = nullptr) {
  pdl_wait();
  if (grp) {
    const RepArgs& a = grp[blockIdx.z];
    spec = (const cplx<T>*)a.spec;
    out = (T*)a.rwork;
    if (ph != nullptr) ph = a.ph;
    sc = a.sc;
    part_k = a.part_k;
  }
  // ph != null: the first row of blocks is no plane; its block 0 finishes the
  // k-space pass that wrote spec: its energies and the homogeneous strain,
  // from that pass's block partials (nothing in this kernel needs them;
  // k_assemble does), beside the transforms instead of ahead of a plane's.
  if (ph != nullptr && blockIdx.y == 0) {
    if (blockIdx.x == 0) homo_strain_tail(ph, sc, part_k, nblk_k, grp && g.didi ? grp[blockIdx.z].didi : g.didi, g);
    return;
  }
  FG_DYN_SMEM(smem_raw);
  using T2 = typename RT2<T>::type;
  const int z = blockIdx.x, c = blockIdx.y - (ph != nullptr ? 1 : 0);
  const cplx<T>* srcp = spec + (long long)(in_comp0 + c) * g.ncplx + (long long)z * g.plane_c;
  T* dst = out + (long long)c * g.nsite + (long long)z * g.plane_r;
  if constexpr (MC > 0) {
    xy_inv_ct<T, MC, LYC>(srcp, dst, g.KXP, smem_raw, twx, twy, posm);
  } else {
    cplx<T>* buf = reinterpret_cast<cplx<T>*>(smem_raw);
    const int m = g.m, Ly = g.Ly, RS = m + 1, Lx = 2 * m;
    const int buf_len = Ly * RS;
    for (int idx = threadIdx.x; idx < Ly * RS; idx += blockDim.x) {
      const int y = idx / RS, col = idx - y * RS;
      cp_async<(int)sizeof(cplx<T>)>(&buf[idx], srcp + (long long)y * g.KXP + col);
    }
    cp_async_wait();
    __syncthreads();
    Batch B{RS, RS, 1, 0, RS, true};
    fft_inverse<T>(buf, B, py, twy, buf_len);
    const int half = m / 2 + 1;
    // lanes run along y (same k): conflict-free rows, uniform posm and twiddle
    for (int idx = threadIdx.x; idx < Ly * half; idx += blockDim.x) {
      const int k = idx / Ly, y = idx - k * Ly;
      cplx<T>* row = buf + y * RS;
      if (k == 0) {
        const T X0 = row[0].x, Xm = row[m].x;
        row[0] = mk<cplx<T>>(X0 + Xm, X0 - Xm);
      } else {
        const int k2 = m - k;
        const int s1 = __ldg(&posm[k]), s2 = __ldg(&posm[k2]);
        const cplx<T> a = row[s1], b = row[s2];
        const cplx<T> w1 = twx[k], w2 = twx[k2];
        // Z(k) = (a + conj b) + i conj(w1) (a - conj b)
        const cplx<T> e1 = mk<cplx<T>>(a.x + b.x, a.y - b.y), d1 = mk<cplx<T>>(a.x - b.x, a.y + b.y);
        const cplx<T> wd1 = cmulc(d1, w1);
        const cplx<T> Z1 = mk<cplx<T>>(e1.x - wd1.y, e1.y + wd1.x);
        const cplx<T> e2 = mk<cplx<T>>(b.x + a.x, b.y - a.y), d2 = mk<cplx<T>>(b.x - a.x, b.y + a.y);
        const cplx<T> wd2 = cmulc(d2, w2);
        const cplx<T> Z2 = mk<cplx<T>>(e2.x - wd2.y, e2.y + wd2.x);
        row[s1] = Z1;
        if (s2 != s1) row[s2] = Z2;
      }
    }
    __syncthreads();
    Batch Bx{Ly, 1, 0, RS, 1, true};
    fft_inverse<T>(buf, Bx, px, twm, buf_len);
    pdl_launch();
    for (int idx = threadIdx.x; idx < Ly * m; idx += blockDim.x) {
      const int y = idx / m, jx = idx - y * m;
      const cplx<T> v = buf[y * RS + jx];
      T2 w;
      w.x = v.x;
      w.y = v.y;
      *reinterpret_cast<T2*>(dst + (long long)y * Lx + 2 * jx) = w;
    }
  }
}

constexpr int kLaneMax = 160;  // longest length of the runtime two-stage transforms

// ------------------------------------------------------- k_xy_fwd_gen / inv_gen
// The x-y passes of planes without a compile-time instance: the algorithm and
// layouts of XyCT with the lengths, strides and counts known at run time and
// the butterflies chosen by radix.  Any Lx = R1 R2 with R1 even (R2 may be
// odd), Ly = RY1 RY2 (lane_split).  Rows of a group past Ly (the last one's
// fourth, for Ly = 5 also its third) are zero;
// with an odd Lx/2 the last column element's second lane is a dummy.  Columns
// cross from the x to the y pass as complex values side by side, two per FP32
// element, in natural order: x slot = kx.
struct XyGeo {
  int R1, R2, RY1, RY2;
  int NQ, NJ, QS, JS;       // row groups, column elements, their strides
  FastDiv dR2, dNQ, dNJ;
  int nt, smem;             // threads, dynamic shared memory (this precision)
};

// f(k, A, B, dc) for every column k < Lx/2 of classes al and a1 held in v0, v1
// with A = Z(k), B = Z(-k); dc: column 0 with A = Z(0), B = Z(Lx/2).
template <int R2, class C, class F>
__device__ __forceinline__ void class_columns(C* v0, C* v1, int al, int a1, int R1, F&& f) {
  if (al != 0) {
#pragma unroll
    for (int t = 0; t < (R2 + 1) / 2; ++t) f(al + R1 * t, v0[t], v1[R2 - 1 - t], false);
#pragma unroll
    for (int t = 0; t < R2 / 2; ++t) f(a1 + R1 * t, v1[t], v0[R2 - 1 - t], false);
  } else {
    f(0, v0[0], R2 % 2 == 0 ? v0[R2 / 2] : v1[(R2 - 1) / 2], true);
#pragma unroll
    for (int t = 1; t < (R2 + 1) / 2; ++t) f(R1 * t, v0[t], v0[R2 - t], false);
#pragma unroll
    for (int t = 0; t < R2 / 2; ++t) f(a1 + R1 * t, v1[t], v1[R2 - 1 - t], false);
  }
}
// complex value of column k, row y in the column layout
template <typename T>
__device__ __forceinline__ cplx<T>* column_at(CV<T>* buf, int JS, int k, int y) {
  constexpr int W = kLanes<T>;
  return reinterpret_cast<cplx<T>*>(buf + k / W * JS + y) + k % W;
}

#if FG_BOUNDS_CHECK
// What the tasks of these kernels touch (fg_in_range):
// the first x stage's butterfly b of group q (elements of buf, rows of the
// plane, twiddles), class al of group q and its partner a1 (elements; columns and
// rows of the column layout) and block a of column element j (elements,
// spectrum rows).
template <int R, int W>
__device__ __forceinline__ bool group_in_range(const Geom& g, const XyGeo& h, int q, int b) {
  const int last = b + (R - 1) * h.R2;
  const int row = q + h.NQ * (2 * W - 1) < g.Ly ? q + h.NQ * (2 * W - 1) : q + 2 * h.NQ < g.Ly && W == 2 ? q + 2 * h.NQ
                  : W == 2 ? q + h.NQ : q;
  return fg_in_range(q * h.QS + b, q * h.QS + last, h.smem / 16) && fg_in_range(b, last, g.Lx) && fg_in_range(q, row, g.Ly) &&
         fg_in_range(0, (R - 1) * b, g.Lx);
}
template <int R, int W>
__device__ __forceinline__ bool classes_in_range(const Geom& g, const XyGeo& h, int q, int al) {
  const int a1 = al == 0 ? h.R1 / 2 : h.R1 - al;
  const int k0 = al + h.R1 * ((R - 1) / 2), k1 = a1 + h.R1 * (R / 2 - 1), k = k0 > k1 ? k0 : k1;
  return fg_in_range(q * h.QS + al * R, q * h.QS + a1 * R + R - 1, h.smem / 16) && fg_in_range(al, a1, h.R1) &&
         fg_in_range(al, k, g.m) && fg_in_range(q, k / W * h.JS + g.Ly - 1, h.smem / 16);
}
template <int R, int W>
__device__ __forceinline__ bool column_in_range(const Geom& g, const XyGeo& h, int j, int a) {
  return fg_in_range(j * h.JS + a * R, j * h.JS + a * R + R - 1, h.smem / 16) && fg_in_range(a * R, a * R + R - 1, g.Ly) &&
         fg_in_range(W * j, W * j + W - 1, g.KXP);
}
#endif

template <typename T, int MODE>
__global__ void __launch_bounds__(512, 1)
    k_xy_fwd_gen(const T* __restrict__ src, cplx<T>* __restrict__ spec, Geom g, XyGeo h, const cplx<T>* __restrict__ twx,
                 const cplx<T>* __restrict__ twy, const int* __restrict__ posm, const T* __restrict__ zstar, int zu0,
                 const RepArgs* __restrict__ grp) {
  constexpr int W = kLanes<T>;
  if (grp) {
    src = (const T*)grp[blockIdx.z].u;
    spec = (cplx<T>*)grp[blockIdx.z].spec;
  }
  FG_DYN_SMEM(smem_raw);
  CV<T>* const buf = reinterpret_cast<CV<T>*>(smem_raw);
  __shared__ cplx<T> tabx[kLaneMax], taby[kLaneMax], col0[kLaneMax];
  const int nt = blockDim.x, tid = threadIdx.x;
  const int Lx = g.Lx, Ly = g.Ly, m = g.m;
  const int z = blockIdx.x, c = blockIdx.y;
  double* const didi = plane_didi<T, MODE>(g, grp, c, z);
  double sum = 0.0;
  for (int k = tid; k < Lx; k += nt) tabx[k] = mk<cplx<T>>((T)0.5 * twx[k].x, (T)0.5 * twx[k].y);  // halved: unpack_rows
  for (int k = tid; k < Ly; k += nt) taby[k] = twy[k];
  __syncthreads();
  pdl_wait();
  const bool zu = MODE == SRC_U9 && zstar != nullptr && c >= zu0;
  const bool plain = !zu && (MODE == SRC_FIELD || c < 3 || c >= 9);
  const bool square = !zu && !plain && c < 6;
  const int ca = zu ? c - zu0
                    : plain ? (c >= 9 && MODE == SRC_U9 ? c - 6 : c) : (c == 3 || c == 8) ? 0 : (c == 4 || c == 6) ? 1 : 2;
  const int cb = (c == 3) ? 0 : (c == 4) ? 1 : (c == 5) ? 2 : (c == 6) ? 2 : (c == 7) ? 0 : 1;
  const long long plane_off = (long long)z * g.plane_r;
  const T* const pa = src + (long long)ca * g.nsite + plane_off;
  const T* const pb = zu ? zstar + plane_off : src + (long long)cb * g.nsite + plane_off;
  cplx<T>* const dst = spec + (long long)c * g.ncplx + (long long)z * g.plane_c;
  const int rows = h.NQ * Lx;  // elements between a group's rows
  // first x stage
  first_radix(h.R1, [&](auto radix) {
    constexpr int R = decltype(radix)::value;
#pragma unroll 1
    for (int t = tid; t < h.NQ * h.R2; t += nt) {
      const int q = fdiv(t, h.dR2), b = t - q * h.R2;
      const bool full = q + h.NQ * (2 * W - 1) < Ly, third = q + 2 * h.NQ < Ly;
      FG_SKIP_UNLESS(continue, group_in_range<R, W>(g, h, q, b));
      auto ld = [&](const T* r) {
        return CV<T>{vpack(r[0], W == 2 && third ? r[2 * rows] : (T)0),
                     vpack(W == 2 || full ? r[rows] : (T)0, W == 2 && full ? r[3 * rows] : (T)0)};
      };
      const T* r = pa + q * Lx + b;
      CV<T> v[R];
#pragma unroll
      for (int s = 0; s < R; ++s) v[s] = ld(r + s * h.R2);
      if (!plain) {
        const T* r2 = pb + q * Lx + b;
#pragma unroll
        for (int s = 0; s < R; ++s) {
          const CV<T> w = square ? v[s] : ld(r2 + s * h.R2);
          v[s] = CV<T>{vmul(v[s].re, w.re), vmul(v[s].im, w.im)};
        }
      }
      if (didi) sum += (double)cv_sum(v, R);
      DftV<T, R, false>::run(v);
      CV<T>* d = buf + q * h.QS + b;
      const lane_t<T> half = vall((T)0.5);
      cv_st(d, CV<T>{vmul(v[0].re, half), vmul(v[0].im, half)});
#pragma unroll
      for (int s = 1; s < R; ++s) cv_st(d + s * h.R2, cvtw<T, false>(v[s], tabx[s * b]));
    }
  });
  if (didi) plane_sum(sum, didi);
  __syncthreads();
  // second x stage with the separation of the rows
  second_radix(h.R2, [&](auto radix) {
    constexpr int R = decltype(radix)::value;
    const int al = fdiv(tid, h.dNQ), q = tid - al * h.NQ;
    const bool on = tid < (h.R1 / 2) * h.NQ FG_AND_CHECKED(classes_in_range<R, W>(g, h, q, al));
    const int a1 = al == 0 ? h.R1 / 2 : h.R1 - al;
    CV<T> v0[R], v1[R];
    if (on) {
      const CV<T>* r = buf + q * h.QS;
#pragma unroll
      for (int t = 0; t < R; ++t) v0[t] = cv_ld(r + al * R + t);
#pragma unroll
      for (int t = 0; t < R; ++t) v1[t] = cv_ld(r + a1 * R + t);
      DftV<T, R, false>::run(v0);
      DftV<T, R, false>::run(v1);
    }
    __syncthreads();
    if (on) {
      const bool full = q + h.NQ * (2 * W - 1) < Ly, third = q + 2 * h.NQ < Ly;
      class_columns<R>(v0, v1, al, a1, h.R1, [&](int k, const CV<T>& A, const CV<T>& B, bool dc) {
        T x0[2], x1[2];
        unpack_rows<0>(A, B, dc, x0, x1);
        *column_at<T>(buf, h.JS, k, q) = mk<cplx<T>>(x0[0], x0[1]);
        if (W == 2 || full) *column_at<T>(buf, h.JS, k, q + h.NQ) = mk<cplx<T>>(x1[0], x1[1]);
        if constexpr (W == 2) {
          unpack_rows<W - 1>(A, B, dc, x0, x1);
          if (third) *column_at<T>(buf, h.JS, k, q + 2 * h.NQ) = mk<cplx<T>>(x0[0], x0[1]);
          if (full) *column_at<T>(buf, h.JS, k, q + 3 * h.NQ) = mk<cplx<T>>(x1[0], x1[1]);
        }
      });
    }
  });
  __syncthreads();
  // first y stage
  first_radix(h.RY1, [&](auto radix) {
    constexpr int R = decltype(radix)::value;
#pragma unroll 1
    for (int t = tid; t < h.NJ * h.RY2; t += nt) {
      const int b = fdiv(t, h.dNJ), j = t - b * h.NJ;
      CV<T>* d = buf + j * h.JS + b;
      FG_SKIP_UNLESS(continue, fg_in_range(j * h.JS + b, j * h.JS + b + (R - 1) * h.RY2, h.smem / 16));
      CV<T> v[R];
#pragma unroll
      for (int s = 0; s < R; ++s) v[s] = cv_of(*reinterpret_cast<const rowvec<T>*>(d + s * h.RY2));
      DftV<T, R, false>::run(v);
      cv_st(d, v[0]);
#pragma unroll
      for (int s = 1; s < R; ++s) cv_st(d + s * h.RY2, cvtw<T, false>(v[s], taby[s * b]));
    }
  });
  __syncthreads();
  pdl_launch();
  // second y stage, to the spectrum rows; column 0 to shared memory first
  second_radix(h.RY2, [&](auto radix) {
    constexpr int R = decltype(radix)::value;
#pragma unroll 1
    for (int t = tid; t < h.NJ * h.RY1; t += nt) {
      const int a = fdiv(t, h.dNJ), j = t - a * h.NJ;
      const CV<T>* d = buf + j * h.JS + a * R;
      FG_SKIP_UNLESS(continue, column_in_range<R, W>(g, h, j, a));
      CV<T> v[R];
#pragma unroll
      for (int s = 0; s < R; ++s) v[s] = cv_ld(d + s);
      DftV<T, R, false>::run(v);
      cplx<T>* o = dst + (long long)(a * R) * g.KXP + W * j;
      if (j > 0 && W * j + W <= m) {
#pragma unroll
        for (int s = 0; s < R; ++s) cv_row(reinterpret_cast<rowvec<T>*>(o + (long long)s * g.KXP), v[s]);
      } else {
#pragma unroll
        for (int s = 0; s < R; ++s) {
          const cplx<T> x = mk<cplx<T>>(vget<0>(v[s].re), vget<0>(v[s].im));
          if (j == 0) col0[a * R + s] = x;
          else o[(long long)s * g.KXP] = x;
          if (W == 2 && W * j + 1 < m) o[(long long)s * g.KXP + 1] = mk<cplx<T>>(vget<W - 1>(v[s].re), vget<W - 1>(v[s].im));
        }
      }
    }
  });
  __syncthreads();
  const int *revy = posm + m, *posy = posm + m + Ly;
  for (int sl = tid; sl < Ly; sl += nt) {
    const int ky = __ldg(&revy[sl]), sp = __ldg(&posy[ky == 0 ? 0 : Ly - ky]);
    cplx<T> y0, ym;
    y_split(col0[sl], col0[sp], y0, ym);
    dst[(long long)sl * g.KXP] = y0;
    dst[(long long)sl * g.KXP + m] = ym;
  }
}

template <typename T>
__global__ void __launch_bounds__(512, 1)
    k_xy_inv_gen(const cplx<T>* __restrict__ spec, T* __restrict__ out, Geom g, XyGeo h, const cplx<T>* __restrict__ twx,
                 const cplx<T>* __restrict__ twy, const int* __restrict__ posm, const Phys* __restrict__ ph,
                 DevScalars* sc, const double* __restrict__ part_k, int nblk_k, const RepArgs* __restrict__ grp) {
  constexpr int W = kLanes<T>;
  pdl_wait();
  if (grp) {
    const RepArgs& a = grp[blockIdx.z];
    spec = (const cplx<T>*)a.spec;
    out = (T*)a.rwork;
    if (ph != nullptr) ph = a.ph;
    sc = a.sc;
    part_k = a.part_k;
  }
  if (ph != nullptr && blockIdx.y == 0) {  // as k_xy_inv
    if (blockIdx.x == 0) homo_strain_tail(ph, sc, part_k, nblk_k, grp && g.didi ? grp[blockIdx.z].didi : g.didi, g);
    return;
  }
  FG_DYN_SMEM(smem_raw);
  CV<T>* const buf = reinterpret_cast<CV<T>*>(smem_raw);
  __shared__ cplx<T> tabx[kLaneMax], taby[kLaneMax], col0[kLaneMax];
  const int nt = blockDim.x, tid = threadIdx.x;
  const int Lx = g.Lx, Ly = g.Ly, m = g.m;
  const int z = blockIdx.x, c = blockIdx.y - (ph != nullptr ? 1 : 0);
  const cplx<T>* const src = spec + (long long)c * g.ncplx + (long long)z * g.plane_c;
  T* const dst = out + (long long)c * g.nsite + (long long)z * g.plane_r;
  const unsigned long long pol = l2_evict_first();
  auto ldc = [&](const cplx<T>* a) {
    if constexpr (sizeof(T) == 4 || FG_L2_HINT_FP64) return ld_first(a, pol);
    else return *a;
  };
  const int *revy = posm + m, *posy = posm + m + Ly;
  for (int sl = tid; sl < Ly; sl += nt) {
    const int ky = __ldg(&revy[sl]), sp = __ldg(&posy[ky == 0 ? 0 : Ly - ky]);
    const cplx<T>*r = src + (long long)sl * g.KXP, *rm = src + (long long)sp * g.KXP;
    col0[sl] = y_join(ldc(r), ldc(rm), ldc(r + m), ldc(rm + m));
  }
  for (int k = tid; k < Lx; k += nt) tabx[k] = twx[k];
  for (int k = tid; k < Ly; k += nt) taby[k] = twy[k];
  __syncthreads();
  second_radix(h.RY2, [&](auto radix) {
    constexpr int R = decltype(radix)::value;
#pragma unroll 1
    for (int t = tid; t < h.NJ * h.RY1; t += nt) {
      const int a = fdiv(t, h.dNJ), j = t - a * h.NJ;
      const cplx<T>* r = src + (long long)(a * R) * g.KXP + W * j;
      FG_SKIP_UNLESS(continue, column_in_range<R, W>(g, h, j, a));
      CV<T> v[R];
#pragma unroll
      for (int s = 0; s < R; ++s) {
        if constexpr (sizeof(T) == 4) v[s] = cv_of(ld_first(reinterpret_cast<const float4*>(r + (long long)s * g.KXP), pol));
        else v[s] = cv_of(ldc(r + (long long)s * g.KXP));
      }
      if (j == 0) {
#pragma unroll
        for (int s = 0; s < R; ++s) {
          const cplx<T> x = col0[a * R + s];
          v[s] = CV<T>{vpack(x.x, vget<W - 1>(v[s].re)), vpack(x.y, vget<W - 1>(v[s].im))};
        }
      }
      DftV<T, R, true>::run(v);
      CV<T>* d = buf + j * h.JS + a * R;
#pragma unroll
      for (int s = 0; s < R; ++s) cv_st(d + s, v[s]);
    }
  });
  __syncthreads();
  first_radix(h.RY1, [&](auto radix) {
    constexpr int R = decltype(radix)::value;
#pragma unroll 1
    for (int t = tid; t < h.NJ * h.RY2; t += nt) {
      const int b = fdiv(t, h.dNJ), j = t - b * h.NJ;
      CV<T>* d = buf + j * h.JS + b;
      FG_SKIP_UNLESS(continue, fg_in_range(j * h.JS + b, j * h.JS + b + (R - 1) * h.RY2, h.smem / 16));
      CV<T> v[R];
      v[0] = cv_ld(d);
#pragma unroll
      for (int s = 1; s < R; ++s) v[s] = cvtw<T, true>(cv_ld(d + s * h.RY2), taby[s * b]);
      DftV<T, R, true>::run(v);
#pragma unroll
      for (int s = 0; s < R; ++s) cv_row(reinterpret_cast<rowvec<T>*>(d + s * h.RY2), v[s]);
    }
  });
  __syncthreads();
  second_radix(h.R2, [&](auto radix) {
    constexpr int R = decltype(radix)::value;
    const int al = fdiv(tid, h.dNQ), q = tid - al * h.NQ;
    const bool on = tid < (h.R1 / 2) * h.NQ FG_AND_CHECKED(classes_in_range<R, W>(g, h, q, al));
    const int a1 = al == 0 ? h.R1 / 2 : h.R1 - al;
    CV<T> v0[R], v1[R];
    if (on) {
      const bool full = q + h.NQ * (2 * W - 1) < Ly, third = q + 2 * h.NQ < Ly;
      class_columns<R>(v0, v1, al, a1, h.R1, [&](int k, CV<T>& A, CV<T>& B, bool dc) {
        T p[2][2], n[2][2];
#pragma unroll
        for (int l = 0; l < W; ++l) {
          const cplx<T> zero = mk<cplx<T>>((T)0, (T)0);
          const cplx<T> x = l == 0 || third ? *column_at<T>(buf, h.JS, k, q + 2 * l * h.NQ) : zero;
          const cplx<T> y = l < W - 1 || full ? *column_at<T>(buf, h.JS, k, q + (2 * l + 1) * h.NQ) : zero;
          const T x0[2] = {x.x, x.y}, x1[2] = {y.x, y.y};
          pack_rows(x0, x1, dc, p[l], n[l]);
        }
        A = CV<T>{vpack(p[0][0], p[W - 1][0]), vpack(p[0][1], p[W - 1][1])};
        B = CV<T>{vpack(n[0][0], n[W - 1][0]), vpack(n[0][1], n[W - 1][1])};
      });
      DftV<T, R, true>::run(v0);
      DftV<T, R, true>::run(v1);
    }
    __syncthreads();
    if (on) {
      CV<T>* r = buf + q * h.QS;
#pragma unroll
      for (int t = 0; t < R; ++t) cv_st(r + al * R + t, v0[t]);
#pragma unroll
      for (int t = 0; t < R; ++t) cv_st(r + a1 * R + t, v1[t]);
    }
  });
  __syncthreads();
  pdl_launch();
  const int rows = h.NQ * Lx;
  first_radix(h.R1, [&](auto radix) {
    constexpr int R = decltype(radix)::value;
#pragma unroll 1
    for (int t = tid; t < h.NQ * h.R2; t += nt) {
      const int q = fdiv(t, h.dR2), b = t - q * h.R2;
      const bool full = q + h.NQ * (2 * W - 1) < Ly, third = q + 2 * h.NQ < Ly;
      const CV<T>* d = buf + q * h.QS + b;
      FG_SKIP_UNLESS(continue, group_in_range<R, W>(g, h, q, b));
      CV<T> v[R];
      v[0] = cv_ld(d);
#pragma unroll
      for (int s = 1; s < R; ++s) v[s] = cvtw<T, true>(cv_ld(d + s * h.R2), tabx[s * b]);
      DftV<T, R, true>::run(v);
      T* r = dst + q * Lx + b;
#pragma unroll
      for (int s = 0; s < R; ++s) {
        T* o = r + s * h.R2;
        o[0] = vget<0>(v[s].re);
        if (W == 2 || full) o[rows] = vget<0>(v[s].im);
        if constexpr (W == 2) {
          if (third) o[2 * rows] = vget<W - 1>(v[s].re);
          if (full) o[3 * rows] = vget<W - 1>(v[s].im);
        }
      }
    }
  });
}

// ------------------------------------------------- z tiles (shared helpers)
// A z tile is CW pencils (kx slot, ky slot) with all z, nc components, held
// in shared memory as buf[c][z][cw].  Blocks [0, nreg) take CW consecutive kx
// slots of one ky slot (CW divides Lx/2); blocks [nreg, nreg + nnyq) take
// the Nyquist slot kx = Lx/2 of CW consecutive ky slots.
struct ZTiles {
  int CW;
  int ntx;   // regular tiles per ky slot (= (Lx/2) / CW)
  int nreg;  // ntx * Ly
  int nnyq;  // ceil(Ly / CW)
};

// Blocks 0 .. nnyq-1 take the Nyquist tiles (kx = Lx/2 batched across ky,
// one uncoalesced 8-byte access per element), the rest the regular tiles:
// the slow tiles start first instead of trailing the grid.
__device__ __forceinline__ bool tile_pencil(const ZTiles& zt, const Geom& g, int cw, int* col, int* yslot) {
  const int b = blockIdx.x;
  if (b >= zt.nnyq) {
    const int r = b - zt.nnyq;
    *yslot = r / zt.ntx;
    *col = (r - *yslot * zt.ntx) * zt.CW + cw;
    return true;
  }
  *col = g.m;
  *yslot = b * zt.CW + cw;
  return *yslot < g.Ly;
}

// Threads own a fixed pencil cw = threadIdx.x % CW (blockDim is a multiple
// of CW) and walk the tile rows r = c * Lz + z, so the pencil decode runs
// once per thread and a row step is an add.  buf[r * CW + cw].
template <typename T, int LZC = 0, int CWC = 0>
__device__ __forceinline__ void z_tile_load(cplx<T>* buf, const cplx<T>* __restrict__ spec, const Geom& g,
                                            const ZTiles& zt, int nc) {
  const int Lz = LZC > 0 ? LZC : g.Lz, CW = CWC > 0 ? CWC : zt.CW;
  const int cw = threadIdx.x % CW, rstep = blockDim.x / CW;
  int col, yslot;
  const bool valid = tile_pencil(zt, g, cw, &col, &yslot);
  const cplx<T>* base = spec + (valid ? (long long)yslot * g.KXP + col : 0);
  for (int r = threadIdx.x / CW; r < nc * Lz; r += rstep) {
    const int c = r / Lz, z = r - c * Lz;
    cplx<T>* dst = &buf[r * CW + cw];
    if (valid) cp_async<(int)sizeof(cplx<T>)>(dst, base + (long long)c * g.ncplx + (long long)z * g.plane_c);
    else *dst = mk<cplx<T>>((T)0, (T)0);
  }
  cp_async_wait();
  __syncthreads();
}

template <typename T, int LZC = 0, int CWC = 0>
__device__ __forceinline__ void z_tile_store(const cplx<T>* buf, cplx<T>* __restrict__ spec, const Geom& g,
                                             const ZTiles& zt, int nc) {
  const int Lz = LZC > 0 ? LZC : g.Lz, CW = CWC > 0 ? CWC : zt.CW;
  const int cw = threadIdx.x % CW, rstep = blockDim.x / CW;
  int col, yslot;
  if (!tile_pencil(zt, g, cw, &col, &yslot)) return;
  cplx<T>* base = spec + (long long)yslot * g.KXP + col;
  for (int r = threadIdx.x / CW; r < nc * Lz; r += rstep) {
    const int c = r / Lz, z = r - c * Lz;
    base[(long long)c * g.ncplx + (long long)z * g.plane_c] = buf[r * CW + cw];
  }
}

// Value q of the dipole table at position pos = (ky slot, kz slot, kx slot):
// the 6 values of W neighbouring kx slots interleaved, [pos / W][6][W], as the
// elements of k_z_lane read them (KXP is even).
template <typename T>
__host__ __device__ __forceinline__ long long tab_index(long long pos, int q) {
  constexpr int W = 16 / (2 * (int)sizeof(T));
  return (pos & ~(long long)(W - 1)) * 6 + q * W + (pos & (W - 1));
}

// ------------------------------------------------------------ scalar kernels
// Grid-wide scalar steps; each runs either as a single-block kernel or in the
// last block of the kernel whose partial sums it reduces (tail).
enum { TAIL_NONE = 0, TAIL_ENERGIES = 1, TAIL_LF_FINAL = 3, TAIL_VS = 4, TAIL_VS_ACOU = 6 };

__device__ __forceinline__ double sum_potential(const double* e) {
  return e[E_SHORT] + e[E_LONG] + e[E_DIPE] + e[E_UNH] + e[E_HS] + e[E_HC] + e[E_IS] + e[E_IC] + e[E_IM];
}

// energy_module.F:128-148 with 1/s^2 and log(s) of the current s given
__device__ __forceinline__ void np_hamiltonian(const Phys* ph, DevScalars* sc, double inv_s2, double log_s) {
  double* e = sc->e;
  double h = e[E_DIPO] * inv_s2 + sum_potential(e) + sc->pi * sc->pi * 0.5 * ph->Qinv + ph->threeN_kT * log_s - sc->H0;
  e[E_HNP] = h * sc->s;
}
__device__ __forceinline__ void np_hamiltonian(const Phys* ph, DevScalars* sc) {
  const double inv_s = 1.0 / sc->s;
  np_hamiltonian(ph, sc, inv_s * inv_s, log(sc->s));
}

__device__ __forceinline__ void check_finite(DevScalars* sc, const double* v, int n) {
  for (int i = 0; i < n; ++i)
    if (!isfinite(v[i])) sc->status = 3;  // FG_ERR_NAN
}

// After the k-space pass: k-space energies, homogeneous strain
// (optimize-homo-strain.F:27-186) and w_hom for k_assemble.
__device__ __noinline__ void homo_strain_tail(const Phys* __restrict__ ph, DevScalars* sc,
                                              const double* __restrict__ part_k, int nblk,
                                              const double* __restrict__ didi, const Geom g) {
  // On one warp: lane i has row i of the products, every lane the energies and
  // the triangular solves; stores at the end, so that all loads go ahead of
  // the chain.
  reduced_tail<NQ_K, 9, 32>(ph, sc, part_k, didi, nblk, didi ? g.didi_rows : 0,
                            [&](const Phys* P, DevScalars* S, const double* v) {
    double es = v[0], edd = v[1];
    if (g.k0_exact) {  // S(0) has no off-diagonal entries
      const double* U = v + NQ_K;
      const double one[3] = {1.0, 1.0, 1.0}, zero[3] = {0.0, 0.0, 0.0};
      double S0[6];
      short_range_k(P->j, P->kap2x2, one, zero, S0);
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const int b = (a + 1) % 3, c = (a + 2) % 3;  // off-diagonal slots: yz 3, zx 4, xy 5
        es += S0[a] * (U[a] * U[a]);
        edd += S->D0[a] * (U[a] * U[a]) + 2 * S->D0[3 + a] * (U[b] * U[c]);
      }
    }
    es = es * P->Ninv / 2;  // (1/2N) sum w' Re(uK* S uK)
    edd = edd / 2;          // (1/2)  sum w' Re(uK* D uK), D = (S + Z*^2 L)/N
    const int i = threadIdx.x % 6;
    const double* dd = didi ? v + NQ_K + 3 : S->didiK0;
    double d[6], hcol[6], hrow[6], hc2uu[6], st[6];
    double t = 0.0;
#pragma unroll
    for (int j = 0; j < 6; ++j) {
      d[j] = dd[j];
      hcol[j] = P->HC2[j][i];
      hrow[j] = P->H[i][j];
      t += P->HC2[i][j] * d[j];
    }
    if (i < 3) t += P->pNa03[i];
#pragma unroll
    for (int j = 0; j < 6; ++j) hc2uu[j] = lane_value(t, j);
    const double(*H)[6] = P->H;
    if (P->bulk_or_film == 2) {  // epit
      st[0] = P->epi_strain;
      st[1] = P->epi_strain;
      st[2] = (-(H[2][0] + H[2][1]) * P->epi_strain - hc2uu[2]) / H[2][2];
      st[3] = -hc2uu[3] / H[3][3];
      st[4] = -hc2uu[4] / H[4][4];
      st[5] = 0.0;
    } else if (P->bulk_or_film == 3) {  // e110
      st[2] = P->epi_strain;
      st[3] = 0.0;
      st[4] = 0.0;
      double num = -(H[0][0] + H[1][1] + 2 * H[1][1]) * P->epi_strain - (H[2][0] + H[2][1]) * st[2] - hc2uu[0] -
                   hc2uu[1] + 2 * hc2uu[5];
      double den = H[0][0] + H[1][1] + 2 * H[1][0] + 4 * H[5][5];
      double delta = num / den;
      st[0] = P->epi_strain + delta;
      st[1] = P->epi_strain + delta;
      st[5] = -2 * delta;
    } else {
#pragma unroll
      for (int r = 0; r < 6; ++r) {
        double x = 0.0;
#pragma unroll
        for (int c = 0; c < r; ++c) x = x + P->HG[r][c] * st[c];
        st[r] = (-hc2uu[r] - x) * P->HG_inv[r];
      }
#pragma unroll
      for (int r = 5; r >= 0; --r) {
        double x = 0.0;
#pragma unroll
        for (int c = r + 1; c < 6; ++c) x = x + st[c] * P->HG[c][r];
        st[r] = (st[r] - x) * P->HG_inv[r];
      }
    }
    double hd = 0.0, w = 0.0, hs = 0.0, hc = 0.0;
#pragma unroll
    for (int j = 0; j < 6; ++j) {
      hd += hrow[j] * st[j];
      w = w + st[j] * hcol[j];
      hc += st[j] * hc2uu[j];
    }
#pragma unroll
    for (int j = 0; j < 6; ++j) hs = hs + st[j] * lane_value(hd, j);
    if (threadIdx.x < 6) S->w_hom[threadIdx.x] = w;
    if (threadIdx.x == 0) {
      S->e[E_SHORT] = es;
      S->e[E_LONG] = edd - es;
      S->e[E_IS] = v[2] * P->Ninv;
      S->e[E_IC] = v[3] * 2 * P->Ninv;
      S->e[E_IM] = P->modulation_on ? v[4] * 2 * P->Ninv : 0.0;
      S->e[E_HS] = hs / 2;
      S->e[E_HC] = hc;
#pragma unroll
      for (int j = 0; j < 6; ++j) {
        S->strain[j] = st[j];
        S->didiK0[j] = d[j];
      }
    }
  });
}

// kinetic_energy_dipo.F:106 from the kick partials
__device__ __forceinline__ double ke_from(const Phys* ph, double sum) { return sum * ph->ke_scale; }

// After k_assemble: real-space energies from the totals v of its partials.
__device__ __forceinline__ void force_energies_body(const Phys* P, DevScalars* S, const double* v) {
  S->e[E_UNH] = v[0];
  S->e[E_DIPE] = P->E_on ? -v[1] : 0.0;
  check_finite(S, S->e + E_SHORT, 9);
}
// A Nose-Poincare step after its force (nose-poincare.F:60-66): the commit of
// the prepared half step ((38), (35c): s, pi, KE at the half step), H_NP and
// the (35e) update of pi.
__device__ __forceinline__ void np_post_body(const Phys* P, DevScalars* S, double inv_s, double log_s) {
  S->s_old = S->s;
  S->s = S->pend_s;
  S->pi = S->pend_pi;
  S->ke_sum = S->pend_ke_sum;
  S->e[E_DIPO] = S->pend_ke;
  S->drift_coef = S->pend_drift;
  const double inv_s2 = inv_s * inv_s;
  np_hamiltonian(P, S, inv_s2, log_s);
  const double delta_H = S->e[E_HNP] * inv_s;
  S->pi = S->pi + P->dt_2 * (2 * S->e[E_DIPO] * inv_s2 - P->nf_kT) - P->dt_2 * delta_H;
}
// End of a Nose-Poincare step from the masked sums v of p^2/m, p.F/m and
// F^2/m after the closing kick (35f).
//  - step_done: KE, H_NP and total of the finished step (nose-poincare.F:
//    74-75, molecular-dynamics.F:293);
//  - always: the first half of the next step (nose-poincare.F:24-41) as far
//    as it is scalar: its kick (35a) p - c F with c = dt/2 s has the kinetic
//    sum  sum p^2/m - 2 c sum p.F/m + c^2 sum F^2/m,  which gives (38) pi,
//    s_{n+1} and the drift coefficient of (35c) before any site is touched.
//    They are kept pending (s and pi still report the finished step).
// One thread's serial FP64 chain: three divisions and a square root.
__device__ __forceinline__ void np_close_body(const Phys* P, DevScalars* S, const double* v, double inv_s, double log_s,
                                              bool step_done) {
  const double s = S->s, inv_s2 = inv_s * inv_s;
  const double epot = sum_potential(S->e);
  if (step_done) {
    S->ke_sum = v[0];
    S->e[E_DIPO] = ke_from(P, v[0]);
    np_hamiltonian(P, S, inv_s2, log_s);
    S->e[E_TOT] = S->e[E_DIPO] * inv_s2 + S->e[E_ACOU] + epot;
    check_finite(S, S->e, E_COUNT);
  }
  const double ca = P->dt_2 * s;
  const double kh = v[0] - 2 * ca * v[1] + ca * ca * v[2];
  const double ke = ke_from(P, kh);
  double CB = P->nf_kT * (1.0 + log_s) - ke * inv_s2 + epot - S->H0;
  CB = P->dt_2 * CB - S->pi;
  const double r = CB * P->dt * P->Qinv;
  if (1.0 - r < 0.0) S->status = 10;  // (38) has no real root: Q_Nose too small
  const double pih = -2 * CB / (1.0 + sqrt(1.0 - r));
  const double a = P->dt_2 * pih * P->Qinv;
  const double sn = s * (1.0 + a) / (1.0 - a);
  S->kick_coef = ca;
  S->pend_ke_sum = kh;
  S->pend_ke = ke;
  S->pend_pi = pih;
  S->pend_s = sn;
  S->pend_drift = P->dt_2 * (1.0 / sn + inv_s);
  S->pend_kick_f = P->dt_2 * sn;
}

__device__ __noinline__ void force_energies_tail(const Phys* __restrict__ ph, DevScalars* sc,
                                                 const double* __restrict__ part_r, int nblk, bool np_close,
                                                 DevScalars* host = nullptr) {
  reduced_tail<NQ_R, 0>(ph, sc, part_r, nullptr, nblk, 0, [&](const Phys* P, DevScalars* S, const double* v) {
    force_energies_body(P, S, v);
    if (np_close) np_post_body(P, S, 1.0 / S->pend_s, log(S->pend_s));
  }, host);
}
__device__ __noinline__ void np_close_tail(const Phys* __restrict__ ph, DevScalars* sc,
                                           const double* __restrict__ part, int nblk, bool step_done,
                                           DevScalars* host) {
  reduced_tail<3, 0>(ph, sc, part, nullptr, nblk, 0, [&](const Phys* P, DevScalars* S, const double* v) {
    np_close_body(P, S, v, 1.0 / S->s, log(S->s), step_done);
  }, host);
}
// Both for k_assemble with the fused closing kick, in one tail.
__device__ __noinline__ void np_step_tail(const Phys* __restrict__ ph, DevScalars* sc,
                                          const double* __restrict__ part_r, const double* __restrict__ part_ke,
                                          int nblk, DevScalars* host) {
  reduced_tail<NQ_R, 3>(ph, sc, part_r, part_ke, nblk, nblk, [&](const Phys* P, DevScalars* S, const double* v) {
    const double inv_s = 1.0 / S->pend_s, log_s = log(S->pend_s);
    force_energies_body(P, S, v);
    np_post_body(P, S, inv_s, log_s);
    np_close_body(P, S, v + NQ_R, inv_s, log_s, true);
  }, host);
}

// Velocity scaling (velocity_scaling.F:74-83): kinetic energy of the kicked
// momenta, the factor sqrt(target / KE) for k_scale, total.  The reported
// dipo_kinetic is the value before rescaling, as in the reference.
__device__ void vs_tail(const Phys* __restrict__ ph, DevScalars* sc, const double* __restrict__ part, int nblk) {
  reduced_tail<1, 0>(ph, sc, part, nullptr, nblk, 0, [&](const Phys* P, DevScalars* S, const double* v) {
    S->ke_sum = v[0];
    S->e[E_DIPO] = ke_from(P, v[0]);
    S->vs_scale = sqrt(P->target_ke / S->e[E_DIPO]);
    S->e[E_TOT] = S->e[E_DIPO] / (S->s * S->s) + S->e[E_ACOU] + sum_potential(S->e);
    check_finite(S, S->e, E_COUNT);
    if (!isfinite(S->vs_scale)) S->status = 3;
  });
}

// Acoustic kinetic energy sum acouP^2 / m / 2 (kinetic_energy_acou.F:15-27);
// the rescale factor (velocity_scaling.F:86-98) and the total.
__device__ void acou_tail(const Phys* __restrict__ ph, DevScalars* sc, const double* __restrict__ part, int nblk) {
  reduced_tail<1, 0>(ph, sc, part, nullptr, nblk, 0, [&](const Phys* P, DevScalars* S, const double* v) {
    S->e[E_ACOU] = v[0] / 2;
    S->vs_scale_acou = sqrt(P->target_ke / S->e[E_ACOU]);
    if (!isfinite(S->vs_scale_acou)) S->status = 3;
    S->e[E_TOT] = S->e[E_DIPO] / (S->s * S->s) + S->e[E_ACOU] + sum_potential(S->e);
  });
}

// Leapfrog closing reduction (leapfrog.F:151) and total; part_acou: the
// acoustic field's sums as well (null without one).
__device__ __forceinline__ void lf_final_body(const Phys* P, DevScalars* S, double sum) {
  S->ke_sum = sum;
  S->e[E_DIPO] = ke_from(P, sum);
  S->e[E_TOT] = S->e[E_DIPO] / (S->s * S->s) + S->e[E_ACOU] + sum_potential(S->e);
  check_finite(S, S->e, E_COUNT);
}
__device__ void lf_final_tail(const Phys* __restrict__ ph, DevScalars* sc, const double* __restrict__ part,
                              const double* __restrict__ part_acou, int nblk) {
  reduced_tail<1, 1>(ph, sc, part, part_acou, nblk, part_acou ? nblk : 0,
                     [&](const Phys* P, DevScalars* S, const double* v) {
                       if (part_acou) S->e[E_ACOU] = v[1] / 2;
                       lf_final_body(P, S, v[0]);
                     });
}

// Wavevectors, trig tables and slot maps shared by the k-space kernels.
struct KMaps {
  const int* revx;     // kx slot -> kx
  const int* revy;     // ky slot -> ky
  const int* revz;     // kz slot -> kz
  const double* kvx;   // k(1) of elastic.F:87 per kx
  const double* kvy;   // k(2) per ky (wrapped to (-1/2, 1/2])
  const double* kvz;   // k(3) per kz
  const double2* trx;  // (cos, sin)(2 pi kx / Lx)
  const double2* try_;
  const double2* trz;
  const double2* trz_s;  // trz and kvz in kz-slot order (no revz lookup first)
  const double* kvz_s;
  const double2* trx_s;  // the same of x (slots 0 .. Lx/2) and y
  const double2* try_s;
  const double* kvx_s;
  const double* kvy_s;
};

// Plain z pass of nc spectra in place: DIF (INV = false) or DIT (INV = true).
// LZC, CWC, NCC > 0: compile-time transforms for Lz = LZC, tile width CWC
// and NCC components (launched with exactly kZThreads threads); 0 = runtime.
template <typename T, bool INV, int LZC = 0, int CWC = 0, int NCC = 0>
__global__ void __launch_bounds__(256) k_z_pass(cplx<T>* __restrict__ spec, Geom g, FftPlan pz,
                                                const cplx<T>* __restrict__ twz, int nc, ZTiles zt) {
  FG_DYN_SMEM(smem_raw);
  cplx<T>* buf = reinterpret_cast<cplx<T>*>(smem_raw);
  if constexpr (LZC > 0) {
    __shared__ cplx<T> tws[LZC];
    for (int i = threadIdx.x; i < LZC; i += blockDim.x) tws[i] = twz[i];
    z_tile_load<T, LZC, CWC>(buf, spec, g, zt, NCC);
    using B = BatchCT<NCC * CWC, CWC, 1, LZC * CWC, CWC>;
    if (INV) ct_inverse<T, LZC, 256, B>(buf, tws);
    else ct_forward<T, LZC, 256, B>(buf, tws);
    z_tile_store<T, LZC, CWC>(buf, spec, g, zt, NCC);
  } else {
    const int CW = zt.CW;
    z_tile_load<T>(buf, spec, g, zt, nc);
    Batch B{nc * CW, CW, 1, g.Lz * CW, CW, true};
    if (INV) fft_inverse<T>(buf, B, pz, twz, nc * g.Lz * CW);
    else fft_forward<T>(buf, B, pz, twz, nc * g.Lz * CW);
    z_tile_store<T>(buf, spec, g, zt, nc);
  }
}

// ------------------------------------------------------------------ k_z_kspace
// Per (kx tile, ky slot): DIF along z of the nine spectra, then for every k
//   F(k)     = D(k) uK(k),  D = (S + Z*^2 L)/N   (dVddi-dipole-dipole.F:20-36)
//   acouK(k) = -K(k)^-1 (c_k_mod + coup2(k) didiK(k))  (optimize-inho-strain.F:28-58)
//   inhoK(k) = k (x) acouK / N                        (dVddi_inho_coupling.F:91-108)
// with K, its Cholesky factor and coup2 evaluated analytically
// (elastic.F:79-180), and the half-spectrum energy sums of
// dVddi-dipole-dipole.F:226-250 (by Parseval) and energy_module.F:150-240;
// then DIT along z.  Slots 0..2 return F(k), slots 3..8 inhoK(k).
// ZSC (per-site Z*, dVddi-dipole-dipole.F:20-60): slots Z0..Z0+2 carry
// FFT(Z*(R) u) in and the long-range part (L/N) FFT(Z* u) out, while slots
// 0..2 return the short-range part (S/N) uK alone; L/N comes from ltab.
constexpr int kZThreads = 256;

template <typename T, bool ACOU = false, bool ZSC = false>
__global__ void __launch_bounds__(256, 2) k_z_kspace(cplx<T>* __restrict__ spec, const T* __restrict__ dtab,
                                                     const cplx<T>* __restrict__ ckmod, cplx<T>* __restrict__ acouK_out,
                                                     Geom g, FftPlan pz, const cplx<T>* __restrict__ twz, KMaps km,
                                                     const Phys* __restrict__ ph, double* __restrict__ part,
                                                     DevScalars* sc, ZTiles zt, const T* __restrict__ ltab,
                                                     const RepArgs* __restrict__ grp = nullptr) {
  pdl_wait();
  if (grp) {
    const RepArgs& a = grp[blockIdx.y];
    spec = (cplx<T>*)a.spec;
    dtab = (const T*)a.dtab;
    ph = a.ph;
    part = a.part_k;
    sc = a.sc;
  }
  FG_DYN_SMEM(smem_raw);
  cplx<T>* buf = reinterpret_cast<cplx<T>*>(smem_raw);
  const int Lz = g.Lz, CW = zt.CW;
  // ACOU: acoustic-displacement MD, three more components in and out
  // (FFT(acouR) in, dVdacK out; acouFFT.F:9-26, dVdac.F:11-63)
  constexpr int Z0 = ACOU ? 12 : 9;  // first Z* u slot (ZSC)
  constexpr int NC = Z0 + (ZSC ? 3 : 0);
  const int buf_len = NC * Lz * CW;
  const int ZS = Lz * CW;  // component stride of the tile
  const int cwp = threadIdx.x % CW;
  int colp = 0, ysp = 0;
  const bool okp = tile_pencil(zt, g, cwp, &colp, &ysp);
  z_tile_load<T>(buf, spec, g, zt, NC);
  const Batch B{NC * CW, CW, 1, Lz * CW, CW, true};
  fft_forward<T>(buf, B, pz, twz, buf_len);
  const double Ninv = ph->Ninv;
  // Energy sums: the per-k products in T (FP32 in the mixed path, whose
  // spectra are FP32), accumulated per thread in FP64
  double acc[NQ_K] = {0, 0, 0, 0, 0};
  // this thread's pencil (fixed cw), decoded once
  const int cw = cwp, col = colp, yslot = ysp;
  const bool pencil_ok = okp;
  const int ky = pencil_ok ? __ldg(&km.revy[yslot]) : 0;
  const int kx = pencil_ok ? __ldg(&km.revx[col]) : 0;
  const double kv2 = __ldg(&km.kvy[ky]);
  const double2 ty = __ldg(&km.try_[ky]);
  const double2 tx = __ldg(&km.trx[kx]);
  const double kv1 = __ldg(&km.kvx[kx]);
  // S(k) of short_range_k along this pencil: with c = cos, s = sin of the
  // x, y and z phases, S_aa = A_a + B_a cz, S_yz = C_3 sz, S_zx = C_4 sz,
  // S_xy = A_5 + B_5 cz (the x-y parts fixed per pencil, FP64)
  double sA[6], sB[6];
  {
    const double* j = ph->j;
    const double kap = ph->kap2x2, c0 = tx.x, c1 = ty.x, s0 = tx.y, s1 = ty.y;
    sA[0] = kap + 2 * j[1] * c0 + 2 * j[0] * c1 + 4 * j[2] * c0 * c1;
    sB[0] = 2 * j[0] + 4 * j[3] * c1 + 4 * j[2] * c0 + 8 * j[5] * c0 * c1;
    sA[1] = kap + 2 * j[1] * c1 + 2 * j[0] * c0 + 4 * j[2] * c1 * c0;
    sB[1] = 2 * j[0] + 4 * j[3] * c0 + 4 * j[2] * c1 + 8 * j[5] * c0 * c1;
    sA[2] = kap + 2 * j[0] * (c0 + c1) + 4 * j[3] * c0 * c1;
    sB[2] = 2 * j[1] + 4 * j[2] * (c0 + c1) + 8 * j[5] * c0 * c1;
    sA[3] = 0.0;
    sB[3] = -4 * j[4] * s1 - 8 * j[6] * s1 * c0;  // times sz
    sA[4] = 0.0;
    sB[4] = -4 * j[4] * s0 - 8 * j[6] * s0 * c1;  // times sz
    sA[5] = -4 * j[4] * s0 * s1;
    sB[5] = -8 * j[6] * s0 * s1;
  }
  const T w1 = (kx == 0 || kx == g.m) ? (T)1 : (T)2;  // full-spectrum multiplicity
  const long long tpos0 = (long long)yslot * Lz * g.KXP + col;
  for (int zs = threadIdx.x / CW; pencil_ok && zs < Lz; zs += blockDim.x / CW) {
    cplx<T> u[3], d[6];
#pragma unroll
    for (int a = 0; a < 3; ++a) u[a] = buf[a * ZS + zs * CW + cw];
#pragma unroll
    for (int i = 0; i < 6; ++i) d[i] = buf[(3 + i) * ZS + zs * CW + cw];
    const bool k0 = kx == 0 && ky == 0 && zs == 0;  // slot 0 holds kz = 0
    if (k0) {
#pragma unroll
      for (int i = 0; i < 6; ++i) sc->didiK0[i] = (double)d[i].x;
      __threadfence();  // read by homo_strain_tail in another block
    }
    // ---- dipole-dipole
    const long long tpos = tpos0 + (long long)zs * g.KXP;
    T D[6];  // D = (S + Z*^2 L)/N; ZSC: L/N
#pragma unroll
    for (int q = 0; q < 6; ++q) D[q] = __ldg((ZSC ? ltab : dtab) + tab_index<T>(tpos, q));
    T qv[6];  // Re(conj(u_a) u_b): xx, yy, zz, yz, zx, xy
    qv[0] = u[0].x * u[0].x + u[0].y * u[0].y;
    qv[1] = u[1].x * u[1].x + u[1].y * u[1].y;
    qv[2] = u[2].x * u[2].x + u[2].y * u[2].y;
    qv[3] = u[1].x * u[2].x + u[1].y * u[2].y;
    qv[4] = u[2].x * u[0].x + u[2].y * u[0].y;
    qv[5] = u[0].x * u[1].x + u[0].y * u[1].y;
    {
      // short- and total dipole energies in FP64 from the same qv, so that
      // their difference (the long-range energy) keeps its digits
      const double2 tz = __ldg(&km.trz_s[zs]);
      double S[6];
      S[0] = sA[0] + sB[0] * tz.x;
      S[1] = sA[1] + sB[1] * tz.x;
      S[2] = sA[2] + sB[2] * tz.x;
      S[3] = sB[3] * tz.y;
      S[4] = sB[4] * tz.y;
      S[5] = sA[5] + sB[5] * tz.x;
      double qd[6];
#pragma unroll
      for (int q = 0; q < 6; ++q) qd[q] = (double)qv[q];
      const bool tail_k0 = !ZSC && k0 && g.k0_exact;
      if (tail_k0) {
#pragma unroll
        for (int q = 0; q < 6; ++q) sc->D0[q] = (double)D[q];
      }
      const double we = tail_k0 ? 0.0 : (double)w1;
      const double es = we * (S[0] * qd[0] + S[1] * qd[1] + S[2] * qd[2] + 2.0 * (S[3] * qd[3] + S[4] * qd[4] + S[5] * qd[5]));
      acc[0] += es;
      if constexpr (ZSC) {
        // short range on uK, long range on FFT(Z* u): Fl = (L/N) ZuK,
        // energy (1/2N) sum w' Re(ZuK* L ZuK) by Parseval
        cplx<T> zu[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) zu[a] = buf[(Z0 + a) * ZS + zs * CW + cw];
        T qz[6];
        qz[0] = zu[0].x * zu[0].x + zu[0].y * zu[0].y;
        qz[1] = zu[1].x * zu[1].x + zu[1].y * zu[1].y;
        qz[2] = zu[2].x * zu[2].x + zu[2].y * zu[2].y;
        qz[3] = zu[1].x * zu[2].x + zu[1].y * zu[2].y;
        qz[4] = zu[2].x * zu[0].x + zu[2].y * zu[0].y;
        qz[5] = zu[0].x * zu[1].x + zu[0].y * zu[1].y;
        acc[1] += es * Ninv + (double)w1 * ((double)D[0] * qz[0] + (double)D[1] * qz[1] + (double)D[2] * qz[2] +
                                            2.0 * ((double)D[3] * qz[3] + (double)D[4] * qz[4] + (double)D[5] * qz[5]));
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const int b = (a + 1) % 3, c3 = (a + 2) % 3;  // off-diagonal slots: yz 3, zx 4, xy 5
          const T dab = D[a == 0 ? 5 : a == 1 ? 3 : 4], dac = D[a == 0 ? 4 : a == 1 ? 5 : 3];
          buf[(Z0 + a) * ZS + zs * CW + cw] =
              mk<cplx<T>>(D[a] * zu[a].x + dab * zu[b].x + dac * zu[c3].x, D[a] * zu[a].y + dab * zu[b].y + dac * zu[c3].y);
        }
#pragma unroll
        for (int q = 0; q < 6; ++q) D[q] = (T)(S[q] * Ninv);
      } else {
        acc[1] += we * ((double)D[0] * qd[0] + (double)D[1] * qd[1] + (double)D[2] * qd[2] +
                                2.0 * ((double)D[3] * qd[3] + (double)D[4] * qd[4] + (double)D[5] * qd[5]));
      }
    }
    cplx<T> F[3];
    F[0] = mk<cplx<T>>(D[0] * u[0].x + D[5] * u[1].x + D[4] * u[2].x, D[0] * u[0].y + D[5] * u[1].y + D[4] * u[2].y);
    F[1] = mk<cplx<T>>(D[5] * u[0].x + D[1] * u[1].x + D[3] * u[2].x, D[5] * u[0].y + D[1] * u[1].y + D[3] * u[2].y);
    F[2] = mk<cplx<T>>(D[4] * u[0].x + D[3] * u[1].x + D[2] * u[2].x, D[4] * u[0].y + D[3] * u[1].y + D[2] * u[2].y);
    // ---- inhomogeneous strain
    const T k1 = (T)kv1, k2 = (T)kv2, k3 = (T)__ldg(&km.kvz_s[zs]);
    const T kk[4] = {(T)0, k1, k2, k3};
    const T B11 = (T)ph->B11, B12 = (T)ph->B12, B44 = (T)ph->B44;
    T K[3][3];
#pragma unroll
    for (int b = 1; b <= 3; ++b) {
      const int o1 = (b + 1) % 3 + 1, o2 = b % 3 + 1;
#pragma unroll
      for (int a = 1; a <= 3; ++a) {
        if (a == b) K[a - 1][b - 1] = B11 * kk[a] * kk[a] + B44 * kk[o1] * kk[o1] + B44 * kk[o2] * kk[o2];
        else K[a - 1][b - 1] = B12 * kk[a] * kk[b] + B44 * kk[a] * kk[b];
      }
    }
    // coup2 . didiK with coup2(a, i) of elastic.F:156-180: k_a B1xx/2 on
    // i = a, k_a B1yy/2 on the other two diagonal entries, k_c B4yz on the
    // shear entries (yz: b = y, c = z ...) that involve a, zero on the third
    const T hx = (T)(ph->HC2[0][0]), hy = (T)(ph->HC2[0][1]), h4 = (T)(ph->HC2[3][3]);
    cplx<T> ck[3] = {mk<cplx<T>>((T)0, (T)0), mk<cplx<T>>((T)0, (T)0), mk<cplx<T>>((T)0, (T)0)};
    if (ph->modulation_on) {
#pragma unroll
      for (int a = 0; a < 3; ++a) ck[a] = ckmod[tpos * 3 + a];
    }
    // rhs = -(c_k_mod + coup2 . didiK)  (optimize-inho-strain.F:28-45)
    cplx<T> cs[3], acou[3];
    {
      auto comb = [&](T ka, int ia, int ib, int ic, T kb, int sb, T kc, int sc_) {
        // ka (hx d_ia + hy (d_ib + d_ic)) + h4 (kb d_sb + kc d_sc)
        return mk<cplx<T>>(ka * (hx * d[ia].x + hy * (d[ib].x + d[ic].x)) + h4 * (kb * d[sb].x + kc * d[sc_].x),
                           ka * (hx * d[ia].y + hy * (d[ib].y + d[ic].y)) + h4 * (kb * d[sb].y + kc * d[sc_].y));
      };
      cs[0] = comb(k1, 0, 1, 2, k3, 4, k2, 5);
      cs[1] = comb(k2, 1, 0, 2, k3, 3, k1, 5);
      cs[2] = comb(k3, 2, 0, 1, k2, 3, k1, 4);
    }
    if constexpr (ACOU) {
      // dynamic acoustic field: acouK = i FFT(acouR) (acouFFT.F:22);
      // dVdacK = -i (c_k + coup2 didiK + K acouK) / N (dVdac.F:30-60);
      // energies with the K acouK of this field (energy_module.F:150-240)
      cplx<T> KA[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const cplx<T> X = buf[(9 + a) * ZS + zs * CW + cw];
        acou[a] = mk<cplx<T>>(-X.y, X.x);
      }
#pragma unroll
      for (int a = 0; a < 3; ++a)
        KA[a] = mk<cplx<T>>(K[a][0] * acou[0].x + K[a][1] * acou[1].x + K[a][2] * acou[2].x,
                            K[a][0] * acou[0].y + K[a][1] * acou[1].y + K[a][2] * acou[2].y);
      const T w2 = (T)0.5 * w1;
      T es = 0, ec = 0, em = 0;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        es += acou[a].x * KA[a].x + acou[a].y * KA[a].y;
        ec += acou[a].x * cs[a].x + acou[a].y * cs[a].y;
        em += acou[a].x * ck[a].x + acou[a].y * ck[a].y;
      }
      acc[2] += (double)(w2 * es);
      acc[3] += (double)(w2 * ec);
      acc[4] += (double)(w2 * em);
      const T ni = (T)Ninv;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const cplx<T> v = mk<cplx<T>>(ck[a].x + cs[a].x + KA[a].x, ck[a].y + cs[a].y + KA[a].y);
        buf[(9 + a) * ZS + zs * CW + cw] = mk<cplx<T>>(v.y * ni, -v.x * ni);
      }
    } else if (k0) {
#pragma unroll
      for (int a = 0; a < 3; ++a) acou[a] = mk<cplx<T>>((T)0, (T)0);  // inhomo_K_G(:,:,0,0,0) = 0
    } else {
      // K acou = rhs with K symmetric positive definite: adjugate over the
      // determinant (the reference factorises K by Cholesky, elastic.F:
      // 110-125; the solution is the same up to rounding)
      const T c00 = K[1][1] * K[2][2] - K[1][2] * K[1][2], c11 = K[0][0] * K[2][2] - K[0][2] * K[0][2];
      const T c22 = K[0][0] * K[1][1] - K[0][1] * K[0][1], c01 = K[0][2] * K[1][2] - K[0][1] * K[2][2];
      const T c02 = K[0][1] * K[1][2] - K[0][2] * K[1][1], c12 = K[0][1] * K[0][2] - K[0][0] * K[1][2];
      const T inv = (T)1 / (K[0][0] * c00 + K[0][1] * c01 + K[0][2] * c02);
      cplx<T> r[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) r[a] = mk<cplx<T>>((-ck[a].x - cs[a].x) * inv, (-ck[a].y - cs[a].y) * inv);
      acou[0] = mk<cplx<T>>(c00 * r[0].x + c01 * r[1].x + c02 * r[2].x, c00 * r[0].y + c01 * r[1].y + c02 * r[2].y);
      acou[1] = mk<cplx<T>>(c01 * r[0].x + c11 * r[1].x + c12 * r[2].x, c01 * r[0].y + c11 * r[1].y + c12 * r[2].y);
      acou[2] = mk<cplx<T>>(c02 * r[0].x + c12 * r[1].x + c22 * r[2].x, c02 * r[0].y + c12 * r[1].y + c22 * r[2].y);
    }
    if constexpr (!ACOU) {
      // coupling Re(acou* . coup2 didiK), modulation Re(acou* . c_k); the
      // strain energy Re(acou* K acou) = -(coupling + modulation) because
      // K acou = -(c_k + coup2 didiK)
      const T w2 = (T)0.5 * w1;  // energy_module.F weights: 1/2 at kx = 0, Lx/2
      T ec = 0, em = 0;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        ec += acou[a].x * cs[a].x + acou[a].y * cs[a].y;
        em += acou[a].x * ck[a].x + acou[a].y * ck[a].y;
      }
      acc[2] -= (double)(w2 * (ec + em));
      acc[3] += (double)(w2 * ec);
      acc[4] += (double)(w2 * em);
    }
    if (acouK_out) {
#pragma unroll
      for (int a = 0; a < 3; ++a) acouK_out[tpos * 3 + a] = acou[a];
    }
    const T ni = (T)Ninv;
    d[0] = mk<cplx<T>>(k1 * acou[0].x * ni, k1 * acou[0].y * ni);
    d[1] = mk<cplx<T>>(k2 * acou[1].x * ni, k2 * acou[1].y * ni);
    d[2] = mk<cplx<T>>(k3 * acou[2].x * ni, k3 * acou[2].y * ni);
    d[3] = mk<cplx<T>>((k3 * acou[1].x + k2 * acou[2].x) * ni, (k3 * acou[1].y + k2 * acou[2].y) * ni);
    d[4] = mk<cplx<T>>((k1 * acou[2].x + k3 * acou[0].x) * ni, (k1 * acou[2].y + k3 * acou[0].y) * ni);
    d[5] = mk<cplx<T>>((k2 * acou[0].x + k1 * acou[1].x) * ni, (k2 * acou[0].y + k1 * acou[1].y) * ni);
#pragma unroll
    for (int a = 0; a < 3; ++a) buf[a * ZS + zs * CW + cw] = F[a];
#pragma unroll
    for (int i = 0; i < 6; ++i) buf[(3 + i) * ZS + zs * CW + cw] = d[i];
  }
  __syncthreads();
  fft_inverse<T>(buf, B, pz, twz, buf_len);
  pdl_launch();
  z_tile_store<T>(buf, spec, g, zt, NC);
  block_partials<NQ_K>(acc, part, blockIdx.x);
}

// ------------------------------------------------------------------- k_z_lane
// k_z_kspace for the compile-time lengths Lz, on elements of W neighbouring kx
// slots (fft_lane.cuh).  A tile holds PW elements (PW W pencils) of all z and
// components as buf[c][z'][pw], z' = z ^ (z / R2 & 1): with that swap of
// neighbours the second stage's lanes (pw, a) fall on different banks.  The
// stages have compile-time offsets; the k-space step works on W wavevectors
// at a time.  Nyquist tiles (kx = Lx/2): the lanes of an element are ky slots.
// LZ = PW = 0: a length of two stages known at run time (ZGeo, up to 160), any
// tile of 1, 2 or 4 elements, and rows whose Lx/2 is no multiple of the tile
// or odd (the last element of a row is then (Lx/2 - 1, Lx/2) and there are no
// Nyquist tiles).
struct ZGeo {
  int R1, R2, lpw;  // stages, log2 of the elements per tile
  int ncol;         // columns of the regular tiles: Lx/2, odd Lx/2: Lx/2 + 1
  FastDiv d1, d2;   // by R1, R2
};
template <typename T, int LZ, int PW, bool ACOU>
struct ZCT {
  static constexpr int W = kLanes<T>, NC = ACOU ? 12 : 9;
  static constexpr int R1 = ct_radix(LZ, 0), R2 = LZ / R1;
  static constexpr int T1 = NC * PW * R2, T2 = NC * PW * R1;
  // Threads: one first-stage butterfly each, up to 288.  128 x 4 elements:
  // 288 threads at 96 registers in FP32 (74.1 us at 128^3; 256 threads 76.8),
  // 256 at 128 in FP64 (131.8 us; 288 threads 133.6, spilling); three tiles per
  // SM at 160 threads each took 96 and 166 us, the pass before this kernel
  // 81.5 and 143.
  static constexpr int NT = T1 > 256 && (ACOU || sizeof(T) == 8) ? 256 : (T1 + 31) / 32 * 32;
  static constexpr int SMEM = NC * LZ * PW * 16;
  static constexpr int MINB = NT >= 576 ? 1 : 576 / NT;
  static_assert(ct_nst(LZ) == 2 && R2 % 2 == 0 && NT % PW == 0, "");
};

template <typename T, bool ACOU>
struct ZCT<T, 0, 0, ACOU> {
  static constexpr int W = kLanes<T>, NC = ACOU ? 12 : 9, R1 = 0, R2 = 0, T1 = 0, T2 = 0, NT = 256, MINB = 2;
};

template <typename T, int LZ, int PW, bool ACOU = false>
__global__ void __launch_bounds__(ZCT<T, LZ, PW, ACOU>::NT, ZCT<T, LZ, PW, ACOU>::MINB)
    k_z_lane(cplx<T>* __restrict__ spec, const T* __restrict__ dtab, const cplx<T>* __restrict__ ckmod,
             cplx<T>* __restrict__ acouK_out, Geom g, ZGeo h, const cplx<T>* __restrict__ twz, KMaps km,
             const Phys* __restrict__ ph, double* __restrict__ part, DevScalars* sc, ZTiles zt,
             const RepArgs* __restrict__ grp = nullptr) {
  using Z = ZCT<T, LZ, PW, ACOU>;
  using V = lane_t<T>;
  constexpr bool RT = LZ == 0;
  constexpr int W = Z::W, NC = Z::NC, NT = Z::NT, PWM = RT ? 4 : PW;
  const int Lz = RT ? g.Lz : LZ, pwn = RT ? 1 << h.lpw : PW, r1 = RT ? h.R1 : Z::R1, r2 = RT ? h.R2 : Z::R2;
  const int ZS = Lz * pwn;  // (pwn: 1, 2 or 4)
  const int swap = RT ? ~r2 & 1 : 1;  // odd R2: the lanes are apart without the swap
  // quotients by the tile width, R1, R2 (compile-time: the compiler's)
  auto by_pw = [&](int n) { return RT ? n >> h.lpw : n / (PW > 0 ? PW : 1); };
  auto by_r1 = [&](int n) { return RT ? fdiv(n, h.d1) : n / (Z::R1 > 0 ? Z::R1 : 1); };
  auto by_r2 = [&](int n) { return RT ? fdiv(n, h.d2) : n / (Z::R2 > 0 ? Z::R2 : 1); };
  if (grp) {
    const RepArgs& a = grp[blockIdx.y];
    spec = (cplx<T>*)a.spec;
    dtab = (const T*)a.dtab;
    ph = a.ph;
    part = a.part_k;
    sc = a.sc;
  }
  FG_DYN_SMEM(smem_raw);
  CV<T>* const buf = reinterpret_cast<CV<T>*>(smem_raw);
  __shared__ cplx<T> tab[RT ? kLaneMax : LZ];
  __shared__ double sAB[PWM][W][10];  // S(k) along a pencil: A_q + B_q cos kz (sin kz for yz, zx)
  __shared__ double reds[NT / 32][NQ_K];
  const int tid = threadIdx.x;
  const int pw = tid & (pwn - 1), tile = blockIdx.x;
  if constexpr (RT) {
    for (int k = tid; k < Lz; k += NT) tab[k] = twz[k];
  } else {
    stage_twiddles<T, LZ, Z::R1, Z::R2>(tab, twz, (T)1);
  }
  auto twid = [&](int s, int b) { return RT ? tab[s * b] : tab[s * r2 + b]; };
  // this thread's element: slots (ys, col) and (ys, col + 1), of a Nyquist
  // tile (ys, m) and (ys + 1, m)
  const bool nyq = tile < zt.nnyq;
  int col, ys;
  {
    const int r = tile - zt.nnyq;
    ys = nyq ? tile * zt.CW + W * pw : r / zt.ntx;
    col = nyq ? g.m : (r - ys * zt.ntx) * zt.CW + W * pw;
  }
  const bool ok = ys < g.Ly && (!RT || nyq || col < h.ncol), okb = nyq && W == 2 ? ys + 1 < g.Ly : ok;
  if (!ok) {  // an element that does not count takes zeros through a regular K(k)
    ys = 1;
    if (RT && !nyq) col = 0;
  }
  const int colb = W == 2 && !nyq ? col + 1 : col, ysb = W == 2 && nyq && okb ? ys + 1 : ys;
  V k1, k2, w1;
  bool has_k0;
  {
    k1 = vpack((T)__ldg(&km.kvx_s[col]), (T)__ldg(&km.kvx_s[colb]));
    k2 = vpack((T)__ldg(&km.kvy_s[ys]), (T)__ldg(&km.kvy_s[ysb]));
    // full-spectrum multiplicity: kx = 0 is slot 0, kx = Lx/2 slot m
    w1 = vpack(!ok ? (T)0 : (col == 0 || col == g.m) ? (T)1 : (T)2, !okb ? (T)0 : colb == g.m ? (T)1 : (T)2);
    has_k0 = ok && !nyq && col == 0 && ys == 0;  // lane 0 (ky = 0 is slot 0)
    // S(k) of a pencil: one thread per pencil, each in a warp of its own
    if (tid % 32 < pwn && tid / 32 < W) {
      const double* j = ph->j;
      const double kap = ph->kap2x2;
      const double2 ty = __ldg(&km.try_s[tid / 32 == 0 ? ys : ysb]), tx = __ldg(&km.trx_s[tid / 32 == 0 ? col : colb]);
      const double c0 = tx.x, c1 = ty.x, s0 = tx.y, s1 = ty.y;
      double* a = sAB[pw][tid / 32];
      {
        a[0] = kap + 2 * j[1] * c0 + 2 * j[0] * c1 + 4 * j[2] * c0 * c1;
        a[1] = kap + 2 * j[1] * c1 + 2 * j[0] * c0 + 4 * j[2] * c1 * c0;
        a[2] = kap + 2 * j[0] * (c0 + c1) + 4 * j[3] * c0 * c1;
        a[3] = -4 * j[4] * s1 - 8 * j[6] * s1 * c0;  // yz, times sin kz
        a[4] = -4 * j[4] * s0 - 8 * j[6] * s0 * c1;  // zx, times sin kz
        a[5] = -4 * j[4] * s0 * s1;
        a[6] = 2 * j[0] + 4 * j[3] * c1 + 4 * j[2] * c0 + 8 * j[5] * c0 * c1;
        a[7] = 2 * j[0] + 4 * j[3] * c0 + 4 * j[2] * c1 + 8 * j[5] * c0 * c1;
        a[8] = 2 * j[1] + 4 * j[2] * (c0 + c1) + 8 * j[5] * c0 * c1;
        a[9] = -8 * j[6] * s0 * s1;
      }
    }
  }
  __syncthreads();
  pdl_wait();
  // Byte offset of this thread's element from the spectrum; a tile of a
  // compile-time Lz spans less than 2 GB
  constexpr unsigned ES = sizeof(cplx<T>);
  const unsigned zstep = (unsigned)g.plane_c * ES, cstep = (unsigned)g.ncplx * ES;
  const unsigned o0 = (unsigned)(ys * g.KXP + col) * ES, o1 = (unsigned)(ysb * g.KXP + colb) * ES;
  const unsigned long long pol = l2_evict_first();  // the input spectrum is consumed
  // element at byte offset off of the spectrum's first z and component
  auto gload = [&](unsigned off, auto nyqt) -> CV<T> {
    const char* q = reinterpret_cast<const char*>(spec) + off;
    if (!decltype(nyqt)::value && !(RT && nyq)) {
      if (RT && !ok) return CV<T>{vall((T)0), vall((T)0)};
      const rowvec<T>* r = reinterpret_cast<const rowvec<T>*>(q + o0);
      if constexpr (sizeof(T) == 4) return cv_of(ld_first(r, pol));
      else return cv_of(*r);
    } else {
      const cplx<T> zero = mk<cplx<T>>((T)0, (T)0);
      const cplx<T> x = ok ? *reinterpret_cast<const cplx<T>*>(q + o0) : zero;
      const cplx<T> y = okb ? *reinterpret_cast<const cplx<T>*>(q + o1) : zero;
      return CV<T>{vpack(x.x, y.x), vpack(x.y, y.y)};
    }
  };
  auto gstore = [&](unsigned off, const CV<T>& v, auto nyqt) {
    char* q = reinterpret_cast<char*>(spec) + off;
    if (!decltype(nyqt)::value && !(RT && nyq)) {
      if (!RT || ok) cv_row(reinterpret_cast<rowvec<T>*>(q + o0), v);
    } else {
      if (ok) *reinterpret_cast<cplx<T>*>(q + o0) = mk<cplx<T>>(vget<0>(v.re), vget<0>(v.im));
      if (W == 2 && okb) *reinterpret_cast<cplx<T>*>(q + o1) = mk<cplx<T>>(vget<W - 1>(v.re), vget<W - 1>(v.im));
    }
  };
  // tasks 0 .. count-1 (compile-time COUNT, or rt at run time)
  auto tasks = [&](auto count, int rt, auto&& f) {
    if constexpr (RT) {
#pragma unroll 1
      for (int t = tid; t < rt; t += NT) f(t);
    } else {
      lane_tasks<decltype(count)::value, NT>(tid, f);
    }
  };
#if FG_BOUNDS_CHECK
  // what a task touches (fg_in_range): butterfly b of the first stage (R
  // elements r2 apart, as many z of the spectrum, twiddles) and block a of the
  // second, in component c
  const int blen = RT ? NC * Lz * (zt.CW / W) : NC * LZ * PW;  // elements of buf
  auto first_in_range = [&](int c, int b, int R) {
    const int lastz = b + (R - 1) * r2, y = ysb > ys ? ysb : ys;
    return fg_in_range(c * ZS + b * pwn, c * ZS + (lastz | swap) * pwn + pw, blen) && fg_in_range(b, lastz, Lz) &&
           fg_in_range(0, (R - 1) * b, Lz) && fg_in_range(ys, y, g.Ly) && fg_in_range(col, nyq ? col : col + W - 1, g.KXP);
  };
  auto second_in_range = [&](int c, int a, int R) {
    return fg_in_range((c * Lz + a * r2) * pwn, (c * Lz + a * r2 + R - 1) * pwn + pw, blen) && fg_in_range(a, a, r1);
  };
#endif
  // forward: first stage from the spectrum
  auto first = [&](auto nyqt, auto radix) {
    constexpr int R = decltype(radix)::value;
    tasks(std::integral_constant<int, Z::T1>(), NC * pwn * r2, [&](int t) {
      const int r = by_pw(t), c = by_r2(r), b = r - c * r2, bx = b ^ swap;
      FG_SKIP_UNLESS(return, first_in_range(c, b, R));
      unsigned off = c * cstep + b * zstep;
      CV<T> v[R];
#pragma unroll
      for (int s = 0; s < R; ++s, off += r2 * zstep) v[s] = gload(off, nyqt);
      DftV<T, R, false>::run(v);
      CV<T>* d = buf + c * ZS + pw;
      cv_st(d + b * pwn, v[0]);
#pragma unroll
      for (int s = 1; s < R; ++s) cv_st(d + (((s & 1) ? bx : b) + r2 * s) * pwn, cvtw<T, false>(v[s], twid(s, b)));
    });
  };
  if constexpr (RT) {
    first_radix(r1, [&](auto radix) { first(std::false_type(), radix); });
  } else {
    if (nyq) first(std::true_type(), std::integral_constant<int, Z::R1>());
    else first(std::false_type(), std::integral_constant<int, Z::R1>());
  }
  // The dipole table's 6 values of W neighbouring slots, [slot / W][6][W], of
  // this thread's k-space element e: the next one's are loaded while the
  // strain part of the present one is computed
  V D[6];
  auto load_D = [&](int e) {
    const unsigned tz = (unsigned)by_pw(e) * g.KXP;
    if (!nyq) {
      const CV<T>* Dp = reinterpret_cast<const CV<T>*>(dtab + ((size_t)ys * Lz * g.KXP + tz + col) * 6);
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const CV<T> v = cv_stream(Dp + q);
        D[2 * q] = v.re;
        D[2 * q + 1] = v.im;
      }
    } else {
#pragma unroll
      for (int q = 0; q < 6; ++q)
        D[q] = vpack(dtab[tab_index<T>((long long)ys * Lz * g.KXP + tz + col, q)],
                     dtab[tab_index<T>((long long)ysb * Lz * g.KXP + tz + colb, q)]);
    }
  };
  if (tid < ZS) load_D(tid);
  __syncthreads();
  auto second = [&](auto inv, auto radix) {
    constexpr int R = decltype(radix)::value;
    tasks(std::integral_constant<int, Z::T2>(), NC * pwn * r1, [&](int t) {
      const int r = by_pw(t), c = by_r1(r), a = r - c * r1, x = a & swap;
      FG_SKIP_UNLESS(return, second_in_range(c, a, R));
      CV<T>*d0 = buf + c * ZS + pw + (a * r2 + x) * pwn, *d1 = d0 - 2 * x * pwn;  // z even / odd of the block
      CV<T> v[R];
#pragma unroll
      for (int q = 0; q < R; ++q) v[q] = cv_ld(((q & 1) ? d1 : d0) + q * pwn);
      DftV<T, R, decltype(inv)::value>::run(v);
#pragma unroll
      for (int q = 0; q < R; ++q) cv_st(((q & 1) ? d1 : d0) + q * pwn, v[q]);
    });
  };
  auto second_stage = [&](auto inv) {
    if constexpr (RT) {
      if (r2 > 1) second_radix(r2, [&](auto radix) { second(inv, radix); });
    } else {
      second(inv, std::integral_constant<int, Z::R2>());
    }
  };
  second_stage(std::false_type());
  __syncthreads();
  // ---- k space
  const double Ninv = ph->Ninv;
  const T ni = (T)Ninv;
  const T B11 = (T)ph->B11, B12 = (T)ph->B12, B44 = (T)ph->B44;
  const T hx = (T)(ph->HC2[0][0]), hy = (T)(ph->HC2[0][1]), h4 = (T)(ph->HC2[3][3]);
  const bool mod = ph->modulation_on != 0;
  double acc[NQ_K] = {0, 0, 0, 0, 0};
#pragma unroll 1
  for (int e = tid; e < ZS; e += NT) {
    const int zs = by_pw(e), zx = zs ^ (by_r2(zs) & swap);
    FG_SKIP_UNLESS(continue, fg_in_range(zx * pwn + pw, (NC - 1) * ZS + zx * pwn + pw, blen) && fg_in_range(zs, zs, Lz));
    CV<T>* el = buf + zx * pwn + pw;
    CV<T> u[3], d[6];
#pragma unroll
    for (int a = 0; a < 3; ++a) u[a] = cv_ld(el + a * ZS);
    const long long tz = (long long)zs * g.KXP;  // table positions of the element's lanes
    const bool k0 = has_k0 && zs == 0;           // slot 0 holds kz = 0
    {
      // Re(conj(u_a) u_b): xx, yy, zz, yz, zx, xy
      const V qv[6] = {vfma(u[0].re, u[0].re, vmul(u[0].im, u[0].im)), vfma(u[1].re, u[1].re, vmul(u[1].im, u[1].im)),
                       vfma(u[2].re, u[2].re, vmul(u[2].im, u[2].im)), vfma(u[1].re, u[2].re, vmul(u[1].im, u[2].im)),
                       vfma(u[2].re, u[0].re, vmul(u[2].im, u[0].im)), vfma(u[0].re, u[1].re, vmul(u[0].im, u[1].im))};
      // short-range and total dipole energies in FP64 from the same products,
      // so that their difference (the long-range energy) keeps its digits
      const double2 tzc = __ldg(&km.trz_s[zs]);
      auto lane_energy = [&](auto lane) {
        constexpr int L = decltype(lane)::value;
        const double* a = sAB[pw][L];
        double qd[6], dd[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) {
          qd[q] = (double)vget<L>(qv[q]);
          dd[q] = (double)vget<L>(D[q]);
        }
        double w = (double)vget<L>(w1);
        if (L == 0 && k0 && g.k0_exact) {  // left to homo_strain_tail
#pragma unroll
          for (int q = 0; q < 6; ++q) sc->D0[q] = dd[q];
          w = 0.0;
        }
        acc[0] += w * ((a[0] + a[6] * tzc.x) * qd[0] + (a[1] + a[7] * tzc.x) * qd[1] + (a[2] + a[8] * tzc.x) * qd[2] +
                       2.0 * (a[3] * tzc.y * qd[3] + a[4] * tzc.y * qd[4] + (a[5] + a[9] * tzc.x) * qd[5]));
        acc[1] += w * (dd[0] * qd[0] + dd[1] * qd[1] + dd[2] * qd[2] + 2.0 * (dd[3] * qd[3] + dd[4] * qd[4] + dd[5] * qd[5]));
      };
      lane_energy(std::integral_constant<int, 0>());
      if constexpr (W == 2) lane_energy(std::integral_constant<int, 1>());
    }
    // F = D u
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const int b = (a + 1) % 3, c = (a + 2) % 3;  // off-diagonal slots: yz 3, zx 4, xy 5
      const V dab = D[a == 0 ? 5 : a == 1 ? 3 : 4], dac = D[a == 0 ? 4 : a == 1 ? 5 : 3];
      cv_st(el + a * ZS, CV<T>{vfma(D[a], u[a].re, vfma(dab, u[b].re, vmul(dac, u[c].re))),
                               vfma(D[a], u[a].im, vfma(dab, u[b].im, vmul(dac, u[c].im)))});
    }
    if (e + NT < ZS) load_D(e + NT);
    // ---- inhomogeneous strain
#pragma unroll
    for (int i = 0; i < 6; ++i) d[i] = cv_ld(el + (3 + i) * ZS);
    if (k0) {
#pragma unroll
      for (int i = 0; i < 6; ++i) sc->didiK0[i] = (double)vget<0>(d[i].re);
      __threadfence();  // read by homo_strain_tail in another kernel
    }
    const V k3 = vall((T)__ldg(&km.kvz_s[zs]));
    // the elastic matrix K(k)
    const V b11 = vall(B11), b44 = vall(B44), bxy = vall(B12 + B44);
    const V k11 = vmul(k1, k1), k22 = vmul(k2, k2), k33 = vmul(k3, k3);
    const V K00 = vfma(b11, k11, vmul(b44, vadd(k22, k33))), K11 = vfma(b11, k22, vmul(b44, vadd(k11, k33)));
    const V K22 = vfma(b11, k33, vmul(b44, vadd(k11, k22)));
    const V K01 = vmul(bxy, vmul(k1, k2)), K02 = vmul(bxy, vmul(k1, k3)), K12 = vmul(bxy, vmul(k2, k3));
    // coup2 . didiK with coup2(a, i) of elastic.F:156-180
    CV<T> cs[3], ck[3], acou[3];
    {
      const V vx = vall(hx), vy = vall(hy), v4 = vall(h4);
      auto comb = [&](const V& ka, int ia, int ib, int ic, const V& kb, int sb, const V& kc, int sc_) {
        // ka (hx d_ia + hy (d_ib + d_ic)) + h4 (kb d_sb + kc d_sc)
        return CV<T>{vfma(ka, vfma(vx, d[ia].re, vmul(vy, vadd(d[ib].re, d[ic].re))),
                          vmul(v4, vfma(kb, d[sb].re, vmul(kc, d[sc_].re)))),
                     vfma(ka, vfma(vx, d[ia].im, vmul(vy, vadd(d[ib].im, d[ic].im))),
                          vmul(v4, vfma(kb, d[sb].im, vmul(kc, d[sc_].im))))};
      };
      cs[0] = comb(k1, 0, 1, 2, k3, 4, k2, 5);
      cs[1] = comb(k2, 1, 0, 2, k3, 3, k1, 5);
      cs[2] = comb(k3, 2, 0, 1, k2, 3, k1, 4);
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      cplx<T> m[2] = {mk<cplx<T>>((T)0, (T)0), mk<cplx<T>>((T)0, (T)0)};
      if (mod) {
#pragma unroll
        for (int l = 0; l < W; ++l)
          m[l] = ckmod[((long long)(l == 0 ? ys : ysb) * Lz * g.KXP + tz + (l == 0 ? col : colb)) * 3 + a];
      }
      ck[a] = CV<T>{vpack(m[0].x, m[1].x), vpack(m[0].y, m[1].y)};
    }
    const V w2 = vmul(vall((T)0.5), w1);  // energy_module.F weights: 1/2 at kx = 0, Lx/2
    auto dot = [&](const CV<T>* x) {
      V s = vmul(acou[0].re, x[0].re);
      s = vfma(acou[0].im, x[0].im, s);
#pragma unroll
      for (int a = 1; a < 3; ++a) s = vfma(acou[a].im, x[a].im, vfma(acou[a].re, x[a].re, s));
      return s;
    };
    auto add = [&](double& to, const V& v) {
      to += (double)vget<0>(v);
      if constexpr (W == 2) to += (double)vget<1>(v);
    };
    if constexpr (ACOU) {
      // dynamic acoustic field: acouK = i FFT(acouR) (acouFFT.F:22);
      // dVdacK = -i (c_k + coup2 didiK + K acouK) / N (dVdac.F:30-60);
      // energies with the K acouK of this field (energy_module.F:150-240)
      CV<T> KA[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const CV<T> X = cv_ld(el + (9 + a) * ZS);
        acou[a] = CV<T>{vneg(X.im), X.re};
      }
      KA[0] = CV<T>{vfma(K00, acou[0].re, vfma(K01, acou[1].re, vmul(K02, acou[2].re))),
                    vfma(K00, acou[0].im, vfma(K01, acou[1].im, vmul(K02, acou[2].im)))};
      KA[1] = CV<T>{vfma(K01, acou[0].re, vfma(K11, acou[1].re, vmul(K12, acou[2].re))),
                    vfma(K01, acou[0].im, vfma(K11, acou[1].im, vmul(K12, acou[2].im)))};
      KA[2] = CV<T>{vfma(K02, acou[0].re, vfma(K12, acou[1].re, vmul(K22, acou[2].re))),
                    vfma(K02, acou[0].im, vfma(K12, acou[1].im, vmul(K22, acou[2].im)))};
      add(acc[2], vmul(w2, dot(KA)));
      add(acc[3], vmul(w2, dot(cs)));
      add(acc[4], vmul(w2, dot(ck)));
      const V n = vall(ni);
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const CV<T> v = cvadd(cvadd(ck[a], cs[a]), KA[a]);
        cv_st(el + (9 + a) * ZS, CV<T>{vmul(v.im, n), vneg(vmul(v.re, n))});
      }
    } else {
      // K acou = rhs = -(c_k + coup2 didiK) with K symmetric positive
      // definite: adjugate over the determinant (the reference factorises K by
      // Cholesky, elastic.F:110-125; the same up to rounding)
      const V c00 = vfma(K11, K22, vneg(vmul(K12, K12))), c11 = vfma(K00, K22, vneg(vmul(K02, K02)));
      const V c22 = vfma(K00, K11, vneg(vmul(K01, K01))), c01 = vfma(K02, K12, vneg(vmul(K01, K22)));
      const V c02 = vfma(K01, K12, vneg(vmul(K02, K11))), c12 = vfma(K01, K02, vneg(vmul(K00, K12)));
      const V det = vfma(K00, c00, vfma(K01, c01, vmul(K02, c02)));
      // inhomo_K_G(:,:,0,0,0) = 0: no acoustic field at k = 0
      const T i0 = k0 ? (T)0 : (T)-1 / vget<0>(det);
      V inv = vpack(i0, (T)0);
      if constexpr (W == 2) inv = vpack(i0, (T)-1 / vget<W - 1>(det));
      CV<T> r[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) r[a] = CV<T>{vmul(vadd(ck[a].re, cs[a].re), inv), vmul(vadd(ck[a].im, cs[a].im), inv)};
      acou[0] = CV<T>{vfma(c00, r[0].re, vfma(c01, r[1].re, vmul(c02, r[2].re))),
                      vfma(c00, r[0].im, vfma(c01, r[1].im, vmul(c02, r[2].im)))};
      acou[1] = CV<T>{vfma(c01, r[0].re, vfma(c11, r[1].re, vmul(c12, r[2].re))),
                      vfma(c01, r[0].im, vfma(c11, r[1].im, vmul(c12, r[2].im)))};
      acou[2] = CV<T>{vfma(c02, r[0].re, vfma(c12, r[1].re, vmul(c22, r[2].re))),
                      vfma(c02, r[0].im, vfma(c12, r[1].im, vmul(c22, r[2].im)))};
      // coupling Re(acou* . coup2 didiK), modulation Re(acou* . c_k); the
      // strain energy Re(acou* K acou) = -(coupling + modulation) because
      // K acou = -(c_k + coup2 didiK)
      double x = 0.0, y = 0.0;
      add(x, vmul(w2, dot(cs)));
      if (mod) add(y, vmul(w2, dot(ck)));
      acc[2] -= x + y;
      acc[3] += x;
      acc[4] += y;
    }
    if (acouK_out) {
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        if (ok) acouK_out[((long long)ys * Lz * g.KXP + tz + col) * 3 + a] = mk<cplx<T>>(vget<0>(acou[a].re), vget<0>(acou[a].im));
        if (W == 2 && okb)
          acouK_out[((long long)ysb * Lz * g.KXP + tz + colb) * 3 + a] = mk<cplx<T>>(vget<W - 1>(acou[a].re), vget<W - 1>(acou[a].im));
      }
    }
    // inhoK = k (x) acou / N
    {
      const V n = vall(ni);
      CV<T> an[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) an[a] = CV<T>{vmul(acou[a].re, n), vmul(acou[a].im, n)};
      auto prod = [&](const V& ka, int a) { return CV<T>{vmul(ka, an[a].re), vmul(ka, an[a].im)}; };
      auto prod2 = [&](const V& ka, int a, const V& kb, int b) {
        return CV<T>{vfma(ka, an[a].re, vmul(kb, an[b].re)), vfma(ka, an[a].im, vmul(kb, an[b].im))};
      };
      cv_st(el + 3 * ZS, prod(k1, 0));
      cv_st(el + 4 * ZS, prod(k2, 1));
      cv_st(el + 5 * ZS, prod(k3, 2));
      cv_st(el + 6 * ZS, prod2(k3, 1, k2, 2));
      cv_st(el + 7 * ZS, prod2(k1, 2, k3, 0));
      cv_st(el + 8 * ZS, prod2(k2, 0, k1, 1));
    }
  }
  // this tile's energies: warps by shuffles, warps in order
#pragma unroll
  for (int q = 0; q < NQ_K; ++q) {
    const double s = warp_sum(acc[q]);
    if (tid % 32 == 0) reds[tid / 32][q] = s;
  }
  __syncthreads();
  // inverse: the last forward stage first, the first one to the spectrum
  second_stage(std::true_type());
  if (tid < NQ_K) {
    double s = 0.0;
    for (int w = 0; w < NT / 32; ++w) s += reds[w][tid];
    part[(long long)tile * NQ_K + tid] = s;
  }
  __syncthreads();
  pdl_launch();
  auto last = [&](auto nyqt, auto radix) {
    constexpr int R = decltype(radix)::value;
    tasks(std::integral_constant<int, Z::T1>(), NC * pwn * r2, [&](int t) {
      const int r = by_pw(t), c = by_r2(r), b = r - c * r2, bx = b ^ swap;
      FG_SKIP_UNLESS(return, first_in_range(c, b, R));
      const CV<T>* d = buf + c * ZS + pw;
      CV<T> v[R];
      v[0] = cv_ld(d + b * pwn);
#pragma unroll
      for (int s = 1; s < R; ++s) v[s] = cvtw<T, true>(cv_ld(d + (((s & 1) ? bx : b) + r2 * s) * pwn), twid(s, b));
      DftV<T, R, true>::run(v);
      unsigned off = c * cstep + b * zstep;
#pragma unroll
      for (int s = 0; s < R; ++s, off += r2 * zstep) gstore(off, v[s], nyqt);
    });
  };
  if constexpr (RT) {
    first_radix(r1, [&](auto radix) { last(std::false_type(), radix); });
  } else {
    if (nyq) last(std::true_type(), std::integral_constant<int, Z::R1>());
    else last(std::false_type(), std::integral_constant<int, Z::R1>());
  }
}

// ------------------------------------------------------------------ k_assemble
// Real-space force (dVddi) on every site:
//   F = F_dd                                      (c2r of k_z_kspace slots 0..2)
//     + anharmonic polynomial force               (dVddi-unharmonic.F:34-65)
//     - Z* E                                      (mirror_force_mirror.F:42-50)
//     + homogeneous strain coupling, w = strain B2 (dVddi-homo-coupling.F:209-237)
//     + inhomogeneous strain coupling, w(R) = eta(R) B2 (dVddi_inho_coupling.F:114-142)
// and the per-block sums of the anharmonic energy (:67-99) and Z* u.E.
// 16-byte vectors of consecutive sites of one component (4 floats or 2
// doubles); used when a vector never straddles a z layer (plane % width == 0).
template <typename T>
struct alignas(16) V16 {
  static constexpr int n = 16 / (int)sizeof(T);
  T v[16 / sizeof(T)];
};
template <typename T>
__device__ __forceinline__ V16<T> ldv(const T* p) { return *reinterpret_cast<const V16<T>*>(p); }
// ldv with the evict_first L2 policy (FP64: when FG_L2_HINT_FP64)
template <typename T>
__device__ __forceinline__ V16<T> ldv_first(const T* p, unsigned long long pol) {
  V16<T> r;
  if constexpr (sizeof(T) == 4) {
    const float4 v = ld_first(reinterpret_cast<const float4*>(p), pol);
    r.v[0] = v.x; r.v[1] = v.y; r.v[2] = v.z; r.v[3] = v.w;
  } else if constexpr (FG_L2_HINT_FP64) {
    const double2 v = ld_first(reinterpret_cast<const double2*>(p), pol);
    r.v[0] = v.x; r.v[1] = v.y;
  } else {
    r = ldv(p);
  }
  return r;
}
template <typename T>
__device__ __forceinline__ void stv(T* p, const V16<T>& a) { *reinterpret_cast<V16<T>*>(p) = a; }

// Constants of the site force, in FP64 for both precisions: the mixed path
// reads FP32 u, the FP32 dipole-dipole force and the FP32 eta, and sums the
// on-site polynomial, the field and both strain couplings in FP64.  Those
// local terms carry the largest forces (|F| up to ~30x the rms force on the
// tail sites of a sigma = 0.1 A configuration), so evaluating them in FP32
// would put their rounding (~1e-6 of the rms force) on exactly those sites.
// On-site polynomial of one species: force combinations and energy
// coefficients (dVddi-unharmonic.F:28-32,67-99)
struct Poly {
  double fa2g, tg, sk, tk2, fk, k4x8;
  double Pa, Pg, P1, P2, P3, P4;
};
struct AsmConst {
  Poly pl;                             // species 1 (the bulk sweeps)
  double hx, hy, h4;                   // homogeneous_coupling_2: B1xx/2, B1yy/2, B4yz
  double Zs;
  int E_on;
  int gap_id;                          // of a film (k_assemble's FILM instance)
};
// Per-step values of the site force, read from DevScalars: strain . B2 and
// the uniform field.
struct AsmDyn {
  double wh[6];
  double E0, E1, E2;
};

// Force on one site from F_dd, u and eta (see k_assemble); acc += energies.
__device__ __forceinline__ void assemble_site(const Poly& pl, const AsmConst& k, double Zs, const AsmDyn& dy,
                                              double ux, double uy, double uz, double f0, double f1, double f2,
                                              const double* eta, double& o0, double& o1, double& o2, double* acc) {
  const double d0 = ux * ux, d1 = uy * uy, d2 = uz * uz;
  const double uu = d0 + d1 + d2;
  // 4th order
  f0 = f0 + ux * (pl.fa2g * uu - pl.tg * d0);
  f1 = f1 + uy * (pl.fa2g * uu - pl.tg * d1);
  f2 = f2 + uz * (pl.fa2g * uu - pl.tg * d2);
  // 6th and 8th order
  const double uu2 = uu * uu, uu3 = uu2 * uu;
  f0 = f0 + ux * (pl.sk * uu2 + pl.k4x8 * uu3 - pl.tk2 * (d0 * d0) - pl.fk * d1 * d2);
  f1 = f1 + uy * (pl.sk * uu2 + pl.k4x8 * uu3 - pl.tk2 * (d1 * d1) - pl.fk * d2 * d0);
  f2 = f2 + uz * (pl.sk * uu2 + pl.k4x8 * uu3 - pl.tk2 * (d2 * d2) - pl.fk * d0 * d1);
  acc[0] += pl.Pa * uu2 + pl.Pg * (d0 * d1 + d1 * d2 + d2 * d0) + pl.P1 * uu3 +
            pl.P2 * ((d0 * d0) * (d1 + d2) + (d1 * d1) * (d2 + d0) + (d2 * d2) * (d0 + d1)) + pl.P3 * d0 * d1 * d2 +
            pl.P4 * (uu2 * uu2);
  if (k.E_on) {
    f0 = f0 - Zs * dy.E0;
    f1 = f1 - Zs * dy.E1;
    f2 = f2 - Zs * dy.E2;
    acc[1] += Zs * (ux * dy.E0 + uy * dy.E1 + uz * dy.E2);
  }
  // homogeneous strain coupling
  f0 = f0 + 2 * dy.wh[0] * ux + dy.wh[4] * uz + dy.wh[5] * uy;
  f1 = f1 + 2 * dy.wh[1] * uy + dy.wh[3] * uz + dy.wh[5] * ux;
  f2 = f2 + 2 * dy.wh[2] * uz + dy.wh[3] * uy + dy.wh[4] * ux;
  // inhomogeneous strain coupling, w_q = sum_j eta_j B2(j, q) with the
  // sparsity of homogeneous_coupling_2 (eta already carries 1/N)
  const double w0 = k.hx * eta[0] + k.hy * (eta[1] + eta[2]);
  const double w1 = k.hx * eta[1] + k.hy * (eta[0] + eta[2]);
  const double w2 = k.hx * eta[2] + k.hy * (eta[0] + eta[1]);
  const double w3 = k.h4 * eta[3], w4 = k.h4 * eta[4], w5 = k.h4 * eta[5];
  o0 = f0 + 2 * w0 * ux + w4 * uz + w5 * uy;
  o1 = f1 + 2 * w1 * uy + w3 * uz + w5 * ux;
  o2 = f2 + 2 * w2 * uz + w3 * uy + w4 * ux;
}

// Film mirror (mirror.F:9-36): layers z and partner(z) hold (f_x, f_y, f_z) and
// (-f_x, -f_y, f_z); the lower one is the source.  z itself: a layer without
// a partner.
__device__ __forceinline__ int film_partner(int z, int Lz, int gap_id) {
  if (gap_id == 0) return Lz - 1 - z;
  return z > 0 ? Lz - z : 0;
}
// Layers that are nobody's image; they are the first ones.
__host__ __device__ __forceinline__ int film_layers(int Lz, int gap_id) { return gap_id == 0 ? (Lz + 1) / 2 : Lz / 2 + 1; }

// The force of one site in the field type T.  The mixed path (T = float)
// rounds the FP64 sum once; with lo != null it also stores the rounding
// residual, so that hi + lo carries the FP64 force to ~2^-48 for a caller
// that reads dVddi, while the integrators consume hi.
template <typename T>
__device__ __forceinline__ T force_hi(double o) { return (T)o; }
template <typename T>
__device__ __forceinline__ T force_lo(double o, T hi) { return sizeof(T) == 4 ? (T)(o - (double)hi) : (T)0; }

// A kick or drift coefficient, FP64, times a field value in T.  FP32: the
// coefficient's rounding would be the same error on every site (6e-8 of each
// kick, which the energy sums up coherently), so its low part is kept; the
// product is rounded once per site.
template <typename T> struct StepCoef;
template <> struct StepCoef<double> {
  double c;
  __device__ __forceinline__ explicit StepCoef(double v) : c(v) {}
  __device__ __forceinline__ double operator*(double x) const { return c * x; }
};
template <> struct StepCoef<float> {
  float hi, lo;
  __device__ __forceinline__ explicit StepCoef(double v) : hi((float)v), lo((float)(v - (double)hi)) {}
  __device__ __forceinline__ float operator*(float x) const { return fmaf(hi, x, lo * x); }
};

// Masked kinetic sums of the closing kick (35f) of one site: p <- p - c F
// and p^2/m, p.F/m, F^2/m, formed in S and added to ke (FP64) when the site
// counts.  S: T; FP64 for films, as k_kick_close's loop over sites.
template <typename S, typename T>
__device__ __forceinline__ void close_site(T* __restrict__ p, long long ns, long long i, const StepCoef<T>& c, T o0, T o1, T o2,
                                           bool counted, double mi, double* ke) {
  const T q0 = p[i] - c * o0, q1 = p[ns + i] - c * o1, q2 = p[2 * ns + i] - c * o2;
  p[i] = q0;
  p[ns + i] = q1;
  p[2 * ns + i] = q2;
  if (counted) {
    ke[0] += (double)((S)q0 * q0 + (S)q1 * q1 + (S)q2 * q2) * mi;
    ke[1] += (double)((S)q0 * o0 + (S)q1 * o1 + (S)q2 * o2) * mi;
    ke[2] += (double)((S)o0 * o0 + (S)o1 * o1 + (S)o2 * o2) * mi;
  }
}

// CLOSE (the force of a Nose-Poincare step, nose-poincare.F:55-71): after the
// force, the closing kick (35f) p <- p - dt/2 s_{n+1} F with the masked sums
// p^2/m, p.F/m, F^2/m of the new p in part_ke; the last block finishes the
// force (energies, commit of the prepared half step, (35e)) and the step
// (np_close_tail: KE, H_NP and (38) of the next step).
// Flo (mixed path, may be null): the FP32 residual of each force component,
// F + Flo = the FP64 site sum.
// FILM (with CLOSE, without per-site arrays): only the source layers' forces
// are computed; each is written to its partner too, with the mirror's signs,
// and both sites' momenta are kicked and counted.  The partner's u is the
// mirrored one, so its on-site energy is the source's.  Half of the field
// sums and of the site polynomials, and no k_mirror between this kernel and a
// closing kick of its own: film step 64x64x32, mixed, 53 -> 44 us with the
// mirrored drift (k_kick_drift).
template <typename T, bool CLOSE = false, bool SITES = false, bool FILM = false>
__global__ void __launch_bounds__(256, 2)
    k_assemble(const T* __restrict__ rw, const T* __restrict__ u, T* __restrict__ F, Geom g,
               const Phys* __restrict__ ph, DevScalars* sc, double* __restrict__ part, int tail, unsigned int* done,
               const unsigned char* __restrict__ site_species, const T* __restrict__ site_zstar,
               const T* __restrict__ site_E, int zl0, T* __restrict__ p, const double* __restrict__ layer_minv,
               const unsigned char* __restrict__ layer_sump, const T* __restrict__ site_minv,
               const unsigned char* __restrict__ site_sump, double* __restrict__ part_ke, T* __restrict__ Flo,
               const AsmConst k, const RepArgs* __restrict__ grp, DevScalars* host) {
  pdl_launch();  // by default one resident wave, with nothing of this grid left to schedule
  pdl_wait();
  if (grp) {
    const RepArgs& a = grp[blockIdx.y];
    rw = (const T*)a.rwork;
    u = (const T*)a.u;
    F = (T*)a.F;
    ph = a.ph;
    sc = a.sc;
    part = a.part_r;
    done = a.done_as;
    p = (T*)a.p;
    layer_minv = a.layer_minv;
    layer_sump = a.layer_sump;
    part_ke = a.part_ke;
  }
  // site_*: per-site species (.relaxor), Z* and local field (.localfield);
  // they take the scalar loop.  zl0 > 0: rw components zl0..zl0+2 hold the
  // long-range dipole field of Z* u, which acts on the site times its Z*
  // (dVddi-dipole-dipole.F:52-60); components 0..2 the short-range part.
  const long long ns = g.nsite;
  // pend_kick_f: prepared by the previous step's tail, not changed by this
  // step's commit
  const StepCoef<T> cf(CLOSE ? __ldcg(&sc->pend_kick_f) : 0.0);
  double ke[3] = {0.0, 0.0, 0.0};
  const unsigned long long pol_rw = l2_evict_first();
  // k: the static constants (kernel parameter, built by asm_const on the
  // host); dy: this step's strain coupling and field
  // (in shared memory: read at each use instead of held in nine FP64
  // register pairs through the loop)
  __shared__ AsmDyn dy;
  if (threadIdx.x < 6) dy.wh[threadIdx.x] = sc->w_hom[threadIdx.x];
  if (threadIdx.x == 6) dy.E0 = sc->E[0];
  if (threadIdx.x == 7) dy.E1 = sc->E[1];
  if (threadIdx.x == 8) dy.E2 = sc->E[2];
  __syncthreads();
  double acc[NQ_R] = {0.0, 0.0};
  // FILM: sources and layers without a partner come first (film_partner)
  const long long nown = FILM ? (long long)film_layers(g.Lz, k.gap_id) * g.plane_r : ns;
  constexpr int NV = V16<T>::n;
  using AV = V16<T>;
  const long long stride = (long long)gridDim.x * blockDim.x;
  // SITES: the per-site loop (any of the site arrays present, chosen on the
  // host); otherwise the bulk loops, compiled without it so that its FP64
  // species polynomial does not set their register budget
  if constexpr (SITES) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < ns; i += stride) {
      AsmDyn dys = dy;
      double dk2 = 0.0;
      Poly pl;  // this site's species (read_relaxor.F)
      if (site_species) {
        const Phys::Species* q = &ph->sp[site_species[i]];
        pl = Poly{q->fa2g, q->tg, q->sk, q->tk2, q->fk, q->k4x8, q->Pa, q->Pg, q->P1, q->P2, q->P3, q->P4};
        dk2 = q->dk2;
      } else {
        pl = k.pl;
      }
      const double Zs = site_zstar ? (double)site_zstar[i] : k.Zs;
      if (site_E) {
        dys.E0 = dy.E0 + (double)site_E[i];
        dys.E1 = dy.E1 + (double)site_E[ns + i];
        dys.E2 = dy.E2 + (double)site_E[2 * ns + i];
      }
      double eta[6];
#pragma unroll
      for (int q = 0; q < 6; ++q) eta[q] = (double)rw[(3 + q) * ns + i];
      const double ux = u[i], uy = u[ns + i], uz = u[2 * ns + i];
      double f0 = rw[i], f1 = rw[ns + i], f2 = rw[2 * ns + i];
      if (zl0 > 0) {
        f0 = f0 + Zs * (double)rw[(zl0 + 0) * ns + i];
        f1 = f1 + Zs * (double)rw[(zl0 + 1) * ns + i];
        f2 = f2 + Zs * (double)rw[(zl0 + 2) * ns + i];
      }
      double o0, o1, o2;
      assemble_site(pl, k, Zs, dys, ux, uy, uz, f0, f1, f2, eta, o0, o1, o2, acc);
      if (dk2 != 0.0) {  // kappa2(s) - kappa2(1) (dVddi-unharmonic.F:40,73)
        const double t = 2 * dk2;
        o0 = o0 + t * ux;
        o1 = o1 + t * uy;
        o2 = o2 + t * uz;
        acc[0] += dk2 * (ux * ux + uy * uy + uz * uz);
      }
      const T h0 = force_hi<T>(o0), h1 = force_hi<T>(o1), h2 = force_hi<T>(o2);
      F[i] = h0;
      F[ns + i] = h1;
      F[2 * ns + i] = h2;
      if (Flo) {
        Flo[i] = force_lo<T>(o0, h0);
        Flo[ns + i] = force_lo<T>(o1, h1);
        Flo[2 * ns + i] = force_lo<T>(o2, h2);
      }
      if constexpr (CLOSE) {
        const int z = (int)(i / g.plane_r);
        close_site<T>(p, ns, i, cf, h0, h1, h2, site_sump ? site_sump[i] != 0 : layer_sump[z] != 0,
                   site_minv ? (double)site_minv[i] : layer_minv[z], ke);
      }
    }
  } else if (g.plane_r % NV == 0) {
    // closing kick of NV sites of layer z and their masked sums
    auto close = [&](long long i, int z, const AV& o0, const AV& o1, const AV& o2) {
      AV q[3] = {ldv(p + i), ldv(p + ns + i), ldv(p + 2 * ns + i)};
      T pp = 0, pf = 0, ff = 0;
#pragma unroll
      for (int l = 0; l < NV; ++l) {
        const T f3[3] = {o0.v[l], o1.v[l], o2.v[l]};
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          q[a].v[l] = q[a].v[l] - cf * f3[a];
          pp += q[a].v[l] * q[a].v[l];
          pf += q[a].v[l] * f3[a];
          ff += f3[a] * f3[a];
        }
      }
#pragma unroll
      for (int a = 0; a < 3; ++a) stv(p + a * ns + i, q[a]);
      if (layer_sump[z]) {
        const double mi = layer_minv[z];
        ke[0] += (double)pp * mi;
        ke[1] += (double)pf * mi;
        ke[2] += (double)ff * mi;
      }
    };
    for (long long iv = (long long)blockIdx.x * blockDim.x + threadIdx.x; iv < nown / NV; iv += stride) {
      const long long i = iv * NV;
      const AV ux = ldv(u + i), uy = ldv(u + ns + i), uz = ldv(u + 2 * ns + i);
      // rw is consumed here: evict_first keeps u, p and F in L2
      const AV a0 = ldv_first(rw + i, pol_rw), a1 = ldv_first(rw + ns + i, pol_rw),
               a2 = ldv_first(rw + 2 * ns + i, pol_rw);
      AV e[6];
#pragma unroll
      for (int q = 0; q < 6; ++q) e[q] = ldv_first(rw + (3 + q) * ns + i, pol_rw);
      AV o0, o1, o2, l0, l1, l2;
      double as[NQ_R] = {0.0, 0.0};
#pragma unroll
      for (int l = 0; l < NV; ++l) {
        const double eta[6] = {e[0].v[l], e[1].v[l], e[2].v[l], e[3].v[l], e[4].v[l], e[5].v[l]};
        double d0, d1, d2;
        assemble_site(k.pl, k, k.Zs, dy, ux.v[l], uy.v[l], uz.v[l], a0.v[l], a1.v[l], a2.v[l], eta, d0, d1, d2,
                      FILM ? as : acc);
        o0.v[l] = force_hi<T>(d0);
        o1.v[l] = force_hi<T>(d1);
        o2.v[l] = force_hi<T>(d2);
        l0.v[l] = force_lo<T>(d0, o0.v[l]);
        l1.v[l] = force_lo<T>(d1, o1.v[l]);
        l2.v[l] = force_lo<T>(d2, o2.v[l]);
      }
      stv(F + i, o0);
      stv(F + ns + i, o1);
      stv(F + 2 * ns + i, o2);
      if (Flo) {
        stv(Flo + i, l0);
        stv(Flo + ns + i, l1);
        stv(Flo + 2 * ns + i, l2);
      }
      if constexpr (CLOSE) {
        const int z = (int)(i / g.plane_r);
        close(i, z, o0, o1, o2);
        if constexpr (FILM) {
          const int zd = film_partner(z, g.Lz, k.gap_id);
          acc[0] += as[0];
          acc[1] += as[1];
          if (zd != z) {
            const long long d = i + (long long)(zd - z) * g.plane_r;
            AV m0, m1;
#pragma unroll
            for (int l = 0; l < NV; ++l) {
              m0.v[l] = -o0.v[l];
              m1.v[l] = -o1.v[l];
              if (k.E_on)
                acc[1] += k.Zs * ((double)uz.v[l] * dy.E2 - ((double)ux.v[l] * dy.E0 + (double)uy.v[l] * dy.E1));
            }
            acc[0] += as[0];
            stv(F + d, m0);
            stv(F + ns + d, m1);
            stv(F + 2 * ns + d, o2);
            close(d, zd, m0, m1, o2);
          }
        }
      }
    }
  } else {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nown; i += stride) {
      double eta[6];
#pragma unroll
      for (int q = 0; q < 6; ++q) eta[q] = (double)rw[(3 + q) * ns + i];
      double o0, o1, o2, as[NQ_R] = {0.0, 0.0};
      const double ux = u[i], uy = u[ns + i], uz = u[2 * ns + i];
      assemble_site(k.pl, k, k.Zs, dy, ux, uy, uz, rw[i], rw[ns + i], rw[2 * ns + i], eta, o0, o1, o2, FILM ? as : acc);
      const T h0 = force_hi<T>(o0), h1 = force_hi<T>(o1), h2 = force_hi<T>(o2);
      F[i] = h0;
      F[ns + i] = h1;
      F[2 * ns + i] = h2;
      if (Flo) {
        Flo[i] = force_lo<T>(o0, h0);
        Flo[ns + i] = force_lo<T>(o1, h1);
        Flo[2 * ns + i] = force_lo<T>(o2, h2);
      }
      if constexpr (CLOSE) {
        const int z = (int)(i / g.plane_r);
        using S = std::conditional_t<FILM, double, T>;
        close_site<S>(p, ns, i, cf, h0, h1, h2, layer_sump[z] != 0, layer_minv[z], ke);
        if constexpr (FILM) {
          const int zd = film_partner(z, g.Lz, k.gap_id);
          acc[0] += as[0];
          acc[1] += as[1];
          if (zd != z) {
            const long long d = i + (long long)(zd - z) * g.plane_r;
            acc[0] += as[0];
            if (k.E_on) acc[1] += k.Zs * (uz * dy.E2 - (ux * dy.E0 + uy * dy.E1));
            F[d] = -h0;
            F[ns + d] = -h1;
            F[2 * ns + d] = h2;
            close_site<S>(p, ns, d, cf, -h0, -h1, h2, layer_sump[zd] != 0, layer_minv[zd], ke);
          }
        }
      }
    }
  }
  if constexpr (CLOSE) {
    block_partials2<NQ_R, 3>(acc, ke, part, part_ke, blockIdx.x);
    if (is_last_block(done)) np_step_tail(ph, sc, part, part_ke, gridDim.x, host);
  } else {
    block_partials<NQ_R>(acc, part, blockIdx.x);
    if (tail == TAIL_ENERGIES && is_last_block(done)) force_energies_tail(ph, sc, part, gridDim.x, false, host);
  }
}

// --------------------------------------------------------------- integrators
// The acoustic field's arrays, for the launches that treat it beside the
// dipoles' as a second row of blocks: one launch and one tail instead of two,
// and twice the blocks in flight (48^3 FP64 has work for 216 of the 1184 that
// fit).  Leapfrog step of 48^3 FP64: 55.7 -> 49.2 us.
template <typename T>
struct SecondField {
  T *u, *p;
  const T* F;
  const double* layer_minv;
  const unsigned char* layer_mask;
  const T* site_minv;
};

// p <- p - coef * F on every site (leapfrog.F:134-138) and the masked sum
// p^2 m^-1 of kinetic_energy_dipo.F:92-105.  Per-layer masses and sum_p
// masks (film halves, dead layers).
template <typename T>
__global__ void __launch_bounds__(256) k_kick(T* __restrict__ p, const T* __restrict__ F, const double* coef, Geom g,
                                              const double* __restrict__ layer_minv,
                                              const unsigned char* __restrict__ layer_sump, double* __restrict__ part,
                                              int tail, unsigned int* done, const Phys* __restrict__ ph,
                                              DevScalars* sc, int zero_unmasked, const T* __restrict__ site_minv,
                                              const unsigned char* __restrict__ site_sump, const SecondField<T> acou) {
  // zero_unmasked: p = 0 outside sum_p (velocity_scaling.F:61-71).
  // site_minv / site_sump: per-site masses and masks (.relaxor, .defects)
  // instead of the per-layer tables; they take the scalar loop.
  const double* const part0 = part;
  if (blockIdx.y == 1) {
    p = acou.p;
    F = acou.F;
    layer_minv = acou.layer_minv;
    layer_sump = acou.layer_mask;
    site_minv = acou.site_minv;
    site_sump = nullptr;
    part += gridDim.x;
  }
  const long long ns = g.nsite;
  const StepCoef<T> c(*coef);
  double acc[1] = {0.0};
  constexpr int NV = V16<T>::n;
  using AV = V16<T>;
  const long long stride = (long long)gridDim.x * blockDim.x;
  if (g.plane_r % NV == 0 && site_minv == nullptr && site_sump == nullptr) {
    for (long long iv = (long long)blockIdx.x * blockDim.x + threadIdx.x; iv < ns / NV; iv += stride) {
      const long long i = iv * NV;
      const int z = (int)(i / g.plane_r);
      V16<T> q0 = ldv(p + i), q1 = ldv(p + ns + i), q2 = ldv(p + 2 * ns + i);
      const V16<T> f0 = ldv(F + i), f1 = ldv(F + ns + i), f2 = ldv(F + 2 * ns + i);
      const T keep = (zero_unmasked && !layer_sump[z]) ? (T)0 : (T)1;
      double ke = 0.0;
#pragma unroll
      for (int l = 0; l < NV; ++l) {
        q0.v[l] = keep * (q0.v[l] - c * f0.v[l]);
        q1.v[l] = keep * (q1.v[l] - c * f1.v[l]);
        q2.v[l] = keep * (q2.v[l] - c * f2.v[l]);
        ke += (double)q0.v[l] * q0.v[l] + (double)q1.v[l] * q1.v[l] + (double)q2.v[l] * q2.v[l];
      }
      stv(p + i, q0);
      stv(p + ns + i, q1);
      stv(p + 2 * ns + i, q2);
      if (layer_sump[z]) acc[0] += ke * layer_minv[z];
    }
  } else {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < ns; i += stride) {
      const int z = (int)(i / g.plane_r);
      const bool counted = site_sump ? site_sump[i] != 0 : layer_sump[z] != 0;
      const T keep = (zero_unmasked && !counted) ? (T)0 : (T)1;
      const T p0 = keep * (p[i] - c * F[i]);
      const T p1 = keep * (p[ns + i] - c * F[ns + i]);
      const T p2 = keep * (p[2 * ns + i] - c * F[2 * ns + i]);
      p[i] = p0;
      p[ns + i] = p1;
      p[2 * ns + i] = p2;
      if (counted) {
        const double mi = site_minv ? (double)site_minv[i] : layer_minv[z];
        acc[0] += (double)p0 * p0 * mi + (double)p1 * p1 * mi + (double)p2 * p2 * mi;
      }
    }
  }
  block_partials<1>(acc, part, blockIdx.x);
  if (tail != TAIL_NONE && is_last_block(done, gridDim.x * gridDim.y)) {
    if (tail == TAIL_LF_FINAL) lf_final_tail(ph, sc, part0, gridDim.y == 2 ? part0 + gridDim.x : nullptr, gridDim.x);
    else if (tail == TAIL_VS) vs_tail(ph, sc, part0, gridDim.x);
    else if (tail == TAIL_VS_ACOU) acou_tail(ph, sc, part0, gridDim.x);
  }
}

// Sum of v over the block, returned to every thread.
__device__ __forceinline__ double block_sum(double v) {
  __shared__ double red[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  v = warp_sum(v);
  if (lane == 0) red[wid] = v;
  __syncthreads();
  double t = 0.0;
  for (int w = 0; w < (int)((blockDim.x + 31) >> 5); ++w) t += red[w];
  __syncthreads();
  return t;
}

// Heat pump of leapfrog.F:44-87: block 0 scales layer Lz/4 up by delta_e
// per site, block 1 layer 3 (Lz/4) down, the dipole momenta by
// sqrt((e_layer +- Lx Ly delta_e) / e_layer) with e_layer the layer's kinetic
// energy (sum p^2/m / 2 times Lx Ly / counted sites), and likewise the
// acoustic momenta with delta_e_acou (sum acouP^2/m / 2).
template <typename T>
__global__ void __launch_bounds__(256) k_layer_pump(T* __restrict__ p, T* __restrict__ pa, Geom g,
                                                    const double* __restrict__ layer_minv,
                                                    const double* __restrict__ layer_macou,
                                                    const unsigned char* __restrict__ layer_sump, double de,
                                                    double dea, const T* __restrict__ site_minv = nullptr,
                                                    const T* __restrict__ site_macou = nullptr,
                                                    const double* __restrict__ layer_nsum = nullptr) {
  const int z = blockIdx.x == 0 ? g.Lz / 4 : (g.Lz / 4) * 3;
  const double sgn = blockIdx.x == 0 ? 1.0 : -1.0;
  const long long ns = g.nsite, pr = g.plane_r, base = (long long)z * pr;
  const double LxLy = (double)pr;
  if (de != 0.0) {
    double s = 0.0;
    for (long long i = threadIdx.x; i < 3 * pr; i += blockDim.x) {
      const long long j = base + i % pr;
      const T q = p[(i / pr) * ns + j];
      s += (double)q * q * (site_minv ? (double)site_minv[j] : layer_minv[z]);
    }
    const double n_layer = layer_nsum ? layer_nsum[z] : (layer_sump[z] ? LxLy : 0.0);
    const double e = block_sum(s) / 2 * LxLy / n_layer;
    const T f = (T)sqrt((e + sgn * LxLy * de) / e);
    for (long long i = threadIdx.x; i < 3 * pr; i += blockDim.x) p[(i / pr) * ns + base + i % pr] *= f;
  }
  if (dea != 0.0 && pa != nullptr) {
    double s = 0.0;
    for (long long i = threadIdx.x; i < 3 * pr; i += blockDim.x) {
      const long long j = base + i % pr;
      const T q = pa[(i / pr) * ns + j];
      s += (double)q * q * (site_macou ? (double)site_macou[j] : layer_macou[z]);
    }
    const double e = block_sum(s) / 2;
    const T f = (T)sqrt((e + sgn * LxLy * dea) / e);
    for (long long i = threadIdx.x; i < 3 * pr; i += blockDim.x) pa[(i / pr) * ns + base + i % pr] *= f;
  }
}

// p <- scale p on every site (velocity_scaling.F:79-83)
template <typename T>
__global__ void __launch_bounds__(256) k_scale(T* __restrict__ p, const double* scale, long long n) {
  const T f = (T)(*scale);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    p[i] = f * p[i];
}

// Opening half of a Nose-Poincare step in one sweep: the kick (35a)
// p <- p - kick_coef F and the drift (35c) u <- u + drift p m^-1
// (nose-poincare.F:24-53).  Both coefficients come from the previous closing
// tail, which already solved (38) with the kinetic energy of the kicked p.
// wave (wave_module.F:8-67): the field added at step i_step.  The
// triangular waves divide by period/4.0, a default-kind (single precision)
// real in the reference, so the quarter period is rounded to float.
__host__ __device__ inline void wave_field(int type, long long i_step, int n_thermalize, int period,
                                           const double a[3], double out[3]) {
  if (a[0] == 0.0 && a[1] == 0.0 && a[2] == 0.0) {
    for (int k = 0; k < 3; ++k) out[k] = a[k];
    return;
  }
  if (type == 1 || type == 2) {  // triangular_cos, triangular_sin
    long long i = i_step - n_thermalize;
    if (i < 0) i = 0;
    const long long P = period;
    const long long it = (type == 1) ? llabs(i % P - P / 2) - P / 4 : llabs((i + 3 * P / 4) % P - P / 2) - P / 4;
    const double tmp = (double)it;
    const float quarter = (float)period / 4.0f;
    for (int k = 0; k < 3; ++k) out[k] = a[k] * tmp / (double)quarter;
  } else if (type == 3 || type == 4) {  // ramping_on, ramping_off
    for (int k = 0; k < 3; ++k) {
      if (type == 3) out[k] = (i_step < period) ? a[k] * (double)i_step / period : a[k];
      else out[k] = (i_step < period) ? a[k] * (double)(period - i_step) / period : 0.0;
    }
  } else {
    for (int k = 0; k < 3; ++k) out[k] = a[k];
  }
}

// fg_set_uniform_E and the thermostat of fg_set_state: the values travel as
// arguments of the launch (a copy from pinned memory took 2 us longer, and
// its source had to stay untouched until it had run).
__global__ void k_set_field(DevScalars* sc, double e0, double e1, double e2) {
  if (threadIdx.x == 0) {
    sc->E[0] = e0;
    sc->E[1] = e1;
    sc->E[2] = e2;
  }
}
__global__ void k_set_thermostat(DevScalars* sc, double s, double pi, double H0, double kick_coef) {
  if (threadIdx.x == 0) {
    sc->s = s;
    sc->pi = pi;
    sc->H0 = H0;
    sc->kick_coef = kick_coef;
  }
}

// Start of a step under the device-side field schedule: the step counter
// advances and the uniform field becomes that step's wave value
// (molecular-dynamics.F:66-76, before the step's force evaluation).
__device__ inline void wave_step(const Phys* __restrict__ ph, DevScalars* sc) {
  const long long i = sc->i_step + 1;
  sc->i_step = i;
  double E[3];
  wave_field(ph->wave_type, i, ph->wave_n_thermalize, ph->wave_period, ph->wave_amp, E);
  for (int k = 0; k < 3; ++k) sc->E[k] = E[k];
}
// in front of the steps whose first kernel is not k_kick_drift
__global__ void k_wave_step(const Phys* __restrict__ ph, DevScalars* sc) {
  if (blockIdx.x == 0 && threadIdx.x == 0) wave_step(ph, sc);
}

template <typename T>
__global__ void __launch_bounds__(256) k_kick_drift(T* __restrict__ p, T* __restrict__ u, const T* __restrict__ F,
                                                    DevScalars* sc, Geom g,
                                                    const double* __restrict__ layer_minv,
                                                    const T* __restrict__ site_minv, const Phys* __restrict__ wave,
                                                    int gap_id, const RepArgs* __restrict__ grp) {
  pdl_launch();  // by default one resident wave, with nothing of this grid left to schedule
  pdl_wait();
  if (grp) {
    const RepArgs& a = grp[blockIdx.y];
    p = (T*)a.p;
    u = (T*)a.u;
    F = (const T*)a.F;
    sc = a.sc;
    layer_minv = a.layer_minv;
  }
  if (wave != nullptr && blockIdx.x == 0 && threadIdx.x == 0) wave_step(wave, sc);
  // gap_id: -1 for no film.  Film: every layer's momenta are kicked, the source layers'
  // dipoles drift and are written to their partners' layer as well
  auto partner = [&](int z) { return gap_id < 0 ? z : film_partner(z, g.Lz, gap_id); };
  const long long ns = g.nsite;
  const StepCoef<T> ck(sc->kick_coef);
  const double cd = sc->pend_drift;
  constexpr int NV = V16<T>::n;
  using AV = V16<T>;
  const long long stride = (long long)gridDim.x * blockDim.x;
  if (g.plane_r % NV == 0 && site_minv == nullptr) {
    for (long long iv = (long long)blockIdx.x * blockDim.x + threadIdx.x; iv < ns / NV; iv += stride) {
      const long long i = iv * NV;
      const int z = (int)(i / g.plane_r), zd = partner(z);
      const StepCoef<T> f(cd * layer_minv[z]);
      V16<T> x[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        V16<T> q = ldv(p + a * ns + i);
        x[a] = zd >= z ? ldv(u + a * ns + i) : q;  // not an image's u: its source is writing it
        const V16<T> y = ldv(F + a * ns + i);
#pragma unroll
        for (int l = 0; l < NV; ++l) {
          q.v[l] = q.v[l] - ck * y.v[l];
          x[a].v[l] = x[a].v[l] + f * q.v[l];
        }
        stv(p + a * ns + i, q);
        if (zd >= z) stv(u + a * ns + i, x[a]);
      }
      if (zd > z) {
        const long long d = i + (long long)(zd - z) * g.plane_r;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
#pragma unroll
          for (int l = 0; l < NV; ++l) x[a].v[l] = a < 2 ? -x[a].v[l] : x[a].v[l];
          stv(u + a * ns + d, x[a]);
        }
      }
    }
  } else {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < ns; i += stride) {
      const int z = (int)(i / g.plane_r), zd = partner(z);
      const StepCoef<T> f(cd * (site_minv ? (double)site_minv[i] : layer_minv[z]));
      const long long d = i + (long long)(zd - z) * g.plane_r;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const T q = p[a * ns + i] - ck * F[a * ns + i];
        p[a * ns + i] = q;
        if (zd >= z) {
          const T x = u[a * ns + i] + f * q;
          u[a * ns + i] = x;
          if (zd > z) u[a * ns + d] = a < 2 ? -x : x;
        }
      }
    }
  }
}

// Closing kick of a Nose-Poincare step (35f), p <- p - dt/2 s_{n+1} F
// (nose-poincare.F:66-71), with per-block masked sums of p^2/m, p.F/m and
// F^2/m of the new p for np_close_tail.  Block 0 first finishes the force
// evaluation of this step (energies from k_assemble's partials, commit of the
// prepared half step, (35e)); the last block to arrive, after block 0, runs
// np_close_tail.  PREP: no kick and no prologue; the sums of the current
// state prepare the first step after the state or the thermostat was set.
template <typename T, bool PREP>
__global__ void __launch_bounds__(256) k_kick_close(T* __restrict__ p, const T* __restrict__ F, Geom g,
                                                    const double* __restrict__ layer_minv,
                                                    const unsigned char* __restrict__ layer_sump,
                                                    double* __restrict__ part, unsigned int* done,
                                                    const Phys* __restrict__ ph, DevScalars* sc,
                                                    const double* __restrict__ part_r, int nblk_r,
                                                    const T* __restrict__ site_minv = nullptr,
                                                    const unsigned char* __restrict__ site_sump = nullptr,
                                                    DevScalars* host = nullptr) {
  pdl_launch();  // by default one resident wave, with nothing of this grid left to schedule
  pdl_wait();
  if (!PREP && blockIdx.x == 0) force_energies_tail(ph, sc, part_r, nblk_r, true);
  const long long ns = g.nsite;
  // pend_kick_f is not changed by block 0's commit
  const StepCoef<T> c(PREP ? 0.0 : __ldcg(&sc->pend_kick_f));
  double acc[3] = {0.0, 0.0, 0.0};
  constexpr int NV = V16<T>::n;
  using AV = V16<T>;
  const long long stride = (long long)gridDim.x * blockDim.x;
  if (g.plane_r % NV == 0 && site_minv == nullptr && site_sump == nullptr) {
    for (long long iv = (long long)blockIdx.x * blockDim.x + threadIdx.x; iv < ns / NV; iv += stride) {
      const long long i = iv * NV;
      const int z = (int)(i / g.plane_r);
      // the vector's 3 NV products summed in T, then accumulated in FP64
      T pp = 0, pf = 0, ff = 0;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        V16<T> q = ldv(p + a * ns + i);
        const V16<T> y = ldv(F + a * ns + i);
#pragma unroll
        for (int l = 0; l < NV; ++l) {
          if (!PREP) q.v[l] = q.v[l] - c * y.v[l];
          pp += q.v[l] * q.v[l];
          pf += q.v[l] * y.v[l];
          ff += y.v[l] * y.v[l];
        }
        if (!PREP) stv(p + a * ns + i, q);
      }
      if (layer_sump[z]) {
        const double mi = layer_minv[z];
        acc[0] += (double)pp * mi;
        acc[1] += (double)pf * mi;
        acc[2] += (double)ff * mi;
      }
    }
  } else {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < ns; i += stride) {
      const int z = (int)(i / g.plane_r);
      double pp = 0.0, pf = 0.0, ff = 0.0;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        T q = p[a * ns + i];
        const T y = F[a * ns + i];
        if (!PREP) {
          q = q - c * y;
          p[a * ns + i] = q;
        }
        pp += (double)q * q;
        pf += (double)q * y;
        ff += (double)y * y;
      }
      if (site_sump ? site_sump[i] != 0 : layer_sump[z] != 0) {
        const double mi = site_minv ? (double)site_minv[i] : layer_minv[z];
        acc[0] += pp * mi;
        acc[1] += pf * mi;
        acc[2] += ff * mi;
      }
    }
  }
  block_partials<3>(acc, part, blockIdx.x);
  if (is_last_block(done)) np_close_tail(ph, sc, part, gridDim.x, !PREP, host);
}

// u <- u + coef * p * m^-1 (nose-poincare.F:41-53, leapfrog.F:104-114)
template <typename T>
__global__ void __launch_bounds__(256) k_drift(T* __restrict__ u, const T* __restrict__ p, const double* coef, Geom g,
                                               const double* __restrict__ layer_minv,
                                               const T* __restrict__ site_minv, const SecondField<T> acou) {
  if (blockIdx.y == 1) {
    u = acou.u;
    p = acou.p;
    layer_minv = acou.layer_minv;
    site_minv = acou.site_minv;
  }
  const long long ns = g.nsite;
  const double c = *coef;
  constexpr int NV = V16<T>::n;
  using AV = V16<T>;
  const long long stride = (long long)gridDim.x * blockDim.x;
  if (g.plane_r % NV == 0 && site_minv == nullptr) {
    for (long long iv = (long long)blockIdx.x * blockDim.x + threadIdx.x; iv < ns / NV; iv += stride) {
      const long long i = iv * NV;
      const StepCoef<T> f(c * layer_minv[(int)(i / g.plane_r)]);
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        V16<T> x = ldv(u + a * ns + i);
        const V16<T> q = ldv(p + a * ns + i);
#pragma unroll
        for (int l = 0; l < NV; ++l) x.v[l] = x.v[l] + f * q.v[l];
        stv(u + a * ns + i, x);
      }
    }
  } else {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < ns; i += stride) {
      const int z = (int)(i / g.plane_r);
      const StepCoef<T> f(c * (site_minv ? (double)site_minv[i] : layer_minv[z]));
      u[i] = u[i] + f * p[i];
      u[ns + i] = u[ns + i] + f * p[ns + i];
      u[2 * ns + i] = u[2 * ns + i] + f * p[2 * ns + i];
    }
  }
}

// Film mirror (mirror.F:9-36): layer z' = Lz-1-z (gap_id = 0) or Lz-z gets
// (-f_x, -f_y, f_z) of layer z.
template <typename T>
__global__ void k_mirror(T* __restrict__ f, Geom g, int gap_id) {
  const long long ns = g.nsite;
  const int z0 = (gap_id == 0) ? 0 : 1;
  const int z1 = (gap_id == 0) ? g.Lz / 2 : (g.Lz + 1) / 2;  // exclusive
  const long long n = (long long)(z1 - z0) * g.plane_r;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int z = z0 + (int)(i / g.plane_r);
    const long long r = i % g.plane_r;
    const int zd = (gap_id == 0) ? g.Lz - 1 - z : g.Lz - z;
    const long long s = (long long)z * g.plane_r + r, d = (long long)zd * g.plane_r + r;
    f[d] = -f[s];
    f[ns + d] = -f[ns + s];
    f[2 * ns + d] = f[2 * ns + s];
  }
}

// KE of the current momenta without changing them.
template <typename T>
__global__ void __launch_bounds__(256) k_ke_only(const T* __restrict__ p, Geom g, const double* __restrict__ layer_minv,
                                                 const unsigned char* __restrict__ layer_sump, double* __restrict__ part,
                                                 const T* __restrict__ site_minv = nullptr,
                                                 const unsigned char* __restrict__ site_sump = nullptr) {
  const long long ns = g.nsite;
  double acc[1] = {0.0};
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < ns; i += (long long)gridDim.x * blockDim.x) {
    const int z = (int)(i / g.plane_r);
    if (site_sump ? site_sump[i] != 0 : layer_sump[z] != 0) {
      const double mi = site_minv ? (double)site_minv[i] : layer_minv[z];
      const double p0 = p[i], p1 = p[ns + i], p2 = p[2 * ns + i];
      acc[0] += p0 * p0 * mi + p1 * p1 * mi + p2 * p2 * mi;
    }
  }
  block_partials<1>(acc, part, blockIdx.x);
}

__global__ void __launch_bounds__(RED_THREADS) k_ke_finish(const Phys* __restrict__ ph, DevScalars* sc,
                                                           const double* __restrict__ part, int nblk) {
  double v = reduce_partials(part, nblk, 1, 0);
  if (threadIdx.x != 0) return;
  sc->ke_sum = v;
  sc->e[E_DIPO] = ke_from(ph, v);
}

// add_to_Average reductions (average_module.F:86-121): masked sum of u and of
// Z* u per component.  part[b*6 + q]: q = 0..2 sum u, 3..5 sum Z* u.
template <typename T>
__global__ void __launch_bounds__(256) k_avg_sums(const T* __restrict__ u, Geom g, double Zs,
                                                  const unsigned char* __restrict__ layer_sump, double* __restrict__ part,
                                                  const unsigned char* __restrict__ site_sump = nullptr,
                                                  const T* __restrict__ site_zstar = nullptr) {
  const long long ns = g.nsite;
  double acc[6] = {0, 0, 0, 0, 0, 0};
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < ns; i += (long long)gridDim.x * blockDim.x) {
    const int z = (int)(i / g.plane_r);
    if (site_sump ? !site_sump[i] : !layer_sump[z]) continue;
    if (site_zstar) Zs = site_zstar[i];
    const double a = u[i], b = u[ns + i], c = u[2 * ns + i];
    acc[0] += a;
    acc[1] += b;
    acc[2] += c;
    acc[3] += Zs * a;
    acc[4] += Zs * b;
    acc[5] += Zs * c;
  }
  block_partials<6>(acc, part, blockIdx.x);
}

__global__ void __launch_bounds__(RED_THREADS) k_avg_finish(double* out6, const double* __restrict__ part, int nblk) {
  for (int q = 0; q < 6; ++q) {
    double v = reduce_partials(part, nblk, 6, q);
    if (threadIdx.x == 0) out6[q] = v;
  }
}

// One row of a context's sample series (fg_sample): the six masked sums of
// k_avg_sums (sum u, sum Z* u), then, from the scalars of the last step, the
// potential energy, the true kinetic energy KE / s^2, s, pi and the six
// homogeneous strains: the per-step quantities add_to_Average accumulates
// (average_module.F:75-128), kept as a series so that their block errors
// can be taken afterwards.
constexpr int kSampleCols = FG_SAMPLE_COLS;
constexpr int kSampleCap = FG_SAMPLE_CAP;  // rows a context holds between reads
__global__ void __launch_bounds__(RED_THREADS) k_sample_row(double* __restrict__ row, const double* __restrict__ part,
                                                            int nblk, const DevScalars* __restrict__ sc) {
  for (int q = 0; q < 6; ++q) {
    double v = reduce_partials(part, nblk, 6, q);
    if (threadIdx.x == 0) row[q] = v;
  }
  if (threadIdx.x == 0) {
    const double s = sc->s;
    row[6] = sum_potential(sc->e);
    row[7] = sc->e[E_DIPO] / (s * s);
    row[8] = s;
    row[9] = sc->pi;
    for (int i = 0; i < 6; ++i) row[10 + i] = sc->strain[i];
  }
}

template <typename T>
__global__ void k_accumulate(double* __restrict__ acc, const T* __restrict__ u, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    acc[i] += (double)u[i];
}

// ------------------------------------------------------- layout conversion
// Padded column-major (nc, 0:NXP-1, 0:NYP-1, 0:Lz-1) FP64 <-> [nc][z][y][x] T.
template <typename T>
__global__ void k_fortran_to_soa(T* __restrict__ dst, const double* __restrict__ src, Geom g, int nc, int NXP, int NYP) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < g.nsite; i += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(i % g.Lx);
    const long long r = i / g.Lx;
    const int y = (int)(r % g.Ly), z = (int)(r / g.Ly);
    const long long s = (long long)nc * ((long long)x + (long long)NXP * ((long long)y + (long long)NYP * z));
    for (int c = 0; c < nc; ++c) dst[(long long)c * g.nsite + i] = (T)src[s + c];
  }
}

template <typename T>
__global__ void k_soa_to_fortran(double* __restrict__ dst, const T* __restrict__ src, Geom g, int nc, int NXP, int NYP) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < g.nsite; i += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(i % g.Lx);
    const long long r = i / g.Lx;
    const int y = (int)(r % g.Ly), z = (int)(r / g.Ly);
    const long long s = (long long)nc * ((long long)x + (long long)NXP * ((long long)y + (long long)NYP * z));
    for (int c = 0; c < nc; ++c) dst[s + c] = (double)src[(long long)c * g.nsite + i];
  }
}

// The same for a field held as a hi/lo pair (the mixed path's force after a
// force evaluation that kept its FP32 residual): dst = hi + lo in FP64.
template <typename T>
__global__ void k_soa2_to_fortran(double* __restrict__ dst, const T* __restrict__ hi, const T* __restrict__ lo, Geom g,
                                  int nc, int NXP, int NYP) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < g.nsite; i += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(i % g.Lx);
    const long long r = i / g.Lx;
    const int y = (int)(r % g.Ly), z = (int)(r / g.Ly);
    const long long s = (long long)nc * ((long long)x + (long long)NXP * ((long long)y + (long long)NYP * z));
    for (int c = 0; c < nc; ++c) dst[s + c] = (double)hi[(long long)c * g.nsite + i] + (double)lo[(long long)c * g.nsite + i];
  }
}

// ------------------------------------------------------- table construction
// Real-space Ewald sum of dipole-dipole-long-range.F:106-149 per site:
// self term at R = 0, images jz, jy, jx in -1-max..max, per element +B on
// the diagonal then -rn_a rn_b C.  Output [6][z][y][x]: xx, yy, zz, yz, zx, xy.
__global__ void k_ewald_real(double* __restrict__ out, Geom g, double a0, double kappa, int max_x, int max_y, int max_z) {
  const double two_over_sqrtpi = 1.12837916709551257390;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < g.nsite; i += (long long)gridDim.x * blockDim.x) {
    const int ix = (int)(i % g.Lx);
    const long long r = i / g.Lx;
    const int iy = (int)(r % g.Ly), iz = (int)(r / g.Ly);
    double t[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
    if (i == 0) {
      const double self = -2 * two_over_sqrtpi * kappa * kappa * kappa / 3;
      t[0][0] = t[1][1] = t[2][2] = self;
    }
    for (int jz = -1 - max_z; jz <= max_z; ++jz)
      for (int jy = -1 - max_y; jy <= max_y; ++jy)
        for (int jx = -1 - max_x; jx <= max_x; ++jx) {
          if (jx == 0 && jy == 0 && jz == 0 && i == 0) continue;
          const double rn[3] = {ix * a0 + jx * (g.Lx * a0), iy * a0 + jy * (g.Ly * a0), iz * a0 + jz * (g.Lz * a0)};
          const double rr = rn[0] * rn[0] + rn[1] * rn[1] + rn[2] * rn[2];
          const double rnorm = sqrt(rr);
          const double ec = erfc(kappa * rnorm), ex = exp(-kappa * kappa * rr);
          const double B = ec / (rnorm * rr) + two_over_sqrtpi * kappa * ex / rr;
          const double C = (3 * ec / (rnorm * rr) + two_over_sqrtpi * kappa * ex * (2 * kappa * kappa + 3 / rr)) / rr;
#pragma unroll
          for (int b = 0; b < 3; ++b)
#pragma unroll
            for (int a = 0; a < 3; ++a) {
              if (a == b) t[a][b] = t[a][b] + B;
              t[a][b] = t[a][b] - rn[a] * rn[b] * C;
            }
        }
    out[i] = t[0][0];
    out[g.nsite + i] = t[1][1];
    out[2 * g.nsite + i] = t[2][2];
    out[3 * g.nsite + i] = t[1][2];
    out[4 * g.nsite + i] = t[2][0];
    out[5 * g.nsite + i] = t[0][1];
  }
}

// Per (kx tile, ky slot) of the six forward-transformed real-space sums:
// DIF along z, then L = (Re FFT + reciprocal sum) * Hartree*Bohr/eps_inf
// (dipole-dipole-long-range.F:151-206), D = (S + Z*^2 L)/N in the table
// layout, and L in FP64 for inspection.
template <typename T>
__global__ void __launch_bounds__(256) k_z_ewald_pack(const cplx<double>* __restrict__ spec, T* __restrict__ dtab,
                                                      double* __restrict__ L64, Geom g, FftPlan pz,
                                                      const cplx<double>* __restrict__ twz, KMaps km,
                                                      const Phys* __restrict__ ph, double a0, double kappa,
                                                      double eps_inf, int max_x, int max_y, int max_z, ZTiles zt) {
  FG_DYN_SMEM(smem_raw);
  cplx<double>* buf = reinterpret_cast<cplx<double>*>(smem_raw);
  const int Lz = g.Lz, CW = zt.CW;
  z_tile_load<double>(buf, spec, g, zt, 6);
  {
    Batch B{6 * CW, CW, 1, Lz * CW, CW, true};
    fft_forward<double>(buf, B, pz, twz, 6 * Lz * CW);
  }
  const double pi = 3.14159265358979323846;
  const double four_pi_over_v = 4 * pi / (a0 * a0 * a0);
  const double two_pi_over_a = 2 * pi / a0;
  const double four_kappa2 = 4 * kappa * kappa;
  const double scale = 14.399644 / eps_inf;  // HARTREE_BOHR (define.h:32)
  for (int idx = threadIdx.x; idx < Lz * CW; idx += blockDim.x) {
    const int zs = idx / CW, cw = idx - zs * CW;
    int col, yslot;
    if (!tile_pencil(zt, g, cw, &col, &yslot)) continue;
    const int ky = km.revy[yslot];
    const int kx = km.revx[col], kz = km.revz[zs];
    double k[3];
    k[2] = (double)kz / g.Lz;
    if (k[2] > 0.5) k[2] = k[2] - 1.0;
    k[1] = (double)ky / g.Ly;
    if (k[1] > 0.5) k[1] = k[1] - 1.0;
    k[0] = (double)kx / g.Lx;
    double Lt[6];
    for (int q = 0; q < 6; ++q) Lt[q] = buf[(q * Lz + zs) * CW + cw].x;
    const int qa[6] = {0, 1, 2, 1, 2, 0}, qb[6] = {0, 1, 2, 2, 0, 1};
    for (int q = 0; q < 6; ++q) {
      double t = Lt[q];
      for (int nz = -max_z; nz <= max_z; ++nz) {
        const double kG2 = two_pi_over_a * (k[2] + nz);
        for (int ny = -max_y; ny <= max_y; ++ny) {
          const double kG1 = two_pi_over_a * (k[1] + ny);
          for (int nx = -max_x; nx <= max_x; ++nx) {
            if (kx == 0 && ky == 0 && kz == 0 && nx == 0 && ny == 0 && nz == 0) continue;
            const double kG0 = two_pi_over_a * (k[0] + nx);
            const double kG[3] = {kG0, kG1, kG2};
            const double kGkG = kG0 * kG0 + kG1 * kG1 + kG2 * kG2;
            t = t + four_pi_over_v * kG[qa[q]] * kG[qb[q]] * exp(-kGkG / four_kappa2) / kGkG;
          }
        }
      }
      Lt[q] = t * scale;
    }
    const double2 tx = km.trx[kx], ty = km.try_[ky], tz = km.trz[kz];
    const double cc[3] = {tx.x, ty.x, tz.x}, ss[3] = {tx.y, ty.y, tz.y};
    double S[6];
    short_range_k(ph->j, ph->kap2x2, cc, ss, S);
    const long long tpos = ((long long)yslot * Lz + zs) * g.KXP + col;
    const double z2 = ph->Zstar * ph->Zstar;
    for (int q = 0; q < 6; ++q) {
      dtab[tab_index<T>(tpos, q)] = (T)((S[q] + z2 * Lt[q]) * ph->Ninv);
      if (L64) L64[tpos * 6 + q] = Lt[q];
    }
  }
}

// dst = (T)(src * scale): the L/N table of the per-site Z* path
template <typename T>
__global__ void __launch_bounds__(256) k_table_scale(T* __restrict__ dst, const double* __restrict__ src, double scale,
                                                     long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    dst[tab_index<T>(i / 6, (int)(i % 6))] = (T)(src[i] * scale);
}

// c_k_modulation_k = modulation_constant * k * r2c(modulation_R) (elastic.F:212-225)
template <typename T>
__global__ void __launch_bounds__(256) k_z_modulation_pack(const cplx<double>* __restrict__ spec, cplx<T>* __restrict__ ck,
                                                           Geom g, FftPlan pz, const cplx<double>* __restrict__ twz,
                                                           KMaps km, double mod_const, ZTiles zt) {
  FG_DYN_SMEM(smem_raw);
  cplx<double>* buf = reinterpret_cast<cplx<double>*>(smem_raw);
  const int Lz = g.Lz, CW = zt.CW;
  z_tile_load<double>(buf, spec, g, zt, 1);
  {
    Batch B{CW, CW, 1, Lz * CW, CW, true};
    fft_forward<double>(buf, B, pz, twz, Lz * CW);
  }
  for (int idx = threadIdx.x; idx < Lz * CW; idx += blockDim.x) {
    const int zs = idx / CW, cw = idx - zs * CW;
    int col, yslot;
    if (!tile_pencil(zt, g, cw, &col, &yslot)) continue;
    const int ky = km.revy[yslot];
    const int kx = km.revx[col], kz = km.revz[zs];
    const double kv[3] = {km.kvx[kx], km.kvy[ky], km.kvz[kz]};
    const cplx<double> mk_ = buf[zs * CW + cw];
    const long long tpos = ((long long)yslot * Lz + zs) * g.KXP + col;
    for (int a = 0; a < 3; ++a)
      ck[tpos * 3 + a] = mk<cplx<T>>((T)(mod_const * kv[a] * mk_.x), (T)(mod_const * kv[a] * mk_.y));
  }
}

}  // namespace fg
