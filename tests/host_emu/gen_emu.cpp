// Host emulation of the runtime two-stage kernels (k_xy_fwd_gen, k_xy_inv_gen
// and k_z_lane<T, 0, 0> of feram_b200/csrc/fg_kernels.cuh) behind
// kernel_emu.h, on shapes that reach every radix of lane_split, odd Lx/2, row
// groups cut by Ly and tiles cut by Lx/2 and Ly.
//
// xy: the forward pass against a direct 2D DFT (x slot = kx, y slots in the
// digit-reversed order of RY1 x RY2), the inverse back to Lx Ly times the
// planes.  z: with D = 1 and no strain coupling the k-space step multiplies
// components 0..2 by one and zeroes the strain components, so the pass must
// return Lz times components 0..2 and zeros; its short-range energy with
// S(k) = 1 is sum w |u|^2 by Parseval.
//
// Output: "<case> <error> <error>" lines, relative.
#include "kernel_emu.h"
#include "feram_gpu.h"
#include "fg_kernels.cuh"

#include <algorithm>
#include <cmath>
#include <complex>
#include <cstdio>
#include <random>
#include <vector>

using namespace fg;
using cld = std::complex<long double>;

template <typename T>
std::vector<cplx<T>> twiddles(int n) {
  std::vector<cplx<T>> w((size_t)n);
  const long double pi = 3.14159265358979323846264338327950288L;
  for (int k = 0; k < n; ++k) w[(size_t)k] = mk<cplx<T>>((T)std::cos(-2 * pi * k / n), (T)std::sin(-2 * pi * k / n));
  return w;
}
std::vector<cld> roots(int n) {
  std::vector<cld> w((size_t)n);
  const long double pi = 3.14159265358979323846264338327950288L;
  for (int k = 0; k < n; ++k) w[(size_t)k] = std::polar(1.0L, -2.0L * pi * (long double)k / (long double)n);
  return w;
}
// slot -> frequency of the two stages r1, r2
std::vector<int> two_stage_rev(int r1, int r2) {
  std::vector<int> rev((size_t)(r1 * r2));
  for (int p = 0; p < r1 * r2; ++p) rev[(size_t)p] = p / r2 + r1 * (p % r2);
  return rev;
}
Geom geom(int Lx, int Ly, int Lz) {
  Geom g{};
  g.Lx = Lx;
  g.Ly = Ly;
  g.Lz = Lz;
  g.m = Lx / 2;
  g.NKX = g.m + 1;
  g.KXP = (g.NKX + 15) / 16 * 16;
  g.plane_r = (long long)Lx * Ly;
  g.plane_c = (long long)Ly * g.KXP;
  g.nsite = (long long)Lx * Ly * Lz;
  g.ncplx = (long long)Lz * g.plane_c;
  g.nkpos = g.ncplx;
  return g;
}

template <typename T>
void xy_case(int Lx, int Ly, bool zstar = false) {
  const int Lz = 1, W = kLanes<T>, nc = zstar ? 12 : 9;
  const Geom g = geom(Lx, Ly, Lz);
  XyGeo h{};
  if (!lane_split(Lx, true, &h.R1, &h.R2) || !lane_split(Ly, false, &h.RY1, &h.RY2)) {
    std::printf("xy_nosplit_%dx%d nan nan\n", Lx, Ly);
    return;
  }
  h.NQ = (Ly + 2 * W - 1) / (2 * W);
  h.NJ = (g.m + W - 1) / W;
  h.QS = Lx + 1;
  h.JS = Ly | 1;
  h.dR2 = fast_div(h.R2);
  h.dNQ = fast_div(h.NQ);
  h.dNJ = fast_div(h.NJ);
  h.nt = (h.R1 / 2 * h.NQ + 31) / 32 * 32;
  h.smem = std::max(h.NQ * h.QS, h.NJ * h.JS) * 16;
  const std::vector<int> revy = two_stage_rev(h.RY1, h.RY2);
  std::vector<int> posm((size_t)(g.m + 2 * Ly), 0);
  for (int s = 0; s < Ly; ++s) {
    posm[(size_t)(g.m + s)] = revy[(size_t)s];
    posm[(size_t)(g.m + Ly + revy[(size_t)s])] = s;
  }
  const auto twx = twiddles<T>(Lx), twy = twiddles<T>(Ly);
  std::mt19937_64 gen(5u + (unsigned)(Lx * 1000 + Ly));
  std::uniform_real_distribution<double> dist(-0.2, 0.2);
  std::vector<T> u((size_t)(3 * g.nsite)), zs((size_t)g.nsite);
  for (auto& v : u) v = (T)dist(gen);
  for (auto& v : zs) v = (T)(1 + dist(gen));
  auto fld = [&](int c, long long i) -> long double {
    const long double x = u[(size_t)i], y = u[(size_t)(g.nsite + i)], z = u[(size_t)(2 * g.nsite + i)];
    const long double f[9] = {x, y, z, x * x, y * y, z * z, y * z, z * x, x * y};
    return c < 9 ? f[c] : (long double)zs[(size_t)i] * f[c - 9];
  };
  const T nan = std::nan("");
  std::vector<cplx<T>> spec((size_t)(nc * g.ncplx), mk<cplx<T>>(nan, nan));
  emu::launch(k_xy_fwd_gen<T, SRC_U9>, dim3((unsigned)Lz, (unsigned)nc, 1), dim3((unsigned)h.nt), (size_t)h.smem,
              (const T*)u.data(), spec.data(), g, h, (const cplx<T>*)twx.data(), (const cplx<T>*)twy.data(),
              (const int*)posm.data(), (const T*)(zstar ? zs.data() : nullptr), 9, (const RepArgs*)nullptr);
  const auto wx = roots(Lx), wy = roots(Ly);
  double ef = 0, xmax = 0, fmax = 0;
  std::vector<cld> row((size_t)Ly * (g.m + 1));
  for (int c = 0; c < nc; ++c) {
    for (int y = 0; y < Ly; ++y)
      for (int k = 0; k <= g.m; ++k) {
        cld s = 0;
        for (int x = 0; x < Lx; ++x) {
          const long double f = fld(c, (long long)y * Lx + x);
          fmax = std::max(fmax, (double)std::fabs(f));
          s += f * wx[(size_t)((k * x) % Lx)];
        }
        row[(size_t)y * (g.m + 1) + k] = s;
      }
    for (int sl = 0; sl < Ly; ++sl)
      for (int k = 0; k <= g.m; ++k) {
        cld s = 0;
        for (int y = 0; y < Ly; ++y) s += row[(size_t)y * (g.m + 1) + k] * wy[(size_t)((revy[(size_t)sl] * y) % Ly)];
        const cplx<T> v = spec[(size_t)(c * g.ncplx + (long long)sl * g.KXP + k)];
        const double d = (double)std::abs(cld(v.x, v.y) - s);
        ef = std::max(ef, std::isfinite(d) ? d : 1e300);
        xmax = std::max(xmax, (double)std::abs(s));
      }
  }
  std::vector<T> out((size_t)(nc * g.nsite), nan);
  emu::launch(k_xy_inv_gen<T>, dim3((unsigned)Lz, (unsigned)nc, 1), dim3((unsigned)h.nt), (size_t)h.smem,
              (const cplx<T>*)spec.data(), out.data(), g, h, (const cplx<T>*)twx.data(), (const cplx<T>*)twy.data(),
              (const int*)posm.data(), (const Phys*)nullptr, (DevScalars*)nullptr, (const double*)nullptr, 0,
              (const RepArgs*)nullptr);
  double eb = 0;
  for (int c = 0; c < nc; ++c)
    for (long long i = 0; i < g.nsite; ++i) {
      const double d = (double)std::fabs((long double)out[(size_t)(c * g.nsite + i)] / (Lx * Ly) - fld(c, i));
      eb = std::max(eb, std::isfinite(d) ? d : 1e300);
    }
  std::printf("xy_%s_%dx%d%s %.3e %.3e\n", W == 2 ? "f32" : "f64", Lx, Ly, zstar ? "_zstar" : "", ef / xmax, eb / fmax);
  std::fflush(stdout);
}

template <typename T>
void z_case(int Lx, int Ly, int Lz, int pw) {
  const int W = kLanes<T>;
  const Geom g = geom(Lx, Ly, Lz);
  ZGeo h{};
  if (!lane_split(Lz, false, &h.R1, &h.R2)) {
    std::printf("z_nosplit_%d nan nan\n", Lz);
    return;
  }
  h.lpw = pw == 4 ? 2 : pw == 2 ? 1 : 0;
  h.d1 = fast_div(h.R1);
  h.d2 = fast_div(h.R2);
  const bool wn = W == 2 && g.m % 2 != 0;
  h.ncol = g.m + (wn ? 1 : 0);
  ZTiles zt{};
  zt.CW = pw * W;
  zt.ntx = (h.ncol + zt.CW - 1) / zt.CW;
  zt.nreg = zt.ntx * Ly;
  zt.nnyq = wn ? 0 : (Ly + zt.CW - 1) / zt.CW;
  const auto twz = twiddles<T>(Lz);
  std::vector<int> ix((size_t)g.NKX);
  for (int k = 0; k < g.NKX; ++k) ix[(size_t)k] = k;
  // wavevectors that keep K regular; S(k) = kap = 1
  std::vector<double> kx((size_t)g.NKX, 0.3), ky((size_t)Ly, 0.2), kz((size_t)Lz, 0.1);
  std::vector<double2> tx((size_t)g.NKX, make_double2(1, 0)), ty((size_t)Ly, make_double2(1, 0)), tz((size_t)Lz, make_double2(1, 0));
  KMaps km{};
  km.kvz_s = kz.data();
  km.trz_s = tz.data();
  km.kvx_s = kx.data();
  km.kvy_s = ky.data();
  km.trx_s = tx.data();
  km.try_s = ty.data();
  Phys ph{};
  ph.Ninv = 1;
  ph.kap2x2 = 1;
  ph.B11 = 1;
  ph.B44 = 1;
  std::vector<T> dtab((size_t)(6 * g.nkpos), (T)0);
  for (long long p = 0; p < g.nkpos; ++p)
    for (int q = 0; q < 3; ++q) dtab[(size_t)tab_index<T>(p, q)] = (T)1;
  std::mt19937_64 gen(9u + (unsigned)(Lx * 1000 + Ly * 10 + Lz));
  std::uniform_real_distribution<double> dist(-1, 1);
  std::vector<cplx<T>> spec((size_t)(9 * g.ncplx), mk<cplx<T>>((T)0, (T)0));
  for (int c = 0; c < 9; ++c)
    for (int r = 0; r < Lz * Ly; ++r)
      for (int k = 0; k <= g.m; ++k)
        spec[(size_t)(c * g.ncplx + (long long)r * g.KXP + k)] = mk<cplx<T>>((T)dist(gen), (T)dist(gen));
  const auto in = spec;
  std::vector<double> part((size_t)(NQ_K * (zt.nreg + zt.nnyq)), std::nan(""));
  DevScalars sc{};
  const size_t smem = (size_t)9 * Lz * pw * 16;
  emu::launch(k_z_lane<T, 0, 0, false>, dim3((unsigned)(zt.nreg + zt.nnyq), 1), dim3(256), smem, spec.data(),
              (const T*)dtab.data(), (const cplx<T>*)nullptr, (cplx<T>*)nullptr, g, h, (const cplx<T>*)twz.data(), km,
              (const Phys*)&ph, part.data(), &sc, zt, (const RepArgs*)nullptr);
  double e = 0, want = 0, got = 0;
  for (int c = 0; c < 9; ++c)
    for (int r = 0; r < Lz * Ly; ++r)
      for (int k = 0; k <= g.m; ++k) {
        const size_t i = (size_t)(c * g.ncplx + (long long)r * g.KXP + k);
        const cld w = c < 3 ? (long double)Lz * cld(in[i].x, in[i].y) : cld(0);
        const double d = (double)std::abs(cld(spec[i].x, spec[i].y) - w) / Lz;
        e = std::max(e, std::isfinite(d) ? d : 1e300);
        if (c < 3) want += (k == 0 || k == g.m ? 1 : 2) * Lz * (double)std::norm(cld(in[i].x, in[i].y));
      }
  for (int b = 0; b < zt.nreg + zt.nnyq; ++b) got += part[(size_t)(NQ_K * b)];
  const double ee = std::fabs(got - want) / want;
  std::printf("z_%s_%dx%dx%d_%d %.3e %.3e\n", W == 2 ? "f32" : "f64", Lx, Ly, Lz, pw, e, std::isfinite(ee) ? ee : 1e300);
  std::fflush(stdout);
}

template <typename T>
void all() {
  const int xy[][2] = {{4, 3}, {6, 5}, {10, 6}, {12, 9}, {18, 10}, {20, 12}, {24, 15}, {30, 18}, {32, 25}, {36, 27},
                       {40, 20}, {48, 30}, {50, 36}, {54, 45}, {60, 50}, {72, 40}, {80, 16}, {90, 8}, {96, 54}, {100, 60},
                       {108, 75}, {120, 4}, {128, 90}, {144, 24}, {160, 96}, {16, 160}, {8, 135}, {64, 100}, {20, 128}};
  for (auto& s : xy) xy_case<T>(s[0], s[1]);
  xy_case<T>(30, 18, true);
  const int z[][4] = {{4, 3, 3, 1}, {6, 5, 4, 2}, {10, 6, 5, 4}, {12, 5, 6, 4}, {20, 6, 8, 4}, {18, 4, 9, 2}, {16, 3, 10, 4},
                      {24, 3, 12, 4}, {14, 4, 15, 4}, {8, 6, 18, 2}, {8, 5, 20, 4}, {10, 3, 25, 2}, {12, 4, 27, 1}, {6, 4, 30, 4},
                      {8, 4, 36, 2}, {10, 4, 40, 4}, {6, 3, 45, 4}, {12, 3, 50, 4}, {4, 3, 54, 2}, {6, 3, 60, 4}, {8, 3, 72, 2},
                      {10, 3, 75, 2}, {4, 4, 80, 4}, {6, 4, 81, 2}, {12, 4, 90, 4}, {8, 4, 96, 4}, {6, 3, 100, 2},
                      {8, 3, 108, 4}, {4, 3, 120, 2}, {6, 3, 135, 4}, {8, 3, 144, 2}, {4, 3, 150, 4}, {6, 3, 160, 1},
                      {8, 3, 16, 1}, {8, 3, 24, 1}, {8, 3, 32, 1}, {8, 3, 48, 1}, {8, 3, 64, 1}, {6, 3, 128, 2}};
  for (auto& s : z) z_case<T>(s[0], s[1], s[2], s[3]);
}

int main() {
  all<double>();
  all<float>();
  return 0;
}
