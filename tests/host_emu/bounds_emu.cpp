// The bounds-checked build (FG_BOUNDS_CHECK) of the runtime x-y and k-space
// kernels of feram_b200/csrc/fg_kernels.cuh, emulated on the host behind
// kernel_emu.h: shapes as the library makes them record nothing; a shape whose
// strides, lengths or tile do not fit the arrays it is launched with is
// recorded.  The arrays here are larger than the kernels are told, so that a
// missed access stays inside them.
//
// Output: "<case> <recorded code> <expected code>" lines.
#define FG_BOUNDS_CHECK 1
#include "kernel_emu.h"
#include "feram_gpu.h"
#include "fg_kernels.cuh"

#include <algorithm>
#include <cstdio>
#include <functional>
#include <vector>

using namespace fg;

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
void report(const char* what, const char* kernel, int W, int a, int b, int c, int want) {
  std::printf("%s_%s_%s_%dx%dx%d %d %d\n", kernel, what, W == 2 ? "f32" : "f64", a, b, c, g_fg_err.code, want);
  std::fflush(stdout);
  g_fg_err = DevError{};
}

template <typename T>
void xy(int Lx, int Ly, const char* what, const std::function<void(Geom&, XyGeo&)>& plant) {
  constexpr int W = kLanes<T>;
  Geom g = geom(Lx, Ly, 1);
  XyGeo h{};
  lane_split(Lx, true, &h.R1, &h.R2);
  lane_split(Ly, false, &h.RY1, &h.RY2);
  h.NQ = (Ly + 2 * W - 1) / (2 * W);
  h.NJ = (g.m + W - 1) / W;
  h.QS = Lx + 1;
  h.JS = Ly | 1;
  h.nt = (h.R1 / 2 * h.NQ + 31) / 32 * 32;
  h.smem = std::max(h.NQ * h.QS, h.NJ * h.JS) * 16;
  const size_t room = (size_t)h.smem * 4;
  // a plane of one row group (column element) does not use that stride
  const bool unused = (what[0] == 'q' && h.NQ == 1) || (what[0] == 'j' && h.NJ == 1);
  const int want = *what == '-' || unused ? 0 : 1;
  plant(g, h);
  h.dR2 = fast_div(h.R2);
  h.dNQ = fast_div(h.NQ);
  h.dNJ = fast_div(h.NJ);
  std::vector<int> posm((size_t)(4 * (Lx + Ly)), 0);
  std::vector<cplx<T>> tw((size_t)(4 * (Lx + Ly)), mk<cplx<T>>((T)1, (T)0)), spec((size_t)(40 * g.ncplx + 4096));
  std::vector<T> f((size_t)(40 * g.nsite + 4096), (T)1);
  emu::launch(k_xy_fwd_gen<T, SRC_U9>, dim3(1, 9, 1), dim3((unsigned)h.nt), room, (const T*)f.data(), spec.data(), g, h,
              (const cplx<T>*)tw.data(), (const cplx<T>*)tw.data(), (const int*)posm.data(), (const T*)nullptr, 9,
              (const RepArgs*)nullptr);
  report(what, "fwd", W, Lx, Ly, 1, want);
  emu::launch(k_xy_inv_gen<T>, dim3(1, 9, 1), dim3((unsigned)h.nt), room, (const cplx<T>*)spec.data(), f.data(), g, h,
              (const cplx<T>*)tw.data(), (const cplx<T>*)tw.data(), (const int*)posm.data(), (const Phys*)nullptr,
              (DevScalars*)nullptr, (const double*)nullptr, 0, (const RepArgs*)nullptr);
  report(what, "inv", W, Lx, Ly, 1, want);
}

template <typename T>
void z(int Lx, int Ly, int Lz, int lpw, const char* what, const std::function<void(Geom&, ZGeo&, ZTiles&)>& plant) {
  constexpr int W = kLanes<T>;
  Geom g = geom(Lx, Ly, Lz);
  ZGeo h{};
  lane_split(Lz, false, &h.R1, &h.R2);
  h.lpw = lpw;
  h.d1 = fast_div(h.R1);
  h.d2 = fast_div(h.R2);
  const bool wn = W == 2 && g.m % 2 != 0;
  h.ncol = g.m + (wn ? 1 : 0);
  ZTiles zt{};
  zt.CW = W << lpw;
  zt.ntx = (h.ncol + zt.CW - 1) / zt.CW;
  zt.nreg = zt.ntx * Ly;
  zt.nnyq = wn ? 0 : (Ly + zt.CW - 1) / zt.CW;
  const size_t room = (size_t)9 * 4 * Lz * 16 << lpw;
  const int big = 4 * (Lx + Ly + Lz);
  std::vector<double> k((size_t)big, 0.3);
  std::vector<double2> t((size_t)big, make_double2(1, 0));
  KMaps km{};
  km.kvz_s = km.kvx_s = km.kvy_s = k.data();
  km.trz_s = km.trx_s = km.try_s = t.data();
  Phys ph{};
  ph.Ninv = ph.kap2x2 = ph.B11 = ph.B44 = 1;
  std::vector<cplx<T>> tw((size_t)big, mk<cplx<T>>((T)1, (T)0)), spec((size_t)(40 * g.ncplx + 4096));
  std::vector<T> dtab((size_t)(24 * g.nkpos), (T)1);
  plant(g, h, zt);
  std::vector<double> part((size_t)(NQ_K * (zt.nreg + zt.nnyq)));
  DevScalars sc{};
  emu::launch(k_z_lane<T, 0, 0, false>, dim3((unsigned)(zt.nreg + zt.nnyq), 1), dim3(256), room, spec.data(),
              (const T*)dtab.data(), (const cplx<T>*)nullptr, (cplx<T>*)nullptr, g, h, (const cplx<T>*)tw.data(), km,
              (const Phys*)&ph, part.data(), &sc, zt, (const RepArgs*)nullptr);
  report(what, "z", W, Lx, Ly, Lz, *what == '-' ? 0 : 1);
}
// a compile-time length, as launched and with spectrum rows cut short
template <typename T>
void zct(int Lx, int Ly, const char* what, const std::function<void(Geom&, ZTiles&)>& plant) {
  constexpr int W = kLanes<T>;
  using Z = ZCT<T, 16, 2, false>;
  Geom g = geom(Lx, Ly, 16);
  ZTiles zt{};
  zt.CW = 2 * W;
  zt.ntx = g.m / zt.CW;
  zt.nreg = zt.ntx * Ly;
  zt.nnyq = (Ly + zt.CW - 1) / zt.CW;
  const int big = 4 * (Lx + Ly + 16);
  std::vector<double> k((size_t)big, 0.3);
  std::vector<double2> t((size_t)big, make_double2(1, 0));
  KMaps km{};
  km.kvz_s = km.kvx_s = km.kvy_s = k.data();
  km.trz_s = km.trx_s = km.try_s = t.data();
  Phys ph{};
  ph.Ninv = ph.kap2x2 = ph.B11 = ph.B44 = 1;
  std::vector<cplx<T>> tw((size_t)big, mk<cplx<T>>((T)1, (T)0)), spec((size_t)(40 * g.ncplx + 4096));
  std::vector<T> dtab((size_t)(24 * g.nkpos), (T)1);
  plant(g, zt);
  std::vector<double> part((size_t)(NQ_K * (zt.nreg + zt.nnyq)));
  DevScalars sc{};
  emu::launch(k_z_lane<T, 16, 2, false>, dim3((unsigned)(zt.nreg + zt.nnyq), 1), dim3(Z::NT), (size_t)Z::SMEM, spec.data(),
              (const T*)dtab.data(), (const cplx<T>*)nullptr, (cplx<T>*)nullptr, g, ZGeo{}, (const cplx<T>*)tw.data(), km,
              (const Phys*)&ph, part.data(), &sc, zt, (const RepArgs*)nullptr);
  report(what, "zct", W, Lx, Ly, 16, *what == '-' ? 0 : 1);
}

template <typename T>
void all() {
  const int s[][2] = {{4, 3}, {10, 6}, {18, 10}, {30, 18}, {50, 36}, {96, 54}, {8, 135}};
  for (auto& a : s) {
    xy<T>(a[0], a[1], "-", [](Geom&, XyGeo&) {});
    xy<T>(a[0], a[1], "smem", [](Geom&, XyGeo& h) { h.smem -= 32 * std::max(h.QS, h.JS); });
    xy<T>(a[0], a[1], "qs", [](Geom&, XyGeo& h) { h.QS = h.smem / 16; });
    xy<T>(a[0], a[1], "js", [](Geom&, XyGeo& h) { h.JS = h.smem / 16; });
    xy<T>(a[0], a[1], "ly", [](Geom& g, XyGeo&) { g.Ly -= 1; });
    xy<T>(a[0], a[1], "lx", [](Geom& g, XyGeo&) { g.m -= 1; g.Lx -= 2; });
  }
  const int q[][4] = {{4, 3, 3, 0}, {10, 6, 5, 2}, {18, 4, 9, 1}, {16, 3, 10, 2}, {12, 4, 90, 1}, {8, 3, 64, 0}};
  for (auto& a : q) {
    z<T>(a[0], a[1], a[2], a[3], "-", [](Geom&, ZGeo&, ZTiles&) {});
    z<T>(a[0], a[1], a[2], a[3], "tile", [](Geom&, ZGeo& h, ZTiles&) { h.lpw += 1; });
    z<T>(a[0], a[1], a[2], a[3], "lz", [](Geom& g, ZGeo&, ZTiles&) { g.Lz -= 1; });
  }
  zct<T>(16, 5, "-", [](Geom&, ZTiles&) {});
  zct<T>(16, 5, "kxp", [](Geom& g, ZTiles&) { g.KXP = 4; });
}

int main() {
  all<double>();
  all<float>();
  return 0;
}
