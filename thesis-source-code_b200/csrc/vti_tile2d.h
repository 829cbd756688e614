// 2D propagation several levels per launch (vti_tile2d.cu): the interface
// used by the 2D forward, gradient and migration drivers.
#pragma once

#include <vector>

#include "vti_internal.h"

namespace vti {
namespace tile2d {

constexpr int kExt = 64;           // cells per side that a CTA holds
constexpr int kMinT = 2, kMinBackT = 3, kMaxT = 5;  // levels per launch

// How a grid is cut: T levels per launch, so a CTA owns the inner tile = 64 - 8 T
// cells per side of the 64 it holds. Every array is padded: grid cell (x, z) at
// (x + off) + (z + off) * W, so that the update region [4, n-4) starts at the
// first owned cell of tile 0; the margins hold zeros.
struct Layout {
  int nnx = 0, nnz = 0, T = 0, tile = 0, off = 0, ntx = 0, ntz = 0, W = 0;
  size_t n = 0;  // floats per array
  __host__ __device__ int at(int x, int z) const { return x + off + (z + off) * W; }
};
// The layout for `shots` grids advanced side by side (backward: by the backward
// kernel too) on sm_count SMs; *us_per_level: what a forward level of all of them
// takes. T = 0: a grid so thin and long that its padded arrays pass the 2^31 cells
// that an index counts, or that a launch's second dimension passes 65535 tiles.
//
// A launch takes about 0.5 us and 3.4 + 0.85 T us per wave of one CTA per SM: the
// first part of a wave is loading the square, so more levels per launch pay while
// the smaller tiles still fit the waves. Forward, us per launch for T = 2 / 3 / 4 / 5:
// one wave (28 to 77 CTAs, 261 x 161) 5.3 / 6.5 / 7.1 / 8.2, two waves (112 to 209 CTAs, 461 x
// 261) 5.5 / 6.8 / 7.4 / 15.4, 4 to 14 waves (three shots of 861 x 461) 19.4 / 34.9 / 55 / 101.
// A gradient's two launches together take about 1 us and 12.6 + 0.85 T us per wave
// (T = 3 / 4 / 5: 461 x 261 16.3 / 17.2 / 34.7 us, 1061 x 561 46 / 71 / 133), a migration's 1.5
// us and 8.6 + 1.45 T (15.1 / 16.1 / 31.9, 39.5 / 68 / 125). Choosing their depth by those
// gives the same one as the forward cost for every grid of 190..861 x 130..461, so one
// rule serves all.
inline Layout make_layout(int sm_count, int nnx, int nnz, int shots, bool backward,
                          double* us_per_level = nullptr) {
  Layout best;
  double cost = 0;
  // backward from 3: the D pairs of two levels and their images and the gradient's
  // images of 48 x 48 cells do not fit shared memory (a migration's one image and two
  // slices would; its kernels are built for the same depths)
  for (int T = backward ? kMinBackT : kMinT; T <= kMaxT; ++T) {
    Layout L;
    L.nnx = nnx;
    L.nnz = nnz;
    L.T = T;
    L.tile = kExt - 2 * kHalo * T;
    L.off = kHalo * T - kHalo;
    L.ntx = (nnx - 2 * kHalo + L.tile - 1) / L.tile;
    L.ntz = (nnz - 2 * kHalo + L.tile - 1) / L.tile;
    L.W = ((L.ntx - 1) * L.tile + kExt + 31) & ~31;
    L.n = (size_t)L.W * ((L.ntz - 1) * L.tile + kExt);
    if (L.n > 0x7fffffff || L.ntz > 65535) continue;
    const long long ctas = (long long)L.ntx * L.ntz * shots;
    const double c = (0.5 + (double)((ctas + sm_count - 1) / sm_count) * (3.4 + 0.85 * T)) / T;
    if (!best.T || c < cost) {
      best = L;
      cost = c;
    }
  }
  if (us_per_level) *us_per_level = cost;
  return best;
}

// Model arrays in the padded layout, zero outside the update region (so a level
// needs no bounds tests: next = taper * (...) is 0 there, as in the frame).
struct Model {
  const float *c11, *c13, *c33, *taper;
  float idx2, idz2, dt2;
};

// Wavefields of one shot: two sets of four arrays (current p, q, previous p, q);
// a launch reads one set and writes the other.
constexpr int kWaveArrays = 8;

enum Keep { kKeepNone = 0, kKeepD = 1, kKeepSlice = 2 };

// Forward levels lev0 .. lev0 + nlev - 1 of `shots` shots (forwardCD,
// lib/vti-fwi-2d/kernels.cu:452-498, taper :304-315).
struct Forward {
  Layout L;
  Model m;
  int lev0, nlev, shots;
  const float* in;   // set read, shot 0; shots are wave_stride floats apart
  float* out;
  size_t wave_stride;
  const int* src;    // per shot: padded index of the source
  const float* amp;  // per level
  int dipole;        // -amp one row below the source
  // traces: receiver of each cell (-1 none, n per shot), row of each level (-1
  // none), per shot offset into rec and receivers per row; null: none
  const int* rmap;
  const int* rec_row;
  float* rec;
  const long long* rec_off;
  const int* nri;
  // kept arrays: kKeepD stores (Dxx p, Dzz q) of the level before `it` where
  // keep[it - 1] >= 0, kKeepSlice 0.5 (p + q) of level `it` where keep[it] >= 0
  int keep_mode;
  const int* keep;
  float* kept;  // slot k at kept + k * (1 or 2) * n
};
int launch_forward(vti_ctx* ctx, const Forward& a);

// One backward level: the current adjoint is imaged against
// (1 - f) kept[a] + f kept[b], stepped, and with inject != 0 the rows r0, r1 of
// the traces (-1: zeros) interpolated with fi enter the new level.
struct BackLevel {
  int a, b;
  float f;
  int r0, r1;
  float fi;
  int inject;
};
// Backward levels: exact: the adjoint of forwardCD (backwardDC) imaged against D
// pairs into g11 | g13 | g33; otherwise forwardCD imaged against slices into g,
// the traces entering as dipoles.
struct Backward {
  Layout L;
  Model m;
  int exact, nlev, image_last;  // image_last: the last level is imaged as well
  const float* in;
  float* out;
  const BackLevel* lv;  // of the first level
  const float* kept;
  float* g;
  const int* rmap;
  const float* rows;  // row r at rows + r * row_stride
  long long row_stride;
};
int launch_backward(vti_ctx* ctx, const Backward& a);

// Contiguous nnx x nnz array into the padded layout and back: the update region,
// zeros in the frame around it.
int launch_pad(vti_ctx* ctx, const Layout& L, const float* src, float* dst);
int launch_unpad(vti_ctx* ctx, const Layout& L, const float* src, float* dst);
// map[cell] = receiver for the given padded cells, -1 elsewhere.
int launch_map(vti_ctx* ctx, const Layout& L, const int* cells, int n, int* map);
// a[i] = b[i] = v at one padded cell.
int launch_point(vti_ctx* ctx, float* a, float* b, int cell, float v);
// Point (dipole: also one row below, negative) injection of dt2 * 0.5 * row into a
// level, times the taper when scale is set.
int launch_inject(vti_ctx* ctx, const Layout& L, float* p, float* q, const float* row,
                  const int* cells, int n, const float* taper, float dt2, int scale, int dipole);

// Carves 256-byte aligned pieces out of one block; with base null it only
// counts the bytes.
struct Carve {
  char* base;
  size_t used = 0;
  template <typename T>
  T* take(size_t count) {
    T* r = base ? reinterpret_cast<T*>(base + used) : nullptr;
    used += (count * sizeof(T) + 255) & ~(size_t)255;
    return r;
  }
};

// Whether the receivers (x, z pairs) lie in the update region, one per cell
// (dipole: with the row below them in it as well).
bool receivers_fit(int nnx, int nnz, const int* rloc, int n, bool dipole);

}  // namespace tile2d
}  // namespace vti
