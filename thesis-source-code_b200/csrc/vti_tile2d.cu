// 2D propagation, several time levels per launch.
//
// A 2D shot is small (0.5 MB per array at 461 x 261), so one launch per level is
// bound by launches: 5.4 us per forward level and 6 per gradient level, whatever
// the work. Here a CTA holds 64 x 64 cells and owns the inner 64 - 8 T: the 4 T-cell
// halo is what T levels of the 8th-order cross stencil reach. It advances T levels
// in shared memory, each on a region 4 cells smaller per side (with T = 4 twice
// the owned cells' work, on SMs that would otherwise wait), and writes its own
// cells of the last two levels into the other of two wavefield sets. Launches
// follow one another as programmatic dependents; every cell is computed by the
// operations of the per-level kernels, so results do not depend on the split (the
// per-level migration injects with global float atomics, which flush subnormal
// contributions; here they are added).
//
// Whole calls, B200, one launch per level -> now: traces 801x401 + 30 cells, 1000
// levels, three shots 24.0 -> 10.3 ms; traces 201x101 + 30 (one cluster before) 2.30
// -> 1.85 ms; gradient 401x201 + 30, 1000 levels 12.3 -> 5.1 ms; RTM 377x183 + 30, 900
// levels, two shots 26.0 -> 7.7 ms. What bounds it now: the launch and the load of the
// square (3.4 us per launch), then instruction issue at one CTA of 16 warps per SM
// (0.85 us per level).
#include <algorithm>
#include <atomic>

#include "vti_pair.cuh"
#include "vti_tile2d.h"

namespace vti {
namespace tile2d {
namespace {

// lib/vti-fwi-2d/kernels.h:4-8 (float literals)
constexpr float kC0 = -2.84722222222f, kC1 = 1.6f, kC2 = -0.2f, kC3 = 0.02539682539f,
                kC4 = -0.00178571428f;
constexpr int kThreads = 512, kRows = 4, kWarps = kThreads / 32;
static_assert(kWarps * kRows == kExt && kExt == 64, "one warp per four rows");
static_assert(kHalo == kRows, "a level drops one warp (and two lanes) at each end");

constexpr int kField = kExt * kExt;             // floats
constexpr int kGuard = 8;                       // reads of x - 4 in row 0, x + 5 in the last
constexpr int kFieldsSmem = 4 * kField + 2 * kGuard;

__device__ __forceinline__ float2 ld2(const float* p) {
  return *reinterpret_cast<const float2*>(p);
}
__device__ __forceinline__ void st2(float* p, float2 v) { *reinterpret_cast<float2*>(p) = v; }

__device__ __forceinline__ float lap1(const float* v) {
  float s = __fmul_rn(kC0, v[4]);
  s = __fmaf_rn(kC1, __fadd_rn(v[3], v[5]), s);
  s = __fmaf_rn(kC2, __fadd_rn(v[2], v[6]), s);
  s = __fmaf_rn(kC3, __fadd_rn(v[1], v[7]), s);
  return __fmaf_rn(kC4, __fadd_rn(v[0], v[8]), s);
}
// x stencil of the pair at `row` (pointer to its first cell)
__device__ __forceinline__ float2 lap_x(const float* row, float2* centre) {
  float v[10];
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const float2 u = ld2(row - 4 + 2 * k);
    v[2 * k] = u.x;
    v[2 * k + 1] = u.y;
  }
  *centre = make_float2(v[4], v[5]);
  return make_float2(lap1(v), lap1(v + 1));
}
__device__ __forceinline__ float2 lap_z(const float2* q) {
  float2 s = mul2(splat(kC0), q[4]);
  s = fma2(splat(kC1), add2(q[3], q[5]), s);
  s = fma2(splat(kC2), add2(q[2], q[6]), s);
  s = fma2(splat(kC3), add2(q[1], q[7]), s);
  return fma2(splat(kC4), add2(q[0], q[8]), s);
}

// 2 cur - taper prev, rounded once: what the compiler makes of the per-level
// gradient and migration kernels' expression; two roundings in the forward
// modeling kernel, which spells it out.
template <bool kFused>
__device__ __forceinline__ float2 carry(float2 cur, float2 t, float2 prev) {
  const float2 two = mul2(splat(2.f), cur);
  return kFused ? fma2(mul2(splat(-1.f), t), prev, two) : sub2(two, mul2(t, prev));
}

template <bool kFused, int T>
__global__ void __launch_bounds__(kThreads, 1) k_tile_forward(const __grid_constant__ Forward a) {
  pdl_launch_next();
  extern __shared__ __align__(16) float sm_raw[];
  float* sm = sm_raw + kGuard;  // [x field 0][z field 0][x field 1][z field 1]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int W = a.L.W, r0 = warp * kRows, c0 = 2 * lane;
  const int shot = blockIdx.z;
  constexpr int tile = kExt - 2 * kHalo * T;
  const int base = blockIdx.x * tile + c0 + (blockIdx.y * tile + r0) * W;  // padded, row r0
  float2 m11[kRows], m13[kRows], m33[kRows], tp[kRows], pp[kRows], qp[kRows];
#pragma unroll
  for (int j = 0; j < kRows; ++j) {
    const int i = base + j * W;
    m11[j] = __ldg(reinterpret_cast<const float2*>(a.m.c11 + i));
    m13[j] = __ldg(reinterpret_cast<const float2*>(a.m.c13 + i));
    m33[j] = __ldg(reinterpret_cast<const float2*>(a.m.c33 + i));
    tp[j] = __ldg(reinterpret_cast<const float2*>(a.m.taper + i));
  }
  const int src = __ldg(a.src + shot) - base;  // 0, 1 in row 0; + j W in row j
  const bool own = warp >= T && warp < kWarps - T && lane >= 2 * T && lane < 32 - 2 * T;
  unsigned rmask = 0;  // cells of this thread that hold a receiver
  const int* rmap = a.rmap ? a.rmap + shot * a.L.n : nullptr;
  const float* in = a.in + shot * a.wave_stride;
  pdl_wait();
#pragma unroll
  for (int j = 0; j < kRows; ++j) {
    const int i = base + j * W, o = (r0 + j) * kExt + c0;
    st2(sm + o, ld2(in + i));
    st2(sm + kField + o, ld2(in + a.L.n + i));
    pp[j] = ld2(in + 2 * a.L.n + i);
    qp[j] = ld2(in + 3 * a.L.n + i);
    if (rmap && own) {
      const int2 m = __ldg(reinterpret_cast<const int2*>(rmap + i));
      rmask |= (m.x >= 0 ? 1u : 0u) << (2 * j) | (m.y >= 0 ? 2u : 0u) << (2 * j);
    }
  }
  __syncthreads();
  for (int k = 1; k <= a.nlev; ++k) {
    const int it = a.lev0 + k - 1;
    const float* P = sm + ((k - 1) & 1) * 2 * kField;
    const float* Q = P + kField;
    float* Pn = sm + (k & 1) * 2 * kField;
    float* Qn = Pn + kField;
    if (warp >= k && warp < kWarps - k) {
      const float amp = __ldg(a.amp + it);
      const int row = a.rec_row ? __ldg(a.rec_row + it) : -1;
      const int slot = a.keep_mode == kKeepD       ? __ldg(a.keep + it - 1)
                       : a.keep_mode == kKeepSlice ? __ldg(a.keep + it)
                                                   : -1;
      float2 q[kRows + 8];
#pragma unroll
      for (int j = 0; j < kRows + 8; ++j) q[j] = ld2(Q + (r0 - 4 + j) * kExt + c0);
#pragma unroll
      for (int j = 0; j < kRows; ++j) {
        const int o = (r0 + j) * kExt + c0, i = base + j * W;
        float2 pc;
        const float2 lx = mul2(lap_x(P + o, &pc), splat(a.m.idx2));
        const float2 lz = mul2(lap_z(q + j), splat(a.m.idz2));
        const float2 qc = q[j + 4], dt2 = splat(a.m.dt2);
        float2 pn = fma2(dt2, fma2(m11[j], lx, mul2(m13[j], lz)), carry<kFused>(pc, tp[j], pp[j]));
        float2 qn = fma2(dt2, fma2(m13[j], lx, mul2(m33[j], lz)), carry<kFused>(qc, tp[j], qp[j]));
        const int e = src - j * W;
        if (e == 0) {
          pn.x = __fadd_rn(pn.x, amp);
          qn.x = __fadd_rn(qn.x, amp);
        } else if (e == 1) {
          pn.y = __fadd_rn(pn.y, amp);
          qn.y = __fadd_rn(qn.y, amp);
        } else if (a.dipole && e == -W) {
          pn.x = __fsub_rn(pn.x, amp);
          qn.x = __fsub_rn(qn.x, amp);
        } else if (a.dipole && e == 1 - W) {
          pn.y = __fsub_rn(pn.y, amp);
          qn.y = __fsub_rn(qn.y, amp);
        }
        pn = mul2(tp[j], pn);
        qn = mul2(tp[j], qn);
        st2(Pn + o, pn);
        st2(Qn + o, qn);
        pp[j] = pc;
        qp[j] = qc;
        if (row >= 0 && (rmask >> (2 * j) & 3u)) {
          float* rec = a.rec + __ldg(a.rec_off + shot) + (long long)row * __ldg(a.nri + shot);
          if (rmask >> (2 * j) & 1u) rec[__ldg(rmap + i)] = 0.5f * (pn.x + qn.x);
          if (rmask >> (2 * j) & 2u) rec[__ldg(rmap + i + 1)] = 0.5f * (pn.y + qn.y);
        }
        if (slot >= 0 && own) {
          if (a.keep_mode == kKeepD) {
            float* d = a.kept + (size_t)slot * 2 * a.L.n + i;
            st2(d, lx);
            st2(d + a.L.n, lz);
          } else {
            st2(a.kept + (size_t)slot * a.L.n + i,
                make_float2(0.5f * (pn.x + qn.x), 0.5f * (pn.y + qn.y)));
          }
        }
      }
    }
    __syncthreads();
  }
  if (own) {
    const float* P = sm + (a.nlev & 1) * 2 * kField;
    float* out = a.out + shot * a.wave_stride;
#pragma unroll
    for (int j = 0; j < kRows; ++j) {
      const int i = base + j * W, o = (r0 + j) * kExt + c0;
      st2(out + i, ld2(P + o));
      st2(out + a.L.n + i, ld2(P + kField + o));
      st2(out + 2 * a.L.n + i, pp[j]);
      st2(out + 3 * a.L.n + i, qp[j]);
    }
  }
}

// ---------------------------------------------------------------- backward
// Waits until at most n of this thread's groups of copies are in flight.
__device__ __forceinline__ void cp_wait(int n) {
  switch (n) {
    case 0: asm volatile("cp.async.wait_group 0;" ::: "memory"); break;
    case 1: asm volatile("cp.async.wait_group 1;" ::: "memory"); break;
    case 2: asm volatile("cp.async.wait_group 2;" ::: "memory"); break;
    case 3: asm volatile("cp.async.wait_group 3;" ::: "memory"); break;
    case 4: asm volatile("cp.async.wait_group 4;" ::: "memory"); break;
    default: asm volatile("cp.async.wait_group 5;" ::: "memory"); break;
  }
}
// 16 bytes of global memory into shared memory, asynchronously.
__device__ __forceinline__ void cp16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}

// Shared memory of a backward CTA: the two fields on two levels, taper and c13
// of the held cells, the image sums of the owned ones and the kept arrays the
// owned cells are imaged against, for every level of the launch: they come from
// HBM, so all are on their way before the levels start (one level ahead made
// every level wait for them).
template <bool kExact>
struct BackSmem {
  static constexpr int kImages = kExact ? 3 : 1;
  static constexpr int kKept = kExact ? 4 : 2;  // (a, b) x (D pair or slice)
  static constexpr int kTaper = kFieldsSmem;
  static constexpr int kC13 = kTaper + kField;
  static constexpr int kImage = kC13 + kField;
  // T levels and the image of the last one
  __host__ __device__ static constexpr int floats(int T) {
    return kImage + (kImages + (T + 1) * kKept) * (kExt - 2 * kHalo * T) * (kExt - 2 * kHalo * T);
  }
  // 16-byte copies into the kept arrays: every piece before them and every row of a
  // tile (8 (8 - T) floats) is a multiple of four floats
  static_assert(kTaper % 4 == 0 && kC13 % 4 == 0 && kImage % 4 == 0 && (2 * kHalo) % 4 == 0 &&
                    kExt % 4 == 0,
                "16-byte pieces");
};

// The kept arrays of level `lv` over the owned cells into buf: [a][b] (exact:
// [a x][a z][b x][b z]).
template <bool kExact, int T>
__device__ __forceinline__ void fetch_kept(const Backward& a, const BackLevel* lv, float* buf) {
  constexpr int kPer = kExact ? 2 : 1;
  constexpr int tile = kExt - 2 * kHalo * T, own = kHalo * T, row4 = tile / 4;
  constexpr int chunks = row4 * tile;
  const int sa = lv->a, sb = lv->b;
#pragma unroll
  for (int t = threadIdx.x; t < BackSmem<kExact>::kKept * chunks; t += kThreads) {
    const int arr = t / chunks, c = t - arr * chunks, z = c / row4, x = 4 * (c - z * row4);
    const int slot = arr < kPer ? sa : sb;
    const float* s = a.kept + ((size_t)slot * kPer + arr % kPer) * a.L.n +
                     (blockIdx.x * tile + own + x) +
                     (size_t)(blockIdx.y * tile + own + z) * a.L.W;
    cp16(buf + arr * tile * tile + z * tile + x, s);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

template <bool kExact, int T>
__global__ void __launch_bounds__(kThreads, 1)
    k_tile_backward(const __grid_constant__ Backward a) {
  using S = BackSmem<kExact>;
  pdl_launch_next();
  extern __shared__ __align__(16) float sm_raw[];
  float* sm = sm_raw + kGuard;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int W = a.L.W, r0 = warp * kRows, c0 = 2 * lane;
  constexpr int tile = kExt - 2 * kHalo * T, kOwned = tile * tile;
  const int base = blockIdx.x * tile + c0 + (blockIdx.y * tile + r0) * W;
  float2 m11[kRows], m33[kRows], pc[kRows], qc[kRows], pp[kRows], qp[kRows];
  float* smT = sm_raw + S::kTaper;
  float* smC = sm_raw + S::kC13;
#pragma unroll
  for (int j = 0; j < kRows; ++j) {
    const int i = base + j * W, o = (r0 + j) * kExt + c0;
    m11[j] = __ldg(reinterpret_cast<const float2*>(a.m.c11 + i));
    m33[j] = __ldg(reinterpret_cast<const float2*>(a.m.c33 + i));
    st2(smC + o, __ldg(reinterpret_cast<const float2*>(a.m.c13 + i)));
    st2(smT + o, __ldg(reinterpret_cast<const float2*>(a.m.taper + i)));
  }
  const bool own = warp >= T && warp < kWarps - T && lane >= 2 * T && lane < 32 - 2 * T;
  // cells of this thread that a receiver injects into (bit e), and for dipoles
  // (bit 8 + e) those one row below a receiver
  unsigned rmask = 0;
  // the levels of this launch
  __shared__ BackLevel lvs[T + 1];
  if (threadIdx.x < (a.nlev + a.image_last) * (sizeof(BackLevel) / 4))
    reinterpret_cast<int*>(lvs)[threadIdx.x] =
        __ldg(reinterpret_cast<const int*>(a.lv) + threadIdx.x);
  __syncthreads();
  // kept arrays are written by the forward pass and read-only here: the first two
  // levels' copies start at once, the others behind the wavefields
  float* kept = sm_raw + S::kImage + S::kImages * kOwned;
  constexpr int kKeptLevel = S::kKept * kOwned;
  const int images = a.nlev + a.image_last;
  const int ahead = images < 2 ? images : 2;
  for (int k = 0; k < ahead; ++k) fetch_kept<kExact, T>(a, lvs + k, kept + k * kKeptLevel);
  pdl_wait();
  if (a.rmap)
#pragma unroll
    for (int e = 0; e < 2 * kRows; ++e) {
      const int i = base + (e >> 1) * W + (e & 1);
      if (__ldg(a.rmap + i) >= 0) rmask |= 1u << e;
      if (!kExact && i >= W && __ldg(a.rmap + i - W) >= 0) rmask |= 256u << e;
    }
#pragma unroll
  for (int j = 0; j < kRows; ++j) {
    const int i = base + j * W, o = (r0 + j) * kExt + c0;
    pc[j] = ld2(a.in + i);
    qc[j] = ld2(a.in + a.L.n + i);
    pp[j] = ld2(a.in + 2 * a.L.n + i);
    qp[j] = ld2(a.in + 3 * a.L.n + i);
    if (kExact) {  // u = c11 p + c13 q along x, w = c13 p + c33 q along z
      const float2 m13 = ld2(smC + o);
      st2(sm + o, fma2(m11[j], pc[j], mul2(m13, qc[j])));
      st2(sm + kField + o, fma2(m13, pc[j], mul2(m33[j], qc[j])));
    } else {
      st2(sm + o, pc[j]);
      st2(sm + kField + o, qc[j]);
    }
  }
  // image sums of the owned cells: a thread's own cells, so no barrier
  const int own0 = (r0 - kHalo * T) * tile + (c0 - kHalo * T);
  float* img = sm_raw + S::kImage + own0;
  if (own)
#pragma unroll
    for (int j = 0; j < kRows; ++j)
#pragma unroll
      for (int c = 0; c < S::kImages; ++c)
        st2(img + c * kOwned + j * tile, ld2(a.g + c * a.L.n + base + j * W));
  for (int k = ahead; k < images; ++k) fetch_kept<kExact, T>(a, lvs + k, kept + k * kKeptLevel);
  for (int k = 1; k <= images; ++k) {
    const BackLevel* lv = lvs + k - 1;
    // this level's kept arrays have arrived; the fields of the level before it
    // are written
    cp_wait(images - k);
    __syncthreads();
    const float* D = kept + (k - 1) * kKeptLevel;
    if (own) {
      const float f = lv->f;
      const float2 g = splat(1.f - f), f2 = splat(f);
      const float* d = D + own0;
#pragma unroll
      for (int j = 0; j < kRows; ++j) {
        const int o = j * tile;
        if (kExact) {  // gradientCrossCor (kernels.cu:438-450), rounded as in the per-level kernel:
          // the product that is rounded by itself is f D_b of Dp and (1 - f) D_a of Dq
          const float2 Dp = fma2(g, ld2(d + o), mul2(f2, ld2(d + 2 * kOwned + o)));
          const float2 Dq = fma2(f2, ld2(d + 3 * kOwned + o), mul2(g, ld2(d + kOwned + o)));
          st2(img + o, fma2(pc[j], Dp, ld2(img + o)));
          st2(img + kOwned + o, add2(ld2(img + kOwned + o), fma2(qc[j], Dp, mul2(pc[j], Dq))));
          st2(img + 2 * kOwned + o, fma2(qc[j], Dq, ld2(img + 2 * kOwned + o)));
        } else {  // imagingCrossCor (kernels.cu:414-423)
          const float2 s = fma2(g, ld2(d + o), mul2(f2, ld2(d + kOwned + o)));
          st2(img + o, fma2(mul2(splat(0.5f), add2(pc[j], qc[j])), s, ld2(img + o)));
        }
      }
    }
    if (k > a.nlev) break;
    const float* P = sm + ((k - 1) & 1) * 2 * kField;
    const float* Q = P + kField;
    float* Pn = sm + (k & 1) * 2 * kField;
    float* Qn = Pn + kField;
    if (warp >= k && warp < kWarps - k) {
      // what the receivers add to this thread's cells: dt2 times half the traces
      // interpolated between the two rows, times the taper; loaded ahead of the
      // stencils, one round trip per level
      const bool inject = rmask && lv->inject;
      float add[2 * kRows], sub[2 * kRows];
      if (inject) {
        const float fi = lv->fi;
        const float* b0 = lv->r0 >= 0 ? a.rows + lv->r0 * a.row_stride : nullptr;
        const float* b1 = lv->r1 >= 0 ? a.rows + lv->r1 * a.row_stride : nullptr;
        auto value = [&](int cell, float t) {
          const int ir = __ldg(a.rmap + cell);
          const float v0 = b0 ? __ldg(b0 + ir) : 0.f, v1 = b1 ? __ldg(b1 + ir) : 0.f;
          const float s = kExact ? __fadd_rn(__fmul_rn(1.f - fi, v0), __fmul_rn(fi, v1))
                                 : __fmaf_rn(1.f - fi, v0, __fmul_rn(fi, v1));
          return __fmul_rn(__fmul_rn(a.m.dt2, __fmul_rn(0.5f, s)), t);
        };
#pragma unroll
        for (int e = 0; e < 2 * kRows; ++e) {
          const int cell = base + (e >> 1) * W + (e & 1);
          const float t = smT[(r0 + (e >> 1)) * kExt + c0 + (e & 1)];
          add[e] = rmask >> e & 1u ? value(cell, t) : 0.f;
          if (!kExact) sub[e] = rmask >> (8 + e) & 1u ? value(cell - W, t) : 0.f;
        }
      }
      float2 q[kRows + 8];
#pragma unroll
      for (int j = 0; j < kRows + 8; ++j) q[j] = ld2(Q + (r0 - 4 + j) * kExt + c0);
#pragma unroll
      for (int j = 0; j < kRows; ++j) {
        const int o = (r0 + j) * kExt + c0;
        float2 unused;
        const float2 lx = mul2(lap_x(P + o, &unused), splat(a.m.idx2));
        const float2 lz = mul2(lap_z(q + j), splat(a.m.idz2));
        const float2 t = ld2(smT + o), m13 = ld2(smC + o), dt2 = splat(a.m.dt2);
        const float2 px = kExact ? lx : fma2(m11[j], lx, mul2(m13, lz));
        const float2 qx = kExact ? lz : fma2(m13, lx, mul2(m33[j], lz));
        float2 pn = mul2(t, fma2(dt2, px, carry<true>(pc[j], t, pp[j])));
        float2 qn = mul2(t, fma2(dt2, qx, carry<true>(qc[j], t, qp[j])));
        if (inject) {
          const float2 v = make_float2(add[2 * j], add[2 * j + 1]);
          pn = add2(pn, v);
          qn = add2(qn, v);
          if (!kExact) {
            const float2 w = make_float2(sub[2 * j], sub[2 * j + 1]);
            pn = sub2(pn, w);
            qn = sub2(qn, w);
          }
        }
        pp[j] = pc[j];
        qp[j] = qc[j];
        pc[j] = pn;
        qc[j] = qn;
        if (kExact) {
          st2(Pn + o, fma2(m11[j], pn, mul2(m13, qn)));
          st2(Qn + o, fma2(m13, pn, mul2(m33[j], qn)));
        } else {
          st2(Pn + o, pn);
          st2(Qn + o, qn);
        }
      }
    }
  }
  if (own) {
#pragma unroll
    for (int j = 0; j < kRows; ++j) {
      const int i = base + j * W;
      st2(a.out + i, pc[j]);
      st2(a.out + a.L.n + i, qc[j]);
      st2(a.out + 2 * a.L.n + i, pp[j]);
      st2(a.out + 3 * a.L.n + i, qp[j]);
#pragma unroll
      for (int c = 0; c < S::kImages; ++c)
        st2(a.g + c * a.L.n + i, ld2(img + c * kOwned + j * tile));
    }
  }
}

// ------------------------------------------------------------ small kernels
// kPad: into the padded layout, otherwise out of it; zero in the outer lo cells of
// the grid (the padded frame at the far sides is owned by tiles and, though its
// fields are zero times whatever its neighbours hold, NaN beside a NaN).
template <bool kPad>
__global__ void k_pad(Layout L, const float* src, float* dst, int lo) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= L.nnx * L.nnz) return;
  const int x = i % L.nnx, z = i / L.nnx, j = L.at(x, z);
  const bool in = x >= lo && x < L.nnx - lo && z >= lo && z < L.nnz - lo;
  const float v = in ? src[kPad ? i : j] : 0.f;
  dst[kPad ? j : i] = v;
}

__global__ void k_map(const int* cells, int n, int* map) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) map[cells[i]] = i;
}

__global__ void k_point(float* a, float* b, int cell, float v) {
  a[cell] = v;
  b[cell] = v;
}

__global__ void k_inject_row(Layout L, float* p, float* q, const float* row, const int* cells, int n,
                             const float* taper, float dt2, int scale, int dipole) {
  const int ir = blockIdx.x * blockDim.x + threadIdx.x;
  if (ir >= n) return;
  const float v = __fmul_rn(dt2, __fmul_rn(0.5f, row[ir]));
  auto add = [&](int i, float w) {
    const float s = scale ? __fmul_rn(taper[i], w) : w;
    atomicAdd(p + i, s);
    atomicAdd(q + i, s);
  };
  add(cells[ir], v);
  if (dipole) add(cells[ir] + L.W, -v);
}

// Once per device and kernel (setting the attribute twice is harmless).
template <typename K>
int smem_attr(vti_ctx* ctx, K kern, int bytes, std::atomic<bool>* done) {
  if (ctx->device < 64 && done[ctx->device].load(std::memory_order_acquire)) return VTI_OK;
  VTI_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  if (ctx->device < 64) done[ctx->device].store(true, std::memory_order_release);
  return VTI_OK;
}
static_assert(sizeof(float) * BackSmem<true>::floats(3) <= 226 * 1024 &&
                  sizeof(float) * BackSmem<true>::floats(4) <= 226 * 1024,
              "one backward CTA per SM");
std::atomic<bool> attr_fwd[2][kMaxT + 1][64], attr_bwd[2][kMaxT + 1][64];

#define TILE_TRY(x)                \
  do {                             \
    const int st_ = (x);           \
    if (st_ != VTI_OK) return st_; \
  } while (0)

}  // namespace

int launch_forward(vti_ctx* ctx, const Forward& a) {
  using Kernel = void (*)(Forward);
  static const Kernel kerns[2][kMaxT + 1] = {
      {nullptr, nullptr, k_tile_forward<false, 2>, k_tile_forward<false, 3>,
       k_tile_forward<false, 4>, k_tile_forward<false, 5>},
      {nullptr, nullptr, nullptr, k_tile_forward<true, 3>, k_tile_forward<true, 4>,
       k_tile_forward<true, 5>}};
  const int fused = a.keep_mode != kKeepNone;  // the gradient's and migration's arithmetic
  constexpr int bytes = kFieldsSmem * sizeof(float);
  const Kernel kern = kerns[fused][a.L.T];
  TILE_TRY(smem_attr(ctx, kern, bytes, attr_fwd[fused][a.L.T]));
  {
    LaunchTimer tm(ctx, kTimedStep2d);
    VTI_CUDA(ctx, launch_ex(true, kern, dim3(a.L.ntx, a.L.ntz, a.shots), dim3(kThreads), bytes,
                            ctx->stream, a));
  }
  VTI_LAUNCHED(ctx, "k_tile_forward");
  return VTI_OK;
}

int launch_backward(vti_ctx* ctx, const Backward& a) {
  using Kernel = void (*)(Backward);
  static const Kernel kerns[2][kMaxT + 1] = {
      {nullptr, nullptr, nullptr, k_tile_backward<false, 3>, k_tile_backward<false, 4>,
       k_tile_backward<false, 5>},
      {nullptr, nullptr, nullptr, k_tile_backward<true, 3>, k_tile_backward<true, 4>,
       k_tile_backward<true, 5>}};
  const int bytes =
      (a.exact ? BackSmem<true>::floats(a.L.T) : BackSmem<false>::floats(a.L.T)) * sizeof(float);
  const Kernel kern = kerns[a.exact ? 1 : 0][a.L.T];
  TILE_TRY(smem_attr(ctx, kern, bytes, attr_bwd[a.exact ? 1 : 0][a.L.T]));
  {
    LaunchTimer tm(ctx, kTimedStep2d);
    VTI_CUDA(ctx, launch_ex(true, kern, dim3(a.L.ntx, a.L.ntz), dim3(kThreads), bytes, ctx->stream,
                            a));
  }
  VTI_LAUNCHED(ctx, "k_tile_backward");
  return VTI_OK;
}

int launch_pad(vti_ctx* ctx, const Layout& L, const float* src, float* dst) {
  const int n = L.nnx * L.nnz;
  k_pad<true><<<(n + 255) / 256, 256, 0, ctx->stream>>>(L, src, dst, kHalo);
  VTI_LAUNCHED(ctx, "k_pad");
  return VTI_OK;
}
int launch_unpad(vti_ctx* ctx, const Layout& L, const float* src, float* dst) {
  const int n = L.nnx * L.nnz;
  k_pad<false><<<(n + 255) / 256, 256, 0, ctx->stream>>>(L, src, dst, kHalo);
  VTI_LAUNCHED(ctx, "k_unpad");
  return VTI_OK;
}
int launch_map(vti_ctx* ctx, const Layout& L, const int* cells, int n, int* map) {
  VTI_CUDA(ctx, cudaMemsetAsync(map, 0xff, L.n * sizeof(int), ctx->stream));
  if (n <= 0) return VTI_OK;
  k_map<<<(n + 127) / 128, 128, 0, ctx->stream>>>(cells, n, map);
  VTI_LAUNCHED(ctx, "k_map");
  return VTI_OK;
}
int launch_point(vti_ctx* ctx, float* a, float* b, int cell, float v) {
  k_point<<<1, 1, 0, ctx->stream>>>(a, b, cell, v);
  VTI_LAUNCHED(ctx, "k_point");
  return VTI_OK;
}
int launch_inject(vti_ctx* ctx, const Layout& L, float* p, float* q, const float* row,
                  const int* cells, int n, const float* taper, float dt2, int scale, int dipole) {
  if (n <= 0) return VTI_OK;
  k_inject_row<<<(n + 127) / 128, 128, 0, ctx->stream>>>(L, p, q, row, cells, n, taper, dt2, scale,
                                                         dipole);
  VTI_LAUNCHED(ctx, "k_inject_row");
  return VTI_OK;
}

bool receivers_fit(int nnx, int nnz, const int* rloc, int n, bool dipole) {
  std::vector<long long> cells(n);
  for (int ir = 0; ir < n; ++ir) {
    const int x = rloc[2 * ir], z = rloc[2 * ir + 1];
    if (x < kHalo || x >= nnx - kHalo || z < kHalo || z + (dipole ? 1 : 0) >= nnz - kHalo)
      return false;
    cells[ir] = x + (long long)z * nnx;
  }
  std::sort(cells.begin(), cells.end());
  return std::adjacent_find(cells.begin(), cells.end()) == cells.end();
}

}  // namespace tile2d
}  // namespace vti
