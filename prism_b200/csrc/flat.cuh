// Predictor and reconstruction of fields with one plane (nz == 1: 2-D and 1-D
// fields), one warp per 16x16 tile.
//
// The expressions, stages and boundary orders are those of the 3-D tiles
// (predict.cuh) with every point at z = 0, where the stages along z, two of
// the three face families and the cube have no points.  A 3-D tile spends a
// CTA of 256 threads, a 17^3 window, some twenty block-wide barriers and a
// 4096-point write-out on such a tile's 256 points; here a tile is a 17^2
// window of one warp (stages separated by warp barriers), eight tiles a CTA,
// and a code goes to its level-major slot as soon as it is made.
// 1799x901 float: 107 us as 3-D edge tiles, 15 us here (the latency of a
// tile's dozen stages).
#pragma once
#include "predict.cuh"

namespace prism_b200 {

constexpr int kFlatWarps = 8;
constexpr int kFlatWin = kWin * kWin;

PRISM_HD bool is_flat(const Geometry& g) { return g.nz == 1; }
PRISM_HD uint64_t flat_ctas(const Geometry& g) { return ((uint64_t)g.ax * g.ay + kFlatWarps - 1) / kFlatWarps; }

template <class T, bool COMPRESS>
struct FlatTile {
  T* win;  // (x, y) at 17 y + x
  const Geometry& g;
  int32_t* qc;              // compression: the code buffer
  const PredParams<T>* pp;
  uint32_t gs[2];           // window origin
  int r[2], l3[2], l1[2];   // AxisLimits of x and y

  __device__ __forceinline__ FlatTile(T* w, const Geometry& geo, int32_t* codes, const PredParams<T>* p, uint32_t tile)
      : win(w), g(geo), qc(codes), pp(p) {
    const uint32_t b[2] = {tile % geo.ax, tile / geo.ax}, n[2] = {geo.ax, geo.ay}, dim[2] = {geo.nx, geo.ny};
#pragma unroll
    for (int d = 0; d < 2; ++d) {
      gs[d] = b[d] * 16u;
      const bool last = b[d] == n[d] - 1;
      const int left = (int)min(dim[d] - gs[d], 17u);
      r[d] = last ? left : kWin;
      l3[d] = last ? min(16, left - 1) : 16;
      l1[d] = last ? left - 1 : 1 << 20;
    }
  }
  // level-major slot of a point of level `lv` (lm_slot at z = 0)
  __device__ __forceinline__ uint64_t slot(int lv, int x, int y) const {
    const uint64_t gx = (uint64_t)(gs[0] + x) >> lv, gy = (uint64_t)(gs[1] + y) >> lv;
    return g.lm_prefix[lv] + gx + gy * g.leaps[lv][0] - ((gy + 1) >> 1) * g.leaps[lv + 1][0] -
           (uint64_t)((gy & 1) == 0) * ((gx + 1) >> 1);
  }
  template <int U>
  __device__ __forceinline__ int order(int d, int c) const {  // order_of with this tile's limits
    const bool f3 = c + 3 * U <= l3[d], f1 = c + U <= l1[d];
    return c >= 3 * U ? (f3 ? 4 : (f1 ? 3 : 0)) : (f3 ? 2 : (f1 ? 1 : 0));
  }
  // line_at with neighbours s slots apart
  __device__ __forceinline__ T line(const T* w, int s, int o, bool md) const {
    using E = Expr<T>;
    const T t1 = w[-s];
    if (o == 0) return t1;
    const T t2 = w[s];
    if (o == 4) {
      const T t0 = w[-3 * s], t3 = w[3 * s];
      return md ? E::cubic_md(t0, t1, t2, t3) : E::cubic_axis(t0, t1, t2, t3, false);
    }
    if (o == 3) return E::quad_l(w[-3 * s], t1, t2);
    if (o == 2) return E::quad_r(t1, t2, w[3 * s]);
    return E::lin(t1, t2);
  }
  // face_at of a point odd along y (the reference's a1) and x (a2)
  __device__ __forceinline__ T face(const T* w, int sy, int sx, int oy, int ox) const {
    using E = Expr<T>;
    using F = Fp<T>;
    if (ox == 4 || oy == 4) {
      if (oy != 4) return line(w, sx, ox, true);
      if (ox != 4) return line(w, sy, oy, true);
      return E::half(F::add(line(w, sy, oy, true), line(w, sx, ox, true)));
    }
    if ((oy >= 2 && ox >= 2) || (oy == 1 && ox == 1))
      return E::half(F::add(line(w, sy, oy, true), line(w, sx, ox, true)));
    if (oy >= 2 || (oy == 1 && ox == 0)) return line(w, sy, oy, true);
    if (ox >= 1) return line(w, sx, ox, true);
    return F::sub(F::add(w[-sy], w[-sx]), w[-sy - sx]);
  }
  __device__ __forceinline__ void emit(int lv, int x, int y, T ebr, T ebx2, T pred) const {
    T& v = win[kWin * y + x];
    if constexpr (COMPRESS) {
      T rec;
      const int32_t code = quantize(v, pred, ebr, ebx2, &rec);
      if ((x | y) < 16) qc[slot(lv, x, y)] = code;
      v = rec;
    } else {
      int32_t c;
      if constexpr (sizeof(T) == 8) c = __double2loint(v);
      else c = __float_as_int(v);
      v = Fp<T>::fma(Fp<T>::from_int(c), ebx2, pred);
    }
  }
  // the points x = U (SX i + OX), i < NX, y alike; AX 0 or 1: predicted along
  // that axis, 2: faces
  template <int U, int AX, int NX, int SX, int OX, int NY, int SY, int OY>
  __device__ __forceinline__ void stage(int lv, bool md, T ebr, T ebx2) const {
#pragma unroll 1
    for (int i = threadIdx.x & 31; i < NX * NY; i += 32) {
      const int x = U * (SX * (i % NX) + OX), y = U * (SY * (i / NX) + OY);
      if (x >= r[0] || y >= r[1]) continue;
      const T* w = win + kWin * y + x;
      T pred;
      if constexpr (AX == 0) pred = line(w, U, order<U>(0, x), md);
      else if constexpr (AX == 1) pred = line(w, kWin * U, order<U>(1, y), md);
      else pred = face(w, kWin * U, U, order<U>(1, y), order<U>(0, x));
      emit(lv, x, y, ebr, ebx2, pred);
    }
  }
  template <int U, int LEVEL>
  __device__ __forceinline__ void level() const {
    if (LEVEL > pp->maxlevel) return;
    constexpr int N = 16 / (2 * U);
    const T ebr = pp->ebr[LEVEL], ebx2 = pp->ebx2[LEVEL];
    if (pp->use_md[LEVEL]) {
      stage<U, 0, N, 2, 1, N + 1, 2, 0>(LEVEL, true, ebr, ebx2);
      stage<U, 1, N + 1, 2, 0, N, 2, 1>(LEVEL, true, ebr, ebx2);
      __syncwarp();
      stage<U, 2, N, 2, 1, N, 2, 1>(LEVEL, true, ebr, ebx2);
    } else if (pp->reverse[LEVEL]) {  // x, then y
      stage<U, 0, N, 2, 1, N + 1, 2, 0>(LEVEL, false, ebr, ebx2);
      __syncwarp();
      stage<U, 1, 2 * N + 1, 1, 0, N, 2, 1>(LEVEL, false, ebr, ebx2);
    } else {  // y, then x
      stage<U, 1, N + 1, 2, 0, N, 2, 1>(LEVEL, false, ebr, ebx2);
      __syncwarp();
      stage<U, 0, N, 2, 1, 2 * N + 1, 1, 0>(LEVEL, false, ebr, ebx2);
    }
    __syncwarp();
  }
  __device__ __forceinline__ void sweep() const {
    level<8, 3>();
    level<4, 2>();
    level<2, 1>();
    level<1, 0>();
  }
};

constexpr int kFlatLoads = (kFlatWin + 31) / 32;

template <class T>
__device__ __forceinline__ void flat_compress_tile(T* win, const T* __restrict__ data, const Geometry& g, uint32_t tile,
                                                   const PredParams<T>* pp, T* __restrict__ anchors,
                                                   int32_t* __restrict__ qc) {
  const FlatTile<T, true> t(win, g, qc, pp, tile);
  const int lane = threadIdx.x & 31;
  const T* base = data + (uint64_t)t.gs[1] * g.nx + t.gs[0];
  T v[kFlatLoads];
#pragma unroll
  for (int k = 0; k < kFlatLoads; ++k) {
    const int i = lane + 32 * k, x = i % kWin, y = i / kWin;
    v[k] = T(0);
    if (i < kFlatWin && x < t.r[0] && y < t.r[1]) v[k] = __ldg(base + (uint64_t)y * g.nx + x);
  }
#pragma unroll
  for (int k = 0; k < kFlatLoads; ++k)
    if (lane + 32 * k < kFlatWin) win[lane + 32 * k] = v[k];
  if (lane == 0) anchors[tile] = v[0];
  __syncwarp();
  t.sweep();
}

template <class T>
__global__ void __launch_bounds__(kFlatWarps * 32)
flat_compress_kernel(const T* __restrict__ data, Geometry g, const PredParams<T>* pp,
                     T* __restrict__ anchors, int32_t* __restrict__ qc) {
  chain_wait();
  __shared__ T win[kFlatWarps][kFlatWin];
  const uint32_t tile = blockIdx.x * kFlatWarps + (threadIdx.x >> 5);
  if (tile < g.ax * g.ay) flat_compress_tile(win[threadIdx.x >> 5], data, g, tile, pp, anchors, qc);
}

template <class T, bool PROG>
__global__ void __launch_bounds__(kFlatWarps * 32)
flat_reconstruct_kernel(const int32_t* __restrict__ qc, const T* __restrict__ anchors, Geometry g,
                        const PredParams<T>* __restrict__ pp, const T* old, T* out) {
  __shared__ T wins[kFlatWarps][kFlatWin];
  const uint32_t tile = blockIdx.x * kFlatWarps + (threadIdx.x >> 5);
  if (tile >= g.ax * g.ay) return;
  T* win = wins[threadIdx.x >> 5];
  const FlatTile<T, false> t(win, g, nullptr, pp, tile);
  const int lane = threadIdx.x & 31, maxlevel = pp->maxlevel;
  // anchors at the corners, the other points' codes in the low words of
  // their slots (points of skipped levels and outside the field: zero)
  T v[kFlatLoads];
#pragma unroll
  for (int k = 0; k < kFlatLoads; ++k) {
    const int i = lane + 32 * k, x = i % kWin, y = i / kWin;
    v[k] = T(0);
    if (i < kFlatWin && x < t.r[0] && y < t.r[1]) {
      const int lv = win_level(x, y, 0);
      if (lv == 4) v[k] = anchors[tile + (x >> 4) + (y >> 4) * g.ax];
      else if (lv <= maxlevel) v[k] = Fp<T>::with_low_word(__ldg(qc + t.slot(lv, x, y)));
    }
  }
  T o[8];  // the previous values of the tile's 256 points
  const uint64_t base = (uint64_t)t.gs[1] * g.nx + t.gs[0];
  if (PROG) {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int i = lane + 32 * k, x = i & 15, y = i >> 4;
      o[k] = x < t.r[0] && y < t.r[1] ? old[base + (uint64_t)y * g.nx + x] : T(0);
    }
  }
#pragma unroll
  for (int k = 0; k < kFlatLoads; ++k)
    if (lane + 32 * k < kFlatWin) win[lane + 32 * k] = v[k];
  __syncwarp();
  t.sweep();
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int i = lane + 32 * k, x = i & 15, y = i >> 4;
    if (x >= t.r[0] || y >= t.r[1]) continue;
    const T val = win[kWin * y + x];
    out[base + (uint64_t)y * g.nx + x] = PROG ? Fp<T>::add(val, o[k]) : val;
  }
}

}  // namespace prism_b200
