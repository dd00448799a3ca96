// Multi-level cubic-spline predictor + error-bounded quantiser (compress) and
// the matching reconstruction (full and progressive), one 16^3 tile per CTA.
//
// Restates InterpolationPredictor.cu (interpolation :2137-2173,
// interpolation_reverse :2177-2207, interpolation_progressive_reverse
// :2209-2239): a tile works in a 17^3 shared-memory window (its own 16^3
// points plus the first plane of the next tile in x, y and z), sweeps levels
// 3..0 (unit 8, 4, 2, 1) and per level runs three stages: either
// line/face/cube ("md") or three axis sweeps in blue-yellow-hollow (z, y, x)
// order or its reverse.  Each stage predicts a set of independent points from
// already reconstructed ones, quantises the residual and reconstructs in
// place.  Codes go straight to their level-major slot (no linear scratch
// pass).  All arithmetic uses explicitly rounded intrinsics (fp.cuh) so the
// results equal the reference build bit for bit.
#pragma once
#include <type_traits>
#include "chain.cuh"
#include "fp.cuh"
#include "geometry.h"

namespace prism_b200 {

// Per-field predictor parameters, resident in device memory so a pipeline can
// compute them on the GPU (REL bound from the extrema kernel, flags from the
// auto-tuner) without a host round trip.
template <class T>
struct PredParams {
  T ebr[4];        // 1/eb scaled per level (calc_eb, :1825-1839)
  T ebx2[4];       // 2*eb scaled per level
  uint8_t use_md[4];
  uint8_t reverse[4];
  uint8_t natural[4];  // always 0: the tile sweeps use the default cubic
  int32_t maxlevel;  // levels above are skipped (:1848-1849)
};

template <class T>
struct Expr {
  using F = Fp<T>;
  // nan_cubic_interp (:1811-1813): (-a + 9b + 9c - d) / 16
  static __device__ __forceinline__ T cubic_md(T a, T b, T c, T d) {
    T s = F::fma(T(9), b, -a);
    s = F::fma(T(9), c, s);
    s = F::sub(s, d);
    return F::mul(s, T(0.0625));
  }
  // nat_cubic_interp (:1815-1817): (-3a + 23b + 23c - 3d) / 40
  static __device__ __forceinline__ T cubic_nat(T a, T b, T c, T d) {
    T s = F::fma(T(-3), a, F::mul(T(23), b));
    s = F::fma(T(23), c, s);
    s = F::fma(T(-3), d, s);
    return F::div(s, T(40));
  }
  static __device__ __forceinline__ T cubic_lambda(T a, T b, T c, T d, bool nat) {
    return nat ? cubic_nat(a, b, c, d) : cubic_md(a, b, c, d);
  }
  // per-axis cubic (:1248-1251, :1325): (p1 a + p2 b + p3 c + p4 d) / p5
  static __device__ __forceinline__ T cubic_axis(T a, T b, T c, T d, bool nat) {
    T p1 = nat ? T(-3) : T(-1), p2 = nat ? T(23) : T(9), p5 = nat ? T(40) : T(16);
    T s = F::fma(p1, a, F::mul(p2, b));
    s = F::fma(p2, c, s);
    s = F::fma(p1, d, s);
    // x/16 and x*0.0625 are the same real number, so they round identically
    return nat ? F::div(s, p5) : F::mul(s, T(0.0625));
  }
  // (-t0 + 6 t1 + 3 t2) / 8
  static __device__ __forceinline__ T quad_l(T t0, T t1, T t2) {
    T s = F::fma(T(6), t1, -t0);
    s = F::fma(T(3), t2, s);
    return F::mul(s, T(0.125));
  }
  // (3 t1 + 6 t2 - t3) / 8
  static __device__ __forceinline__ T quad_r(T t1, T t2, T t3) {
    T s = F::fma(T(3), t1, F::mul(T(6), t2));
    s = F::sub(s, t3);
    return F::mul(s, T(0.125));
  }
  // the same expression inside the md cube stage is contracted the other way
  // round: fma(6, t2, 3*t1) - t3 (measured against the reference build)
  static __device__ __forceinline__ T quad_r_cube(T t1, T t2, T t3) {
    T s = F::fma(T(6), t2, F::mul(T(3), t1));
    s = F::sub(s, t3);
    return F::mul(s, T(0.125));
  }
  static __device__ __forceinline__ T lin(T a, T b) { return F::mul(F::add(a, b), T(0.5)); }
  static __device__ __forceinline__ T half(T a) { return F::mul(a, T(0.5)); }
};

constexpr int kWin = 17;
constexpr int kWinVol = kWin * kWin * kWin;

// Window layout of the tile kernels: the slot of window point (x, y, z) is
//   x + 17 y + (y >> 1) + RZ z + SZ (z >> 1)
// (double: RZ = 297, SZ = 0, 5049 slots; float: RZ = 299, SZ = 3, 5105).
// Every stage of a sweep touches points of one parity class; in a plain
// 17^3 layout their slots differ by even multiples of the pitches, so a warp
// uses half of the shared-memory banks (double: 8 of the 16 bank pairs) and
// each access costs at least twice its wavefronts.  The skews after every
// second row and plane spread a class over all banks.  The constants minimise
// the wavefronts of the level-0 stages' lane-by-lane accesses over this
// family of layouts (with the stage-to-lane maps below), within the
// shared-memory budget of four double compression tiles per SM.
template <class T>
struct Win {
  static constexpr int RY = 17, SY = 1;
  static constexpr int RZ = sizeof(T) == 8 ? 297 : 299, SZ = sizeof(T) == 8 ? 0 : 3;
  // the part of a slot that coordinate c along axis d contributes
  static __host__ __device__ constexpr int axis(int d, int c) {
    return d == 0 ? c : (d == 1 ? RY * c + SY * (c >> 1) : RZ * c + SZ * (c >> 1));
  }
  static __host__ __device__ constexpr int at(int x, int y, int z) { return axis(0, x) + axis(1, y) + axis(2, z); }
  static constexpr int kSize = at(16, 16, 16) + 1;
  // slots between coordinates c and c + 2 along axis d (the same for every c)
  static __host__ __device__ constexpr int step2(int d) { return d == 0 ? 2 : (d == 1 ? 2 * RY + SY : 2 * RZ + SZ); }
  // slots between coordinates 2m and 2m + 1 along axis d
  static __host__ __device__ constexpr int one(int d) { return d == 0 ? 1 : (d == 1 ? RY : RZ); }
  static __host__ __device__ constexpr int skew(int d) { return d == 0 ? 0 : (d == 1 ? SY : SZ); }
};

// Slot offsets of the neighbours -3u, -u, +u, +3u of a point along one axis.
// Around an odd coordinate (u = 1) the skew makes them uneven; around an even
// coordinate with an even unit u they are multiples of step2.
struct Nb {
  int m3, m1, p1, p3;
};
template <class T>
__device__ __forceinline__ Nb nb_odd(int d) {
  using W = Win<T>;
  const int r = W::one(d), k = W::skew(d);
  return {-3 * r - k, -r, r + k, 3 * r + 2 * k};
}
template <class T>
__device__ __forceinline__ Nb nb_even(int d, int u) {
  const int s = (u >> 1) * Win<T>::step2(d);
  return {-3 * s, -s, s, 3 * s};
}

// Word of the compression tile's code block (16^3 int32) that holds the code
// of own point i = x + 16 y + 256 z: x XOR a function of the row.  A stage's
// lanes write the same x of different rows, which in the plain layout (row
// pitch 16 words) falls into one or two banks; the row-dependent XOR (a
// permutation within each row, so the block keeps its size) spreads them,
// and a row still reads out as 16 distinct banks.
__device__ __forceinline__ int cw_term(int y, int z) { return z + 2 * (y >> 1) + 3 * (z >> 1); }
__device__ __forceinline__ int cw_word(int i) { return i ^ (cw_term((i >> 4) & 15, i >> 8) & 15); }
// The term along a job's odd points (coordinate 2j + 1 along axis J) is
// t0 + j step(J): computed once per job instead of from each point's index
// (1024^3 floats 5228 -> 5165 us, 384x384x256 doubles 281 -> 276 us).
__device__ __forceinline__ int cw_term_step(int J) { return J == 0 ? 0 : (J == 1 ? 2 : 5); }
__device__ __forceinline__ int cw_term_first(int J, int cw0) {  // of point 0 (coordinate 1)
  const int y = (cw0 >> 4) & 15, z = cw0 >> 8;
  return J == 2 ? cw_term(y, 0) + 1 : cw_term(y, z);
}

// FAST marks an interior tile: its whole 17^3 window lies inside the field and
// it is not the last tile along any axis, so every boundary test below folds
// to a constant.  Both forms evaluate the same expressions on the same values.
template <class T, bool FAST = false>
struct TileCtx {
  T* s;  // shared window, s[(z*17 + y)*17 + x]
  uint32_t gs[3];      // global start of the window (uint32 arithmetic)
  bool notlast_[3];    // the window does not reach the field's end
  uint32_t dim[3];
  // per-axis fields through selects (a dynamic index would move the context
  // to local memory)
  __device__ __forceinline__ bool notlast(int d) const {
    return FAST ? true : (d == 0 ? notlast_[0] : (d == 1 ? notlast_[1] : notlast_[2]));
  }
  __device__ __forceinline__ uint32_t start(int d) const { return d == 0 ? gs[0] : (d == 1 ? gs[1] : gs[2]); }
  __device__ __forceinline__ uint32_t extent(int d) const { return d == 0 ? dim[0] : (d == 1 ? dim[1] : dim[2]); }
  __device__ __forceinline__ T& at(int x, int y, int z) const { return s[(z * kWin + y) * kWin + x]; }
  __device__ __forceinline__ T get(int axis, int x, int y, int z, int c) const {
    return axis == 0 ? at(c, y, z) : (axis == 1 ? at(x, c, z) : at(x, y, c));
  }
  __device__ __forceinline__ bool in_data(int x, int y, int z) const {
    if (FAST) return true;
    return gs[0] + (uint32_t)x < dim[0] && gs[1] + (uint32_t)y < dim[1] && gs[2] + (uint32_t)z < dim[2];
  }
  // xyz_predicate (:1173-1185); the exclusive form is used by the last stage
  // of level 0
  __device__ __forceinline__ bool pred_ok(int x, int y, int z, bool inclusive) const {
    if (inclusive) return in_data(x, y, z);
    return x < 16 && y < 16 && z < 16 + !notlast(2) && in_data(x, y, z);
  }
  __device__ __forceinline__ bool owned(int x, int y, int z) const {
    return (x < 16 || !notlast(0)) && (y < 16 || !notlast(1)) && (z < 16 || !notlast(2));
  }
};

__device__ __forceinline__ int nb_idx(int c, int u, int k) {  // id_x/id_y/id_z (:1426-1439)
  switch (k) {
    case 0: return c - 3 * u >= 0 ? c - 3 * u : 0;
    case 1: return c - u >= 0 ? c - u : 0;
    case 2: return c + u <= 16 ? c + u : 0;
    default: return c + 3 * u <= 16 ? c + 3 * u : 0;
  }
}

// 1-D prediction with the per-axis boundary cases (:1300-1326, :1506-1535)
template <class T, bool FAST>
__device__ __forceinline__ T pred_line(const TileCtx<T, FAST>& t, int axis, int x, int y, int z, int u,
                                       bool md, bool nat) {
  using E = Expr<T>;
  int ix = axis == 0 ? x : (axis == 1 ? y : z);
  uint32_t gx = t.start(axis) + (uint32_t)ix, gs = t.extent(axis);
  bool c1 = t.notlast(axis);
  bool c2 = ix >= 3 * u, c3 = ix + 3 * u <= 16;
  bool c4 = gx + 3u * u < gs, c5 = gx + (uint32_t)u < gs;
  T t1 = t.get(axis, x, y, z, nb_idx(ix, u, 1));
  if ((c1 && !c2 && !c3) || (!c1 && !c2 && !(c3 && c4) && c5))
    return E::lin(t1, t.get(axis, x, y, z, nb_idx(ix, u, 2)));
  if ((c1 && !c2 && c3) || (!c1 && !c2 && c3 && c4))
    return E::quad_r(t1, t.get(axis, x, y, z, nb_idx(ix, u, 2)), t.get(axis, x, y, z, nb_idx(ix, u, 3)));
  if ((c1 && c2 && !c3) || (!c1 && c2 && !(c3 && c4) && c5))
    return E::quad_l(t.get(axis, x, y, z, nb_idx(ix, u, 0)), t1, t.get(axis, x, y, z, nb_idx(ix, u, 2)));
  if ((c1 && c2 && c3) || (!c1 && c2 && c3 && c4)) {
    T t0 = t.get(axis, x, y, z, nb_idx(ix, u, 0)), t2 = t.get(axis, x, y, z, nb_idx(ix, u, 2));
    T t3 = t.get(axis, x, y, z, nb_idx(ix, u, 3));
    return md ? E::cubic_lambda(t0, t1, t2, t3, nat) : E::cubic_axis(t0, t1, t2, t3, nat);
  }
  return t1;
}

// get_interp_order (:1538-1545): 4 cubic, 3 quad-left, 2 quad-right, 1 linear, 0 none
template <class T, bool FAST>
__device__ __forceinline__ int interp_order(const TileCtx<T, FAST>& t, int axis, int c, int u) {
  uint32_t gx = t.start(axis) + (uint32_t)c, gs = t.extent(axis);
  bool notlast = t.notlast(axis);
  int b = c >= 3 * u ? 3 : 1;
  int f = (c + 3 * u <= 16 && (notlast || gx + 3u * u < gs)) ? 3 : ((notlast || gx + (uint32_t)u < gs) ? 1 : 0);
  return b == 3 ? (f == 3 ? 4 : (f == 1 ? 3 : 0)) : (f == 3 ? 2 : (f == 1 ? 1 : 0));
}

// FACE (:1546-1668)
template <class T, bool FAST>
__device__ __forceinline__ T pred_face(const TileCtx<T, FAST>& t, int x, int y, int z, int u, bool nat) {
  using E = Expr<T>;
  using F = Fp<T>;
  int a1, a2;
  T pred;
  if (x % (2 * u) == 0) { a1 = 2; a2 = 1; pred = t.at(x, nb_idx(y, u, 1), nb_idx(z, u, 1)); }
  else if (y % (2 * u) == 0) { a1 = 2; a2 = 0; pred = t.at(nb_idx(x, u, 1), y, nb_idx(z, u, 1)); }
  else { a1 = 1; a2 = 0; pred = t.at(nb_idx(x, u, 1), nb_idx(y, u, 1), z); }
  int c1 = a1 == 1 ? y : z, c2 = a2 == 0 ? x : y;
  T s1[4], s2[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    s1[k] = t.get(a1, x, y, z, nb_idx(c1, u, k));
    s2[k] = t.get(a2, x, y, z, nb_idx(c2, u, k));
  }
  int i1 = interp_order(t, a1, c1, u), i2 = interp_order(t, a2, c2, u);
  if (i1 == 4 && i2 == 4)
    return E::half(F::add(E::cubic_lambda(s1[0], s1[1], s1[2], s1[3], nat),
                          E::cubic_lambda(s2[0], s2[1], s2[2], s2[3], nat)));
  if (i1 != 4 && i2 == 4) return E::cubic_lambda(s2[0], s2[1], s2[2], s2[3], nat);
  if (i1 == 4 && i2 != 4) return E::cubic_lambda(s1[0], s1[1], s1[2], s1[3], nat);
  if (i1 == 3 && i2 == 3) return E::half(F::add(E::quad_l(s2[0], s2[1], s2[2]), E::quad_l(s1[0], s1[1], s1[2])));
  if (i1 == 3 && i2 == 2) return E::half(F::add(E::quad_r(s2[1], s2[2], s2[3]), E::quad_l(s1[0], s1[1], s1[2])));
  if (i1 == 3 && i2 < 2) return E::quad_l(s1[0], s1[1], s1[2]);
  if (i1 == 2 && i2 == 3) return E::half(F::add(E::quad_r(s1[1], s1[2], s1[3]), E::quad_l(s2[0], s2[1], s2[2])));
  if (i1 == 2 && i2 == 2) return E::half(F::add(E::quad_r(s1[1], s1[2], s1[3]), E::quad_r(s2[1], s2[2], s2[3])));
  if (i1 == 2 && i2 < 2) return E::quad_r(s1[1], s1[2], s1[3]);
  if (i1 <= 1 && i2 == 3) return E::quad_l(s2[0], s2[1], s2[2]);
  if (i1 <= 1 && i2 == 2) return E::quad_r(s2[1], s2[2], s2[3]);
  if (i1 == 1 && i2 == 1) return E::half(F::add(E::lin(s2[1], s2[2]), E::lin(s1[1], s1[2])));
  if (i1 == 1 && i2 < 1) return E::lin(s1[1], s1[2]);
  if (i1 == 0 && i2 == 1) return E::lin(s2[1], s2[2]);
  return F::sub(F::add(s1[1], s2[1]), pred);
}

// CUBE (:1671-1723)
template <class T, bool FAST>
__device__ __forceinline__ T pred_cube(const TileCtx<T, FAST>& t, int x, int y, int z, int u, bool nat) {
  using E = Expr<T>;
  using F = Fp<T>;
  int oz = interp_order(t, 2, z, u), oy = interp_order(t, 1, y, u), ox = interp_order(t, 0, x, u);
  T tx[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) tx[k] = t.at(nb_idx(x, u, k), y, z);
  auto cz = [&]() { return E::cubic_lambda(t.at(x, y, nb_idx(z, u, 0)), t.at(x, y, nb_idx(z, u, 1)),
                                           t.at(x, y, nb_idx(z, u, 2)), t.at(x, y, nb_idx(z, u, 3)), nat); };
  auto cy = [&]() { return E::cubic_lambda(t.at(x, nb_idx(y, u, 0), z), t.at(x, nb_idx(y, u, 1), z),
                                           t.at(x, nb_idx(y, u, 2), z), t.at(x, nb_idx(y, u, 3), z), nat); };
  auto cx = [&]() { return E::cubic_lambda(tx[0], tx[1], tx[2], tx[3], nat); };
  if (oz == 4 && oy == 4 && ox == 4) return F::div(F::add(F::add(cx(), cy()), cz()), T(3));
  if (oz == 4 && oy == 4) return E::half(F::add(cz(), cy()));
  if (oz == 4 && ox == 4) return E::half(F::add(cz(), cx()));
  if (oy == 4 && ox == 4) return E::half(F::add(cy(), cx()));
  if (oz == 4) return cz();
  if (oy == 4) return cy();
  if (ox == 4) return cx();
  if (ox == 3) return E::quad_l(tx[0], tx[1], tx[2]);
  if (ox == 2) return E::quad_r_cube(tx[1], tx[2], tx[3]);
  if (ox == 1) return E::lin(tx[1], tx[2]);
  return tx[1];
}

// Quantise one residual (:1330-1342) and reconstruct; returns the code.
template <class T>
__device__ __forceinline__ int32_t quantize(T orig, T pred, T ebr, T ebx2, T* rec) {
  using F = Fp<T>;
  T err = F::sub(orig, pred);
  T code = F::fma(F::abs(err), ebr, T(1));
  code = err < T(0) ? -code : code;
  int qi = F::to_int_rz(F::mul(code, T(0.5)));
  T qt = F::from_int(qi);
  *rec = F::fma(qt, ebx2, pred);
  // the code is (int)qt: qi itself for double (every int is exact there);
  // float rounds |qi| > 2^24, so it converts back
  if constexpr (sizeof(T) == 8) return qi;
  else return F::to_int_rz(qt);
}

constexpr int kPredThreads = 256;
constexpr int kPrefetch = 8;  // independent global loads in flight per thread

// Asynchronous global -> shared copies (cp.async, no register staging): a
// thread issues every copy of its window points before waiting for any, and
// after cp.async.wait_all sees the data it copied itself.
template <int BYTES>
__device__ __forceinline__ void copy_async(void* smem_dst, const void* gmem_src) {
  static_assert(BYTES == 4 || BYTES == 8, "4- or 8-byte copies");
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(d), "l"(gmem_src), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void copy_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }
__device__ __forceinline__ void copy_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
// wait until at most N of this thread's committed groups are still in flight
template <int N>
__device__ __forceinline__ void copy_async_wait_group() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// ---- tile sweep --------------------------------------------------------------
//
// Every boundary case of pred_line / pred_face / pred_cube depends only on
// the point's coordinate c along each interpolation axis and on three per-axis
// limits of the tile:
//   f3 (the +3u neighbour exists):  c + 3u <= L3  (L3 = 16, or min(16, r-1)
//                                                  on the field's last tile)
//   f1 (the +u neighbour exists):   c + u  <= L1  (no limit, or r-1)
//   in data:                        c < R          (17, or r)
// where r = extent - tile start.  interp_order (:1538-1545) becomes
// order = c >= 3u ? (f3 ? 4 : f1 ? 3 : 0) : (f3 ? 2 : f1 ? 1 : 0), and the
// neighbours sit at fixed offsets from the point in the window.  The functions
// below evaluate exactly the expressions the generic ones choose, in the same
// operation order, with the neighbours addressed directly.  For interior tiles
// (EDGE = false) the limits are constants.  Points are enumerated with an axis
// the prediction does not interpolate along varying fastest, so a warp mostly
// shares one formula.

struct AxisLimits {
  int l3[3], l1[3], r[3];
};

template <bool EDGE>
struct Limits {
  AxisLimits a;  // by value: stays in registers
  __device__ __forceinline__ int l3(int d) const { return EDGE ? a.l3[d] : 16; }
  __device__ __forceinline__ int l1(int d) const { return EDGE ? a.l1[d] : 1 << 20; }
  __device__ __forceinline__ int r(int d) const { return EDGE ? a.r[d] : kWin; }
  __device__ __forceinline__ bool in_data(int x, int y, int z) const {
    return EDGE ? (x < a.r[0] && y < a.r[1] && z < a.r[2]) : true;
  }
};

template <int U, bool EDGE, int D>
__device__ __forceinline__ int order_of(const Limits<EDGE>& L, int c) {
  const bool b = c >= 3 * U, f3 = c + 3 * U <= L.l3(D), f1 = c + U <= L.l1(D);
  return b ? (f3 ? 4 : (f1 ? 3 : 0)) : (f3 ? 2 : (f1 ? 1 : 0));
}

// window slots between coordinates c and c + U along axis D, U even
template <class T, int U, int D>
constexpr int unit_stride() {
  static_assert(U % 2 == 0, "even units");
  return (U / 2) * Win<T>::step2(D);
}

// 1-D prediction along window axis D at coordinate c (pred_line :1300-1326)
template <class T, int U, int D, bool MD>
__device__ __forceinline__ T line_at(const T* w, int o, bool nat) {
  using E = Expr<T>;
  constexpr int S = unit_stride<T, U, D>();
  const T t1 = w[-S];
  if (o == 0) return t1;
  const T t2 = w[S];
  if (o == 4) {
    const T t0 = w[-3 * S], t3 = w[3 * S];
    return MD ? E::cubic_lambda(t0, t1, t2, t3, nat) : E::cubic_axis(t0, t1, t2, t3, nat);
  }
  if (o == 3) return E::quad_l(w[-3 * S], t1, t2);
  if (o == 2) return E::quad_r(t1, t2, w[3 * S]);
  return E::lin(t1, t2);
}

// FACE (:1546-1668): interpolation along axes D1 (the reference's a1) and D2
// (a2).  add() is commutative bit for bit, which folds the reference's operand
// orders into one form.
template <class T, int U, int D1, int D2>
__device__ __forceinline__ T face_at(const T* w, int o1, int o2, bool nat) {
  using E = Expr<T>;
  using F = Fp<T>;
  if (o1 == 4 || o2 == 4) {
    if (o1 != 4) return line_at<T, U, D2, true>(w, o2, nat);
    if (o2 != 4) return line_at<T, U, D1, true>(w, o1, nat);
    return E::half(F::add(line_at<T, U, D1, true>(w, o1, nat), line_at<T, U, D2, true>(w, o2, nat)));
  }
  if ((o1 >= 2 && o2 >= 2) || (o1 == 1 && o2 == 1))
    return E::half(F::add(line_at<T, U, D1, true>(w, o1, nat), line_at<T, U, D2, true>(w, o2, nat)));
  if (o1 >= 2 || (o1 == 1 && o2 == 0)) return line_at<T, U, D1, true>(w, o1, nat);
  if (o2 >= 1) return line_at<T, U, D2, true>(w, o2, nat);
  constexpr int S1 = unit_stride<T, U, D1>(), S2 = unit_stride<T, U, D2>();
  return F::sub(F::add(w[-S1], w[-S2]), w[-S1 - S2]);
}

// CUBE (:1671-1723)
template <class T, int U>
__device__ __forceinline__ T cube_at(const T* w, int ox, int oy, int oz, bool nat) {
  using E = Expr<T>;
  using F = Fp<T>;
  auto cub = [&](auto D) {
    constexpr int s = unit_stride<T, U, decltype(D)::value>();
    return E::cubic_lambda(w[-3 * s], w[-s], w[s], w[3 * s], nat);
  };
  using DX = std::integral_constant<int, 0>;
  using DY = std::integral_constant<int, 1>;
  using DZ = std::integral_constant<int, 2>;
  if (oz == 4 && oy == 4 && ox == 4) return F::div(F::add(F::add(cub(DX()), cub(DY())), cub(DZ())), T(3));
  if (oz == 4 && oy == 4) return E::half(F::add(cub(DZ()), cub(DY())));
  if (oz == 4 && ox == 4) return E::half(F::add(cub(DZ()), cub(DX())));
  if (oy == 4 && ox == 4) return E::half(F::add(cub(DY()), cub(DX())));
  if (oz == 4) return cub(DZ());
  if (oy == 4) return cub(DY());
  if (ox == 4) return cub(DX());
  constexpr int SX = unit_stride<T, U, 0>();
  if (ox == 3) return E::quad_l(w[-3 * SX], w[-SX], w[SX]);
  if (ox == 2) return E::quad_r_cube(w[-SX], w[SX], w[3 * SX]);
  if (ox == 1) return E::lin(w[-SX], w[SX]);
  return w[-SX];
}

// One level (unit U) of a tile sweep.
// In a compression, levels 3 and 2 (U = 8, 4; at most 50 points a stage) are
// swept by warp 0 alone, with warp barriers between their six stages: the
// other warps wait once instead of stepping through every stage's loop and
// barrier.  (The reconstruction, with more tiles an SM and less to do per
// point, was 1.5% slower that way: 1885 -> 1914 us on 1000x777x513 floats.)
template <class T, bool COMPRESS, int U, bool EDGE>
struct LevelSweep {
  static constexpr int N = 16 / (2 * U);
  static constexpr bool kWarp = COMPRESS && U >= 4;
  static constexpr int kThreads = kWarp ? 32 : kPredThreads;
  static __device__ __forceinline__ void sync() {
    if constexpr (kWarp) __syncwarp();
    else __syncthreads();
  }
  T* win;
  int32_t* cw;
  Limits<EDGE> L;
  bool zlast;  // the tile is the last along z (exclusive form allows z = 16)
  T ebr, ebx2;
  // The tile sweeps evaluate the default cubic (nan_cubic_interp): the
  // natural cubic is selected only by the reference's hidden `-cubic
  // natural` test flag (parameters.cu:199-204), which this library does not
  // offer (PredParams::natural is always 0; the auto-tuner still sums the
  // natural candidate's errors with its own code).  A compile-time constant
  // removes a branch per cubic and the unused form's division from every
  // stage.
  static constexpr bool nat = false;

  // The reconstruction keeps each point's code as an int32 in the low word of
  // the point's own window slot until the point is predicted (no prediction
  // reads a point of its own or a later stage), and converts it there.
  __device__ __forceinline__ T code_of(int wi) const {
    const T v = win[wi];  // read as T, then the low word: no type-punned access
    int32_t c;
    if constexpr (sizeof(T) == 8) c = __double2loint(v);
    else c = __float_as_int(v);
    return Fp<T>::from_int(c);
  }
  // Compression keeps the codes of the tile's own 16^3 points only (the
  // codes of the shared faces belong to the neighbouring tiles).
  __device__ __forceinline__ void emit(int wi, const int c[3], T pred) const {
    if (COMPRESS) {
      T rec;
      const int32_t code = quantize(win[wi], pred, ebr, ebx2, &rec);
      if ((c[0] | c[1] | c[2]) < 16) cw[cw_word((c[2] * 16 + c[1]) * 16 + c[0])] = code;
      win[wi] = rec;
    } else {
      win[wi] = Fp<T>::fma(code_of(wi), ebx2, pred);
    }
  }
  // xyz_predicate (:1173-1185)
  __device__ __forceinline__ bool pred_ok(const int c[3], bool exclusive) const {
    if (!L.in_data(c[0], c[1], c[2])) return false;
    return !exclusive || (c[0] < 16 && c[1] < 16 && c[2] < 16 + (EDGE && zlast));
  }
  // Per-axis sweep along AX over a box of points.  Dimension d of the box has
  // ND points at window coordinate U*(k*STD + OFD); dimension 0 varies
  // fastest and is an axis other than AX.  AXES packs the window axis of
  // dimensions 0, 1, 2 (two bits each).
  template <int AX, bool MD, int AXES, int N0, int ST0, int OF0, int N1, int ST1, int OF1, int N2, int ST2, int OF2,
            bool SYNC = true>
  __device__ __forceinline__ void sweep(bool exclusive) const {
    constexpr int total = N0 * N1 * N2;
    constexpr int A0 = AXES & 3, A1 = (AXES >> 2) & 3, A2 = (AXES >> 4) & 3;
#pragma unroll 2
    for (int i = threadIdx.x; i < total; i += kThreads) {
      const int k0 = i % N0, k1 = (i / N0) % N1, k2 = i / (N0 * N1);
      int c[3];
      c[A0] = U * (k0 * ST0 + OF0);
      c[A1] = U * (k1 * ST1 + OF1);
      c[A2] = U * (k2 * ST2 + OF2);
      if (!pred_ok(c, exclusive)) continue;
      const int wi = Win<T>::at(c[0], c[1], c[2]);
      emit(wi, c, line_at<T, U, AX, MD>(win + wi, order_of<U, EDGE, AX>(L, c[AX]), nat));
    }
    if (SYNC) sync();
  }
  // md faces: the point is even along axis E (dimension 0, fastest) and odd
  // along the two interpolation axes P1 (the reference's a1) and P2 (a2)
  template <int E, int P1, int P2, bool SYNC = true>
  __device__ __forceinline__ void faces() const {
    constexpr int total = (N + 1) * N * N;
#pragma unroll 2
    for (int i = threadIdx.x; i < total; i += kThreads) {
      const int k0 = i % (N + 1), k1 = (i / (N + 1)) % N, k2 = i / ((N + 1) * N);
      int c[3];
      c[E] = 2 * U * k0;
      c[P1] = 2 * U * k1 + U;
      c[P2] = 2 * U * k2 + U;
      if (!pred_ok(c, false)) continue;
      const int wi = Win<T>::at(c[0], c[1], c[2]);
      emit(wi, c, face_at<T, U, P1, P2>(win + wi, order_of<U, EDGE, P1>(L, c[P1]), order_of<U, EDGE, P2>(L, c[P2]),
                                      nat));
    }
    if (SYNC) sync();
  }
  __device__ __forceinline__ void cube(bool exclusive) const {
    constexpr int total = N * N * N;
#pragma unroll 2
    for (int i = threadIdx.x; i < total; i += kThreads) {
      int c[3] = {2 * U * (i % N) + U, 2 * U * ((i / N) % N) + U, 2 * U * (i / (N * N)) + U};
      if (!pred_ok(c, exclusive)) continue;
      const int wi = Win<T>::at(c[0], c[1], c[2]);
      emit(wi, c, cube_at<T, U>(win + wi, order_of<U, EDGE, 0>(L, c[0]), order_of<U, EDGE, 1>(L, c[1]),
                             order_of<U, EDGE, 2>(L, c[2]), nat));
    }
    sync();
  }
  // Level 0 of an interior tile, per-axis mode, by lines: a job predicts the
  // odd points 2j+1, j in [J0, J1), of the line along AX through window point
  // (c[P], c[Q]) = (p, q).  The line's even points come from earlier stages
  // and every odd point reads only those, so the points of a job are
  // independent; the even points are read once per job.  Interior orders
  // (order_of with no limits): j = 0 quadratic from the right, j = 7
  // quadratic from the left, cubic in between.
  // order along an axis at odd coordinate c of an interior tile, level 0
  static __device__ __forceinline__ int order0(int c) { return c == 1 ? 2 : (c == 15 ? 3 : 4); }
  // ---- level 0 of an interior tile by jobs along one odd axis ------------
  // A job predicts the odd points 2j+1, j in [j0, j1), of a line with window
  // stride S.  cw0/cs locate the points' codes in the tile's 16^3 code block;
  // `own` tells whether the line's fixed coordinates lie in the tile's own
  // region.  Points go in groups: a group first reads every value it needs
  // (the line's even values E[g-1 .. g+G+1], its points' codes -- compression:
  // their original values -- and, for faces, the neighbours on the second
  // line), then predicts, then writes.  No point of a stage reads a point of
  // the same stage, so the reads of a group are in flight together instead
  // of each waiting behind the previous point's write.
  __device__ __forceinline__ void emit_at(int wi, int cwi, bool own, T pred) const {
    if (COMPRESS) {
      T rec;
      const int32_t code = quantize(win[wi], pred, ebr, ebx2, &rec);
      if (own) cw[cw_word(cwi)] = code;
      win[wi] = rec;
    } else {
      win[wi] = Fp<T>::fma(code_of(wi), ebx2, pred);
    }
  }
  // emit_at with the point's code (compression: its original value) read
  // beforehand and its code-block word known
  __device__ __forceinline__ void emit_read(int wi, int word, bool own, T v, T pred) const {
    if (COMPRESS) {
      T rec;
      const int32_t code = quantize(v, pred, ebr, ebx2, &rec);
      if (own) cw[word] = code;
      win[wi] = rec;
    } else {
      win[wi] = Fp<T>::fma(v, ebx2, pred);
    }
  }
  __device__ __forceinline__ T read_point(int wi) const { return COMPRESS ? win[wi] : code_of(wi); }
  // KIND 0: md line points (prediction along the job axis only);
  // KIND 2: per-axis points (the same with the per-axis cubic);
  // KIND 1: md faces, the job axis J and a second odd axis with stride SK
  // and order ok (face_at: both cubic -> the mean of the two lines, one cubic
  // -> that line, neither -> the mean; add() is commutative bit for bit).
  // Interior orders along the job axis: j = 0 quadratic from the right, j = 7
  // from the left, cubic in between.  j0 and j1 are multiples of the group.
  // w0: the slot of the line's point at coordinate 0 along the job axis J;
  // K: the second odd axis of a face job.
  template <int KIND>
  __device__ __forceinline__ void md_job(int w0, int J, int cw0, int cs, bool own, int j0, int j1, int K,
                                         int ok) const {
    using E = Expr<T>;
    using F = Fp<T>;
    constexpr int G = KIND == 1 ? 2 : 4;
    const int E2 = Win<T>::step2(J), O1 = Win<T>::one(J);  // even point e at w0 + e E2, odd point j at + O1
    const Nb nk = nb_odd<T>(K);
    const int t0 = cw_term_first(J, cw0), dt = cw_term_step(J);
#pragma unroll
    for (int g = 0; g < 8; g += G) {
      if (g < j0 || g >= j1) continue;
      T ev[G + 3];  // E[g - 1 + k]
#pragma unroll
      for (int k = 0; k < G + 3; ++k) {
        const int e = g - 1 + k;
        ev[k] = e >= 0 && e <= 8 ? win[w0 + e * E2] : T(0);
      }
      T v[G], k0[G], k1[G], k2[G], k3[G];  // faces: the second line at -3, -1, +1, +3
#pragma unroll
      for (int i = 0; i < G; ++i) {
        const int j = g + i;
        const int wi = w0 + j * E2 + O1;
        v[i] = read_point(wi);
        // the second line is read where face_at uses it: unless the job
        // axis alone is cubic
        if (KIND == 1 && (ok == 4 || j == 0 || j == 7)) {
          k1[i] = win[wi + nk.m1];
          k2[i] = win[wi + nk.p1];
          k0[i] = ok != 2 ? win[wi + nk.m3] : T(0);
          k3[i] = ok != 3 ? win[wi + nk.p3] : T(0);
        }
      }
#pragma unroll
      for (int i = 0; i < G; ++i) {
        const int j = g + i;
        const int oj = j == 0 ? 2 : (j == 7 ? 3 : 4);
        const T lj = oj == 4 ? (KIND == 2 ? E::cubic_axis(ev[i], ev[i + 1], ev[i + 2], ev[i + 3], nat)
                                          : E::cubic_lambda(ev[i], ev[i + 1], ev[i + 2], ev[i + 3], nat))
                             : (oj == 2 ? E::quad_r(ev[i + 1], ev[i + 2], ev[i + 3]) : E::quad_l(ev[i], ev[i + 1], ev[i + 2]));
        T pred = lj;
        if (KIND == 1 && !(oj == 4 && ok != 4)) {
          const T lk = ok == 4 ? E::cubic_lambda(k0[i], k1[i], k2[i], k3[i], nat)
                               : (ok == 3 ? E::quad_l(k0[i], k1[i], k2[i]) : E::quad_r(k1[i], k2[i], k3[i]));
          pred = (oj != 4 && ok == 4) ? lk : E::half(F::add(lj, lk));
        }
        emit_read(w0 + j * E2 + O1, (cw0 + (2 * j + 1) * cs) ^ ((t0 + j * dt) & 15), own, v[i], pred);
      }
    }
  }
  // md cube points (x odd, cy, cz) along x, j in [j0, j0 + 2): cube_at's
  // cases for interior orders with its summation order for three cubics.
  // The reads of both points come first (the directions along y and z only
  // where they are cubic).
  __device__ __forceinline__ void md_cube_job(int cy, int cz, int j0) const {
    using E = Expr<T>;
    using F = Fp<T>;
    const int w0 = Win<T>::at(0, cy, cz), cw0 = (cz * 16 + cy) * 16, term = cw_term(cy, cz) & 15;
    const int oy = order0(cy), oz = order0(cz);
    const Nb ny = nb_odd<T>(1), nz = nb_odd<T>(2);
    T ev[5];  // E[j0 - 1 + k] along x
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const int e = j0 - 1 + k;
      ev[k] = e >= 0 && e <= 8 ? win[w0 + 2 * e] : T(0);
    }
    T v[2], ya[2][4], za[2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int wi = w0 + 2 * (j0 + i) + 1;
      v[i] = read_point(wi);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int dy = k == 0 ? ny.m3 : (k == 1 ? ny.m1 : (k == 2 ? ny.p1 : ny.p3));
        const int dz = k == 0 ? nz.m3 : (k == 1 ? nz.m1 : (k == 2 ? nz.p1 : nz.p3));
        ya[i][k] = oy == 4 ? win[wi + dy] : T(0);
        za[i][k] = oz == 4 ? win[wi + dz] : T(0);
      }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int j = j0 + i;
      const int ox = j == 0 ? 2 : (j == 7 ? 3 : 4);
      const T p = ev[i], a = ev[i + 1], b = ev[i + 2], c = ev[i + 3];
      auto cyf = [&]() { return E::cubic_lambda(ya[i][0], ya[i][1], ya[i][2], ya[i][3], nat); };
      auto czf = [&]() { return E::cubic_lambda(za[i][0], za[i][1], za[i][2], za[i][3], nat); };
      T pred;
      if (ox == 4) {
        const T cx = E::cubic_lambda(p, a, b, c, nat);
        if (oz == 4 && oy == 4) pred = F::div(F::add(F::add(cx, cyf()), czf()), T(3));
        else if (oz == 4) pred = E::half(F::add(czf(), cx));
        else if (oy == 4) pred = E::half(F::add(cyf(), cx));
        else pred = cx;
      } else if (oz == 4 || oy == 4) {
        if (oz == 4 && oy == 4) pred = E::half(F::add(czf(), cyf()));
        else if (oz == 4) pred = czf();
        else pred = cyf();
      } else if (ox == 3) {
        pred = E::quad_l(p, a, b);
      } else {
        pred = E::quad_r_cube(a, b, c);
      }
      emit_read(w0 + 2 * j + 1, (cw0 + 2 * j + 1) ^ term, true, v[i], pred);
    }
  }
  // ---- level 0 of an edge tile (the last slab along some axis) by jobs ----
  // The same jobs as on interior tiles with the orders of order_of under the
  // tile's runtime limits, and with jobs and points outside the field
  // skipped (the generic sweeps skip them through pred_ok).
  __device__ __forceinline__ int lim3(int d) const { return d == 0 ? L.l3(0) : (d == 1 ? L.l3(1) : L.l3(2)); }
  __device__ __forceinline__ int lim1(int d) const { return d == 0 ? L.l1(0) : (d == 1 ? L.l1(1) : L.l1(2)); }
  __device__ __forceinline__ int lim_r(int d) const { return d == 0 ? L.r(0) : (d == 1 ? L.r(1) : L.r(2)); }
  // order_of at coordinate c (an odd multiple of the unit U)
  static __device__ __forceinline__ int order_rt(int c, int l3, int l1) {
    const bool f3 = c + 3 * U <= l3, f1 = c + U <= l1;
    return c >= 3 * U ? (f3 ? 4 : (f1 ? 3 : 0)) : (f3 ? 2 : (f1 ? 1 : 0));
  }
  // line_at from a job's sliding window (p, a, b, c) = E[j-1..j+2]
  template <bool MD>
  __device__ __forceinline__ T window_line(int o, T p, T a, T b, T c) const {
    using E = Expr<T>;
    if (o == 4) return MD ? E::cubic_lambda(p, a, b, c, nat) : E::cubic_axis(p, a, b, c, nat);
    if (o == 3) return E::quad_l(p, a, b);
    if (o == 2) return E::quad_r(a, b, c);
    if (o == 1) return E::lin(a, b);
    return a;
  }
  // line_at (MD) along an axis given by its neighbour offsets, every order
  __device__ __forceinline__ T line_rt(const T* w, const Nb& n, int o) const {
    using E = Expr<T>;
    const T t1 = w[n.m1];
    if (o == 0) return t1;
    const T t2 = w[n.p1];
    if (o == 4) return E::cubic_lambda(w[n.m3], t1, t2, w[n.p3], nat);
    if (o == 3) return E::quad_l(w[n.m3], t1, t2);
    if (o == 2) return E::quad_r(t1, t2, w[n.p3]);
    return E::lin(t1, t2);
  }
  // neighbour offsets along axis d of this level's points (odd coordinates
  // at level 0, even ones above)
  static __device__ __forceinline__ Nb nb(int d) { return U == 1 ? nb_odd<T>(d) : nb_even<T>(d, U); }
  // KIND 0 md lines, 2 per-axis lines, 1 md faces (J = the reference's a2,
  // K = a1, at odd coordinate ck: face_at's full case table).  Point j of a
  // job is at coordinate (2j+1)U along J; its line's even values at 2kU.
  // w0: the slot of the line's point at coordinate 0 along J.  The line's
  // even point k (coordinate 2kU) sits at w0 + k E2, its point j (coordinate
  // (2j+1)U) at w0 + j E2 + P0.
  template <int KIND>
  __device__ __forceinline__ void edge_job(int w0, int J, int K, int cw0, int cs, bool own, int j0, int j1,
                                           int ck) const {
    using E = Expr<T>;
    using F = Fp<T>;
    const int E2 = U * Win<T>::step2(J), P0 = U == 1 ? Win<T>::one(J) : (U / 2) * Win<T>::step2(J);
    const int l3 = lim3(J), l1 = lim1(J), r = lim_r(J);
    int ok = 0;
    Nb nk{0, 0, 0, 0}, nj{0, 0, 0, 0};
    if (KIND == 1) {
      nk = nb(K);
      nj = nb(J);
      ok = order_rt(ck, lim3(K), lim1(K));
    }
    T p = j0 > 0 ? win[w0 + (j0 - 1) * E2] : T(0);
    T a = win[w0 + j0 * E2], b = win[w0 + (j0 + 1) * E2];
    T c = j0 + 2 <= N ? win[w0 + (j0 + 2) * E2] : T(0);
#pragma unroll 1
    for (int j = j0; j < j1 && (2 * j + 1) * U < r; ++j) {
      const int wi = w0 + j * E2 + P0;
      const int oj = order_rt((2 * j + 1) * U, l3, l1);
      const T lj = window_line<KIND != 2>(oj, p, a, b, c);
      T pred = lj;
      if (KIND == 1) {
        if (ok == 4 || oj == 4) {
          if (ok != 4) pred = lj;
          else if (oj != 4) pred = line_rt(win + wi, nk, ok);
          else pred = E::half(F::add(line_rt(win + wi, nk, ok), lj));
        } else if ((ok >= 2 && oj >= 2) || (ok == 1 && oj == 1)) {
          pred = E::half(F::add(line_rt(win + wi, nk, ok), lj));
        } else if (ok >= 2 || (ok == 1 && oj == 0)) {
          pred = line_rt(win + wi, nk, ok);
        } else if (oj >= 1) {
          pred = lj;
        } else {
          pred = F::sub(F::add(win[wi + nk.m1], win[wi + nj.m1]), win[wi + nk.m1 + nj.m1]);
        }
      }
      emit_at(wi, cw0 + (2 * j + 1) * U * cs, own, pred);
      p = a;
      a = b;
      b = c;
      if (j + 3 <= N) c = win[w0 + (j + 3) * E2];
    }
  }
  // md cube points (x odd, cy, cz) along x with cube_at's full case order
  __device__ __forceinline__ void edge_cube_job(int cy, int cz, int j0, int j1) const {
    using E = Expr<T>;
    using F = Fp<T>;
    constexpr int SX = U;  // x is not skewed
    const int w0 = Win<T>::at(0, cy, cz), cw0 = (cz * 16 + cy) * 16;
    const Nb ny = nb(1), nz = nb(2);
    const int oy = order_rt(cy, lim3(1), lim1(1)), oz = order_rt(cz, lim3(2), lim1(2));
    const int l3 = lim3(0), l1 = lim1(0), r = lim_r(0);
    T p = j0 > 0 ? win[w0 + 2 * (j0 - 1) * SX] : T(0);
    T a = win[w0 + 2 * j0 * SX], b = win[w0 + 2 * (j0 + 1) * SX];
    T c = j0 + 2 <= N ? win[w0 + 2 * (j0 + 2) * SX] : T(0);
#pragma unroll 1
    for (int j = j0; j < j1 && (2 * j + 1) * U < r; ++j) {
      const int wi = w0 + (2 * j + 1) * SX;
      const T* w = win + wi;
      const int ox = order_rt((2 * j + 1) * U, l3, l1);
      auto cy_ = [&]() { return E::cubic_lambda(w[ny.m3], w[ny.m1], w[ny.p1], w[ny.p3], nat); };
      auto cz_ = [&]() { return E::cubic_lambda(w[nz.m3], w[nz.m1], w[nz.p1], w[nz.p3], nat); };
      auto cx_ = [&]() { return E::cubic_lambda(p, a, b, c, nat); };
      T pred;
      if (oz == 4 && oy == 4 && ox == 4) pred = F::div(F::add(F::add(cx_(), cy_()), cz_()), T(3));
      else if (oz == 4 && oy == 4) pred = E::half(F::add(cz_(), cy_()));
      else if (oz == 4 && ox == 4) pred = E::half(F::add(cz_(), cx_()));
      else if (oy == 4 && ox == 4) pred = E::half(F::add(cy_(), cx_()));
      else if (oz == 4) pred = cz_();
      else if (oy == 4) pred = cy_();
      else if (ox == 4) pred = cx_();
      else if (ox == 3) pred = E::quad_l(p, a, b);
      else if (ox == 2) pred = E::quad_r_cube(a, b, c);
      else if (ox == 1) pred = E::lin(a, b);
      else pred = a;
      emit_at(wi, cw0 + (2 * j + 1) * U, true, pred);
      p = a;
      a = b;
      b = c;
      if (j + 3 <= N) c = win[w0 + 2 * (j + 3) * SX];
    }
  }
  // slot of the window point with coordinate ca on axis a, cb on axis b and
  // 0 on the third
  static __device__ __forceinline__ int at2(int a, int ca, int b, int cb) {
    return Win<T>::axis(a, ca) + Win<T>::axis(b, cb);
  }
  // Level 1 (unit 2, four odd points per line) of any tile by half-line jobs
  // with the runtime orders; not the last level, so every point in the field
  // is predicted.  md: 150 line, 120 face and 32 cube jobs; per axis: 50,
  // 90 and 162 jobs.
  __device__ __forceinline__ void mid_md_jobs() const {
    static_assert(U == 2, "level 1");
    const int t = threadIdx.x;
    auto kC = [](int a) { return a == 0 ? 1 : (a == 1 ? 16 : 256); };
    if (t < 150) {
      const int h = t / 75, r = t - 75 * h, f = r / 25, l = r - 25 * f, u = 4 * (l % 5), v = 4 * (l / 5);
      const int P = f == 0 ? 1 : 0, Q = f == 2 ? 1 : 2;
      if (u < lim_r(P) && v < lim_r(Q))
        edge_job<0>(at2(P, u, Q, v), f, 0, u * kC(P) + v * kC(Q), kC(f), (u | v) < 16, 2 * h, 2 * h + 2, 0);
    }
    __syncthreads();
    if (t < 120) {
      const int h = t / 60, r = t - 60 * h, f = r / 20, l = r - 20 * f, ce = 4 * (l % 5), ck = 4 * (l / 5) + 2;
      const int J = f == 0 ? 1 : 0, K = f == 1 ? 2 : (f == 0 ? 2 : 1);
      if (ce < lim_r(f) && ck < lim_r(K))
        edge_job<1>(at2(f, ce, K, ck), J, K, ce * kC(f) + ck * kC(K), kC(J), ce < 16, 2 * h, 2 * h + 2, ck);
    }
    __syncthreads();
    if (t < 32) {
      const int line = t >> 1, h = t & 1, cy = 4 * (line & 3) + 2, cz = 4 * (line >> 2) + 2;
      if (cy < lim_r(1) && cz < lim_r(2)) edge_cube_job(cy, cz, 2 * h, 2 * h + 2);
    }
    __syncthreads();
  }
  __device__ __forceinline__ void mid_axis_jobs(bool rev) const {
    static_assert(U == 2, "level 1");
    using W = Win<T>;
    const int t = threadIdx.x;
    const int r0 = lim_r(0), r1 = lim_r(1), r2 = lim_r(2);
    if (!rev) {  // z at (x, y) even; y at (x even, z any); x at (y, z any)
      if (t < 50) {
        const int h = t / 25, l = t - 25 * h, x = 4 * (l % 5), y = 4 * (l / 5);
        if (x < r0 && y < r1) edge_job<2>(W::at(x, y, 0), 2, 0, x + 16 * y, 256, (x | y) < 16, 2 * h, 2 * h + 2, 0);
      }
      __syncthreads();
      if (t < 90) {
        const int h = t / 45, l = t - 45 * h, x = 4 * (l % 5), z = 2 * (l / 5);
        if (x < r0 && z < r2) edge_job<2>(W::at(x, 0, z), 1, 0, x + 256 * z, 16, (x | z) < 16, 2 * h, 2 * h + 2, 0);
      }
      __syncthreads();
      if (t < 162) {
        const int h = t / 81, l = t - 81 * h, y = 2 * (l % 9), z = 2 * (l / 9);
        if (y < r1 && z < r2) edge_job<2>(W::at(0, y, z), 0, 0, 16 * y + 256 * z, 1, (y | z) < 16, 2 * h, 2 * h + 2, 0);
      }
    } else {  // x at (y, z) even; y at (x any, z even); z at (x, y any)
      if (t < 50) {
        const int h = t / 25, l = t - 25 * h, y = 4 * (l % 5), z = 4 * (l / 5);
        if (y < r1 && z < r2) edge_job<2>(W::at(0, y, z), 0, 0, 16 * y + 256 * z, 1, (y | z) < 16, 2 * h, 2 * h + 2, 0);
      }
      __syncthreads();
      if (t < 90) {
        const int h = t / 45, l = t - 45 * h, x = 2 * (l % 9), z = 4 * (l / 9);
        if (x < r0 && z < r2) edge_job<2>(W::at(x, 0, z), 1, 0, x + 256 * z, 16, (x | z) < 16, 2 * h, 2 * h + 2, 0);
      }
      __syncthreads();
      if (t < 162) {
        const int h = t / 81, l = t - 81 * h, x = 2 * (l % 9), y = 2 * (l / 9);
        if (x < r0 && y < r1) edge_job<2>(W::at(x, y, 0), 2, 0, x + 16 * y, 256, (x | y) < 16, 2 * h, 2 * h + 2, 0);
      }
    }
    __syncthreads();
  }
  __device__ __forceinline__ void edge_md_lines() const {
    const int t = threadIdx.x;
    auto kC = [](int a) { return a == 0 ? 1 : (a == 1 ? 16 : 256); };
    if (t < 243) {
      const int f = t / 81, l = t - 81 * f, u = 2 * (l % 9), v = 2 * (l / 9);
      const int P = f == 0 ? 1 : 0, Q = f == 2 ? 1 : 2;
      if (u < lim_r(P) && v < lim_r(Q))
        edge_job<0>(at2(P, u, Q, v), f, 0, u * kC(P) + v * kC(Q), kC(f), (u | v) < 16, 0, 8, 0);
    }
    __syncthreads();
    if (t < 216) {
      const int f = t / 72, l = t - 72 * f, ce = 2 * (l % 9), ck = 2 * (l / 9) + 1;
      const int J = f == 0 ? 1 : 0, K = f == 1 ? 2 : (f == 0 ? 2 : 1);
      if (ce < lim_r(f) && ck < lim_r(K))
        edge_job<1>(at2(f, ce, K, ck), J, K, ce * kC(f) + ck * kC(K), kC(J), ce < 16, 0, 8, ck);
    }
    __syncthreads();
    {
      const int line = t >> 2, q = t & 3, cy = 2 * (line & 7) + 1, cz = 2 * (line >> 3) + 1;
      if (cy < lim_r(1) && cz < lim_r(2)) edge_cube_job(cy, cz, 2 * q, 2 * q + 2);
    }
    __syncthreads();
  }
  __device__ __forceinline__ void edge_axis_lines(bool rev) const {
    using W = Win<T>;
    const int t = threadIdx.x;
    const int r0 = lim_r(0), r1 = lim_r(1), r2 = lim_r(2);
    if (!rev) {  // z, then y, then x
      if (t < 162) {
        const int l = t >> 1, x = 2 * (l % 9), y = 2 * (l / 9), j0 = (t & 1) * 4;
        if (x < r0 && y < r1) edge_job<2>(W::at(x, y, 0), 2, 0, x + 16 * y, 256, (x | y) < 16, j0, j0 + 4, 0);
      }
      __syncthreads();
      if (t < 144) {
        const int x = 2 * (t % 9), z = t / 9;
        if (x < r0 && z < r2) edge_job<2>(W::at(x, 0, z), 1, 0, x + 256 * z, 16, x < 16, 0, 8, 0);
      }
      __syncthreads();
      const int y = t & 15, z = t >> 4;
      if (y < r1 && z < r2) edge_job<2>(W::at(0, y, z), 0, 0, 16 * y + 256 * z, 1, true, 0, 8, 0);
    } else {  // x, then y, then z
      if (t < 162) {
        const int l = t >> 1, y = 2 * (l % 9), z = 2 * (l / 9), j0 = (t & 1) * 4;
        if (y < r1 && z < r2) edge_job<2>(W::at(0, y, z), 0, 0, 16 * y + 256 * z, 1, (y | z) < 16, j0, j0 + 4, 0);
      }
      __syncthreads();
      if (t < 144) {
        const int x = t & 15, z = 2 * (t >> 4);
        if (x < r0 && z < r2) edge_job<2>(W::at(x, 0, z), 1, 0, x + 256 * z, 16, z < 16, 0, 8, 0);
      }
      __syncthreads();
      const int x = t & 15, y = t >> 4;
      if (x < r0 && y < r1) edge_job<2>(W::at(x, y, 0), 2, 0, x + 16 * y, 256, true, 0, 8, 0);
    }
    __syncthreads();
  }
  // Stage-to-lane maps of the interior md level 0, chosen with the window
  // layout (Win) to spread each warp's accesses over the banks: a face
  // family whose bit is set in kFaceSwap takes its jobs with the odd
  // coordinate fastest; the cube's quarter-line jobs go line-fastest, with y
  // (double) or z (float) fastest across the lines.
  static constexpr int kFaceSwap = sizeof(T) == 8 ? 6 : 4;
  // md level 0: lines (243 jobs), faces (216 jobs), cube (256 quarter-line
  // jobs), one barrier per stage
  __device__ __forceinline__ void level0_md_lines() const {
    static_assert(kPredThreads == 256, "one cube quarter-line per thread");
    const int t = threadIdx.x;
    auto kC = [](int a) { return a == 0 ? 1 : (a == 1 ? 16 : 256); };  // code-block stride
    if (t < 243) {
      // family f: lines along axis f through the other two (even) coordinates
      const int f = t / 81, l = t - 81 * f, u = 2 * (l % 9), v = 2 * (l / 9);
      const int P = f == 0 ? 1 : 0, Q = f == 2 ? 1 : 2;  // the fixed axes
      md_job<0>(at2(P, u, Q, v), f, u * kC(P) + v * kC(Q), kC(f), (u | v) < 16, 0, 8, 0, 0);
    }
    __syncthreads();
    if (t < 216) {
      // family f: the even axis EA = f; jobs along J, second odd axis K
      const int f = t / 72, l = t - 72 * f;
      const bool swap = (kFaceSwap >> f) & 1;
      const int ce = swap ? 2 * (l >> 3) : 2 * (l % 9), ck = swap ? 2 * (l & 7) + 1 : 2 * (l / 9) + 1;
      const int J = f == 0 ? 1 : 0, K = f == 1 ? 2 : (f == 0 ? 2 : 1);
      md_job<1>(at2(f, ce, K, ck), J, ce * kC(f) + ck * kC(K), kC(J), ce < 16, 0, 8, K, order0(ck));
    }
    __syncthreads();
    {
      const int line = t & 63, q = t >> 6;
      const int a = 2 * (line & 7) + 1, b = 2 * (line >> 3) + 1;
      if (sizeof(T) == 8) md_cube_job(b, a, 2 * q);
      else md_cube_job(a, b, 2 * q);
    }
    __syncthreads();
  }
  // Per-axis level 0 of an interior tile by jobs (md_job<2>).  Points that no
  // later prediction reads and whose codes belong to a neighbouring tile
  // (the last stage's lines at coordinate 16, the middle stage's lines in
  // the last stage's plane 16) are skipped: their values and codes would be
  // dropped.  First stage: 81 lines as 162 half-line jobs; middle stage: 144
  // lines; last stage: the tile's 256 lines, one per thread.
  __device__ __forceinline__ void level0_lines(bool rev) const {
    static_assert(kPredThreads == 256, "one last-stage line per thread");
    using W = Win<T>;
    const int t = threadIdx.x;
    if (!rev) {  // z, then y, then x
      if (t < 162) {
        const int l = t >> 1, x = 2 * (l % 9), y = 2 * (l / 9), j0 = (t & 1) * 4;
        md_job<2>(W::at(x, y, 0), 2, x + 16 * y, 256, (x | y) < 16, j0, j0 + 4, 0, 0);
      }
      __syncthreads();
      if (t < 144) {
        const int x = 2 * (t % 9), z = t / 9;
        md_job<2>(W::at(x, 0, z), 1, x + 256 * z, 16, x < 16, 0, 8, 0, 0);
      }
      __syncthreads();
      const int y = t & 15, z = t >> 4;
      md_job<2>(W::at(0, y, z), 0, 16 * y + 256 * z, 1, true, 0, 8, 0, 0);
    } else {  // x, then y, then z
      if (t < 162) {
        const int l = t >> 1, y = 2 * (l % 9), z = 2 * (l / 9), j0 = (t & 1) * 4;
        md_job<2>(W::at(0, y, z), 0, 16 * y + 256 * z, 1, (y | z) < 16, j0, j0 + 4, 0, 0);
      }
      __syncthreads();
      if (t < 144) {
        const int x = t & 15, z = 2 * (t >> 4);
        md_job<2>(W::at(x, 0, z), 1, x + 256 * z, 16, z < 16, 0, 8, 0, 0);
      }
      __syncthreads();
      const int x = t & 15, y = t >> 4;
      md_job<2>(W::at(x, y, 0), 2, x + 16 * y, 256, true, 0, 8, 0, 0);
    }
    __syncthreads();
  }
  // the three stages of the level (spline_layout_interpolate :1771-2027)
  __device__ __forceinline__ void run(bool md, bool rev) const {
    constexpr bool kLast = U == 1;
    // axis codes: x = 0, y = 1, z = 2; AXES = a0 | a1 << 2 | a2 << 4
    if constexpr (U == 2) {
      if (md) mid_md_jobs();
      else mid_axis_jobs(rev);
      return;
    }
    if constexpr (U == 1) {
      if constexpr (EDGE) {
        if (md) edge_md_lines();
        else edge_axis_lines(rev);
      } else {
        if (md) level0_md_lines();
        else level0_lines(rev);
      }
      return;
    } else {
    if (md) {
      // lines (xyzmap_line): x-lines vary y fastest, y- and z-lines vary x.
      // Points of one stage only read coarser points, so the three groups
      // share one barrier.
      sweep<0, true, 1 | (2 << 2) | (0 << 4), N + 1, 2, 0, N + 1, 2, 0, N, 2, 1, false>(false);
      sweep<1, true, 0 | (2 << 2) | (1 << 4), N + 1, 2, 0, N + 1, 2, 0, N, 2, 1, false>(false);
      sweep<2, true, 0 | (1 << 2) | (2 << 4), N + 1, 2, 0, N + 1, 2, 0, N, 2, 1>(false);
      // faces (xyzmap_face): x even -> z,y; y even -> z,x; z even -> y,x
      faces<0, 2, 1, false>();
      faces<1, 2, 0, false>();
      faces<2, 1, 0>();
      cube(kLast);
    } else if (rev) {
      // x: (x odd, y even, z even), vary y fastest
      sweep<0, false, 1 | (0 << 2) | (2 << 4), N + 1, 2, 0, N, 2, 1, N + 1, 2, 0>(false);
      // y: (x any, y odd, z even), vary x
      sweep<1, false, 0 | (1 << 2) | (2 << 4), 2 * N + 1, 1, 0, N, 2, 1, N + 1, 2, 0>(false);
      // z: (x any, y any, z odd), vary x
      sweep<2, false, 0 | (1 << 2) | (2 << 4), 2 * N + 1, 1, 0, 2 * N + 1, 1, 0, N, 2, 1>(kLast);
    } else {
      // z: (x even, y even, z odd), vary x
      sweep<2, false, 0 | (1 << 2) | (2 << 4), N + 1, 2, 0, N + 1, 2, 0, N, 2, 1>(false);
      // y: (x even, y odd, z any), vary x
      sweep<1, false, 0 | (1 << 2) | (2 << 4), N + 1, 2, 0, N, 2, 1, 2 * N + 1, 1, 0>(false);
      // x: (x odd, y any, z any), vary y
      sweep<0, false, 1 | (0 << 2) | (2 << 4), 2 * N + 1, 1, 0, N, 2, 1, 2 * N + 1, 1, 0>(kLast);
    }
    }
  }
};

template <class T, bool COMPRESS, bool EDGE, int U, int LEVEL>
__device__ __forceinline__ void sweep_level(T* win, int32_t* cw, const AxisLimits& lim, bool zlast,
                                            const PredParams<T>& p) {
  if (LEVEL > p.maxlevel || (LevelSweep<T, COMPRESS, U, EDGE>::kWarp && threadIdx.x >= 32)) return;
  LevelSweep<T, COMPRESS, U, EDGE> lv{win, cw, Limits<EDGE>{lim}, zlast, p.ebr[LEVEL], p.ebx2[LEVEL]};
  lv.run(p.use_md[LEVEL] != 0, p.reverse[LEVEL] != 0);
}

// spline_layout_interpolate (:1771-2027): levels 3..0
// in two parts: levels 3..1 only touch the 9^3 window points whose
// coordinates are all even, level 0 the rest as well
template <class T, bool COMPRESS, bool EDGE>
__device__ void sweep_coarse(T* win, int32_t* cw, const AxisLimits& lim, bool zlast, const PredParams<T>& p) {
  sweep_level<T, COMPRESS, EDGE, 8, 3>(win, cw, lim, zlast, p);
  sweep_level<T, COMPRESS, EDGE, 4, 2>(win, cw, lim, zlast, p);
  if (COMPRESS) __syncthreads();
  sweep_level<T, COMPRESS, EDGE, 2, 1>(win, cw, lim, zlast, p);
}
template <class T, bool COMPRESS, bool EDGE>
__device__ void sweep_fine(T* win, int32_t* cw, const AxisLimits& lim, bool zlast, const PredParams<T>& p) {
  sweep_level<T, COMPRESS, EDGE, 1, 0>(win, cw, lim, zlast, p);
}

// window slot of the j-th of the 9^3 points with all coordinates even
template <class T>
__device__ __forceinline__ int even_point(int j, int& x, int& y, int& z) {
  x = 2 * (j % 9);
  y = 2 * ((j / 9) % 9);
  z = 2 * (j / 81);
  return Win<T>::at(x, y, z);
}

// ---- tiles -------------------------------------------------------------------

// Tiles are launched in two parts so that each kernel runs one code path:
// part 0 = interior tiles ((ax-1)(ay-1)(az-1) of them), part 1 = the tiles
// on the last slab along z, then y, then x.
PRISM_HD uint64_t tiles_in_part(const Geometry& g, int part) {
  uint64_t inner = (uint64_t)(g.ax - 1) * (g.ay - 1) * (g.az - 1);
  return part == 0 ? inner : (uint64_t)g.ax * g.ay * g.az - inner;
}

template <int PART, class G = Geometry>
__device__ __forceinline__ void tile_of_index(const G& g, uint32_t j, uint32_t bi[3]) {
  if (PART == 0) {
    bi[0] = j % (g.ax - 1); bi[1] = (j / (g.ax - 1)) % (g.ay - 1); bi[2] = j / ((g.ax - 1) * (g.ay - 1));
    return;
  }
  if (j < g.ax * g.ay) { bi[0] = j % g.ax; bi[1] = j / g.ax; bi[2] = g.az - 1; return; }
  j -= g.ax * g.ay;
  if (j < g.ax * (g.az - 1)) { bi[0] = j % g.ax; bi[1] = g.ay - 1; bi[2] = j / g.ax; return; }
  j -= g.ax * (g.az - 1);
  bi[0] = g.ax - 1; bi[1] = j % (g.ay - 1); bi[2] = j / (g.ay - 1);
}

template <int PART>
__device__ __forceinline__ void tile_of_block(const Geometry& g, uint32_t bi[3]) {
  tile_of_index<PART>(g, blockIdx.x, bi);
}

// Per-tile frame: window origin, limits, and the level-0 slot of each window
// row (y, z) at x = 0 (level-major order, :2070-2085), which makes the slot of
// a level-0 point one add.
struct TileFrame {
  uint32_t gs[3];
  bool last[3];
  AxisLimits lim;
};

template <class G>
__device__ __forceinline__ void tile_frame(const G& g, const uint32_t bi[3], TileFrame& f) {
  const uint32_t gd[3] = {g.ax, g.ay, g.az}, dim[3] = {g.nx, g.ny, g.nz};
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    f.gs[d] = bi[d] * 16u;
    f.last[d] = bi[d] == gd[d] - 1;
    int r = (int)min(dim[d] - f.gs[d], 17u);
    f.lim.r[d] = f.last[d] ? r : kWin;
    f.lim.l3[d] = f.last[d] ? min(16, r - 1) : 16;
    f.lim.l1[d] = f.last[d] ? r - 1 : 1 << 20;
  }
}


// level of a window point: 0..3, or 4 for the stride-16 anchors (the window
// starts on a multiple of 16, so window and global coordinates agree mod 16)
__device__ __forceinline__ int win_level(int x, int y, int z) { return __ffs(x | y | z | 16) - 1; }

// Level-major slot of a point whose level (0..3) is known (the formula of
// level_major_index without its level search).
template <class G>
__device__ __forceinline__ uint64_t lm_slot(const G& g, int level, uint64_t gx, uint64_t gy, uint64_t gz) {
  gx >>= level; gy >>= level; gz >>= level;
  uint64_t gid = gx + gy * g.leaps[level][0] + gz * g.leaps[level][1];
  gid += g.lm_prefix[level] - ((gz + 1) >> 1) * g.leaps[level + 1][1] -
         (uint64_t)((gz & 1) == 0) * ((gy + 1) >> 1) * g.leaps[level + 1][0] -
         (uint64_t)(((gz | gy) & 1) == 0) * ((gx + 1) >> 1);
  return gid;
}

// Row table of a tile: for each level l and each window row (y, z) whose
// coordinates are multiples of 2^l, the level-major slot of the row's level-l
// point at x = 0 (lm_slot with gx = gs[0]).  Along a row the level-l points
// are consecutive slots: writing x' = x >> l, a point's slot is
// rows[row] + x' when (y >> l) or (z >> l) is odd, else rows[row] + x' / 2
// (x' is then odd; gs[0] >> l is even, which makes the x part split off).
// Level l has (16 >> l) + 1 window coordinates per axis: 17^2 + 9^2 + 5^2 +
// 3^2 = 404 rows.
constexpr int kRowTable = 404;

__device__ __forceinline__ int row_of(int l, int y, int z) {
  const int w = (16 >> l) + 1;
  const int off = l == 0 ? 0 : (l == 1 ? 289 : (l == 2 ? 370 : 395));
  return off + (z >> l) * w + (y >> l);
}

template <bool NARROW, class G>
__device__ __forceinline__ void fill_rows(const G& g, const TileFrame& f, uint64_t* rows) {
  // NARROW: in 32 bits where the slots allow it (rows past the field may wrap
  // and are not used): 2% of the predictor's time, nothing in the
  // reconstruction, which fills the table while other tiles' loads are waited
  // for
  const bool small = NARROW && g.n + 64 * (uint64_t)g.anchors < (1ull << 31);
  for (int r = threadIdx.x; r < kRowTable; r += kPredThreads) {
    const int l = r < 289 ? 0 : (r < 370 ? 1 : (r < 395 ? 2 : 3));
    const int w = (16 >> l) + 1, k = r - (l == 0 ? 0 : (l == 1 ? 289 : (l == 2 ? 370 : 395)));
    const int y = (k % w) << l, z = (k / w) << l;
    if (small) {  // every product and sum fits
      const uint32_t gx = f.gs[0] >> l, gy = (f.gs[1] + y) >> l, gz = (f.gs[2] + z) >> l;
      const uint32_t a0 = (uint32_t)g.leaps[l][0], a1 = (uint32_t)g.leaps[l][1];
      const uint32_t b0 = (uint32_t)g.leaps[l + 1][0], b1 = (uint32_t)g.leaps[l + 1][1];
      uint32_t s = (uint32_t)g.lm_prefix[l] + gx + gy * a0 + gz * a1 - ((gz + 1) >> 1) * b1;
      if (!(gz & 1)) s -= ((gy + 1) >> 1) * b0;
      if (!((gz | gy) & 1)) s -= (gx + 1) >> 1;
      rows[r] = s;
    } else {
      rows[r] = lm_slot(g, l, (uint64_t)f.gs[0], (uint64_t)f.gs[1] + y, (uint64_t)f.gs[2] + z);
    }
  }
}

// Slot of window point (x, y, z) of level lv (0..3) from the row table.
__device__ __forceinline__ uint64_t slot_of(const uint64_t* rows, int lv, int x, int y, int z) {
  const int ee = (((y | z) >> lv) & 1) == 0;
  return rows[row_of(lv, y, z)] + (uint64_t)((x >> lv) >> ee);
}

// Shared memory of a compression tile: the value window and the codes of the
// tile's own points (~56 KB for double, so four tiles fit an SM; ~36 KB for
// float, six).  The row table takes the window's place once the sweeps are
// done.
template <class T>
struct CompressSmem {
  T win[Win<T>::kSize];  // after the sweeps: the row table
  int32_t cw[16 * 16 * 16];  // codes of the tile's own points (cw_word order)
  PredParams<T> p;
};
static_assert(sizeof(float) * Win<float>::kSize >= sizeof(uint64_t) * kRowTable, "row table fits the window");

template <class T> struct PairOf;
template <> struct PairOf<double> { using type = double2; };
template <> struct PairOf<float> { using type = float2; };

// Shared memory of a reconstruction tile: the window (codes travel in the
// window slots) and the row table (~44 KB for double, ~24 KB for float).
template <class T>
struct ReconSmem {
  T win[Win<T>::kSize];
  uint64_t rows[kRowTable];
  PredParams<T> p;
};

// Compression: data -> anchors + level-major codes (interpolation :2137-2173).
// The window is loaded with asynchronous copies, all in flight at once,
// the 12 stages run in shared memory, and the codes of the points the tile
// owns leave in one pass at the end.
// One tile of the compression (the body of predict_compress_kernel and of the
// batched persistent kernel).  The caller guarantees that no thread still
// reads `sm` from a previous tile.
template <class T, bool EDGE, class G = Geometry>
__device__ __forceinline__ void compress_tile(CompressSmem<T>& sm, const T* __restrict__ data, const G& g,
                                              const uint32_t bi[3], const PredParams<T>* pp, T* __restrict__ anchors,
                                              int32_t* __restrict__ qc) {
  TileFrame f;
  tile_frame(g, bi, f);
  const Limits<EDGE> L{f.lim};
  const int tid = threadIdx.x;
  if (tid == 0) sm.p = *pp;
  const uint64_t sy = g.nx, sz = (uint64_t)g.nx * g.ny;
  const T* base = data + (uint64_t)f.gs[0] + (uint64_t)f.gs[1] * sy + (uint64_t)f.gs[2] * sz;
  // two copy groups: the points levels 3..1 use, then the rest, which
  // arrive while those levels run
  for (int j = tid; j < 729; j += kPredThreads) {
    int x, y, z;
    const int i = even_point<T>(j, x, y, z);
    if (L.in_data(x, y, z)) copy_async<sizeof(T)>(&sm.win[i], base + x + (uint64_t)y * sy + (uint64_t)z * sz);
    else sm.win[i] = T(0);
  }
  copy_async_commit();
  // the rest by window rows r = 17 z + y: a half-warp takes x = 0..15 of a
  // row (rows advance by 16), then a thread per row takes x = 16
  {
    static_assert(2 * (kPredThreads / 32) == 16, "rows advance by 16: (y, z) -> (y - 1, z + 1) or (16, z)");
    const int lane = tid & 31, x = lane & 15;
    int r = (tid >> 5) * 2 + (lane >> 4), y = r, z = 0;
    const T* src = base + x + (uint64_t)y * sy;
    for (; r < kWin * kWin; r += 16) {
      if (((x | y | z) & 1) != 0) {
        T* dst = &sm.win[Win<T>::at(x, y, z)];
        if (L.in_data(x, y, z)) copy_async<sizeof(T)>(dst, src);
        else *dst = T(0);
      }
      if (y == 0) {
        y = 16;
        src += 16 * sy;
      } else {
        --y;
        ++z;
        src += sz - sy;
      }
    }
    for (int q = tid; q < kWin * kWin; q += kPredThreads) {
      const int yq = q % kWin, zq = q / kWin;
      if (((yq | zq) & 1) == 0) continue;  // (16, even, even): an even point
      T* dst = &sm.win[Win<T>::at(16, yq, zq)];
      if (L.in_data(16, yq, zq)) copy_async<sizeof(T)>(dst, base + 16 + (uint64_t)yq * sy + (uint64_t)zq * sz);
      else *dst = T(0);
    }
  }
  copy_async_commit();
  copy_async_wait_group<1>();
  __syncthreads();
  if (tid == 0) anchors[bi[0] + (uint64_t)bi[1] * g.ax + (uint64_t)bi[2] * g.ax * g.ay] = sm.win[0];
  sweep_coarse<T, true, EDGE>(sm.win, sm.cw, f.lim, f.last[2], sm.p);
  copy_async_wait_group<0>();
  __syncthreads();
  sweep_fine<T, true, EDGE>(sm.win, sm.cw, f.lim, f.last[2], sm.p);
  // Every non-anchor point of the tile's own 16^3 that lies in the field was
  // emitted (on a last tile the plane at 16 lies outside the field).
  __syncthreads();
  uint64_t* rows = reinterpret_cast<uint64_t*>(sm.win);
  fill_rows<true>(g, f, rows);
  __syncthreads();
  // Thread t takes point (t mod 16, t / 16) of each z-plane: on an odd plane
  // (and an odd row) the row is all level 0 (slot rows[r] + x), on the others
  // the odd x are (rows[r] + x / 2); only the even x of those go through the
  // level lookup.
  static_assert(kPredThreads == 256, "a z-plane per pass");
  const int x = tid & 15, y = tid >> 4;
  if (!L.in_data(x, y, 0)) return;
  const int zs = EDGE ? (f.lim.r[2] < 16 ? f.lim.r[2] : 16) : 16;
  const bool odd_row = y & 1;
#pragma unroll 4
  for (int z = 0; z < zs; z += 2) {
    uint64_t slot;
    if (odd_row || (x & 1)) {
      slot = rows[z * kWin + y] + (uint64_t)(odd_row ? x : x >> 1);
      qc[slot] = sm.cw[cw_word(256 * z + tid)];
    } else {
      const int lv = win_level(x, y, z);
      if (lv < 4) qc[slot_of(rows, lv, x, y, z)] = sm.cw[cw_word(256 * z + tid)];
    }
    if (!EDGE || z + 1 < zs) qc[rows[(z + 1) * kWin + y] + (uint64_t)x] = sm.cw[cw_word(256 * (z + 1) + tid)];
  }
}

// CTAs per SM the compiler must leave room for: a float tile's shared memory
// (window + codes, 36 KB) admits six on an SM when its registers do, a double
// one (55 KB) four.  For float last-slab tiles six (40 registers, a few
// spilled) measured 7-9% faster than four (55 registers).
template <class T, int PART>
constexpr int predict_min_ctas() { return sizeof(T) == 4 ? 6 : 4; }

template <class T, int PART>
__global__ void __launch_bounds__(kPredThreads, predict_min_ctas<T, PART>())
predict_compress_kernel(const T* __restrict__ data, Geometry g, const PredParams<T>* __restrict__ pp,
                        T* __restrict__ anchors, int32_t* __restrict__ qc) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  CompressSmem<T>& sm = *reinterpret_cast<CompressSmem<T>*>(smem_raw);
  uint32_t bi[3];
  tile_of_block<PART>(g, bi);
  compress_tile<T, PART == 1>(sm, data, g, bi, pp, anchors, qc);
}

// Both parts in one launch, the (longer) last-slab tiles first: for fields
// whose tiles are all on the GPU at once, where a second stream's events cost
// more than the wider register budget of the joined kernel: the two parts of
// a 64x48x40 float field (12 and 16 us) took 19 us from the first start to the
// last end and two gaps of 8 us around them.  A whole compression with two
// launches and with one, just below the limit (592 tiles, 64x64x592): float 124
// -> 113 us, double 120 -> 114.  Above it, one launch would still take 1-8 us
// less up to 2048 tiles and as much at 2304.
template <class T>
__global__ void __launch_bounds__(kPredThreads, 4)
predict_compress_both_kernel(const T* __restrict__ data, Geometry g, const PredParams<T>* pp,
                             T* __restrict__ anchors, int32_t* __restrict__ qc) {
  chain_wait();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  CompressSmem<T>& sm = *reinterpret_cast<CompressSmem<T>*>(smem_raw);
  const uint32_t edge = (uint32_t)tiles_in_part(g, 1);
  uint32_t bi[3];
  if (blockIdx.x < edge) {
    tile_of_index<1>(g, blockIdx.x, bi);
    compress_tile<T, true>(sm, data, g, bi, pp, anchors, qc);
  } else {
    tile_of_index<0>(g, blockIdx.x - edge, bi);
    compress_tile<T, false>(sm, data, g, bi, pp, anchors, qc);
  }
}

// Reconstruction: anchors + codes -> values (interpolation_reverse
// :2177-2207); PROG adds the previous values (interpolation_progressive_reverse
// :2209-2239, shmem2global_data_progressive :1123-1147).  All codes the tile
// can use are fetched up front with asynchronous copies.
// a float interior tile's 23 KB of shared memory leaves room for seven
// CTAs on an SM when its registers do; a double one (43 KB) for five.  The
// last-slab tiles, with more live state, take six (float) and five (double):
// 2-3% faster than four at 64 registers, with a few registers spilled.
template <class T, int PART>
constexpr int reconstruct_min_ctas() { return PART == 0 ? (sizeof(T) == 4 ? 7 : 5) : (sizeof(T) == 4 ? 6 : 5); }


// The level-0 codes of an interior tile from a 16-byte aligned code buffer:
// a row's codes lie in at most five aligned 16-byte chunks (offset o =
// rows[r] mod 4 plus 17 codes, or 8 on a row with y and z even), and chunk s
// of the tile is chunk s mod 5 of row s / 5.  A thread's loads are in flight
// three at a time before their stores; the words a chunk holds beyond the
// row (neighbouring rows' codes, or the code buffer's slack past the last
// slot) are not stored.
template <class T>
__device__ __forceinline__ void fetch_level0_vec(ReconSmem<T>& sm, const int32_t* __restrict__ qc, int tid) {
  constexpr int kChunks = kWin * kWin * 5, kIt = (kChunks + kPredThreads - 1) / kPredThreads;
  constexpr int kBatch = (kIt + 1) / 2;
#pragma unroll
  for (int k0 = 0; k0 < kIt; k0 += kBatch) {
    int4 v[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
      const int s = tid + (k0 + k) * kPredThreads, r = s / 5, c = s - 5 * r;
      v[k] = make_int4(0, 0, 0, 0);
      if (k0 + k < kIt && s < kChunks) {
        const int y = r % kWin, z = r / kWin, n = ((y | z) & 1) ? kWin : 8;
        const uint64_t first = sm.rows[r];
        const int o = (int)(first & 3);
        if (4 * c < o + n) v[k] = __ldg(reinterpret_cast<const int4*>(qc + (first - o)) + c);
      }
    }
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
      const int s = tid + (k0 + k) * kPredThreads, r = s / 5, c = s - 5 * r;
      if (k0 + k >= kIt || s >= kChunks) continue;
      const int y = r % kWin, z = r / kWin, ee = ((y | z) & 1) == 0, n = ee ? 8 : kWin;
      const int o = (int)(sm.rows[r] & 3);
      const int32_t w[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int xi = 4 * c + i - o;
        if (xi >= 0 && xi < n) sm.win[Win<T>::at(ee ? 2 * xi + 1 : xi, y, z)] = Fp<T>::with_low_word(w[i]);
      }
    }
  }
}

template <class T, bool PROG, bool EDGE>
__device__ __forceinline__ void reconstruct_tile(ReconSmem<T>& sm, const int32_t* __restrict__ qc,
                                                 const T* __restrict__ anchors, const Geometry& g, const uint32_t bi[3],
                                                 const PredParams<T>* __restrict__ pp, const T* old, T* out) {
  TileFrame f;
  tile_frame(g, bi, f);
  const Limits<EDGE> L{f.lim};
  const int tid = threadIdx.x;
  const int maxlevel = pp->maxlevel;
  if (tid == 0) sm.p = *pp;
  fill_rows<false>(g, f, sm.rows);
  const uint64_t sy = g.nx, sz = (uint64_t)g.nx * g.ny;
  const uint64_t base = (uint64_t)f.gs[0] + (uint64_t)f.gs[1] * sy + (uint64_t)f.gs[2] * sz;
  if (PROG) {
    // the previous values are read after the sweeps: start bringing the
    // tile's rows (16 values, one or two 128-byte lines) into L2 now
    const int y = tid & 15, z = tid >> 4;
    if (L.in_data(0, y, z)) {
      const T* row = old + base + (uint64_t)y * sy + (uint64_t)z * sz;
      prefetch_l2(row);
      if (L.in_data(15, y, z)) prefetch_l2(row + 15);
    }
  }
  __syncthreads();
  // each code lands in the low word of its window slot (converted when its
  // point is predicted); every other slot reads as zero.  The codes of
  // levels 3..1 (points with all coordinates even) come first; the level-0
  // codes follow by one of the three ways below.
  for (int j = tid; j < 729; j += kPredThreads) {
    int x, y, z;
    const int i = even_point<T>(j, x, y, z);
    const int lv = win_level(x, y, z);
    int32_t* dst = reinterpret_cast<int32_t*>(&sm.win[i]);
    if (lv < 4 && lv <= maxlevel && L.in_data(x, y, z)) copy_async<4>(dst, qc + slot_of(sm.rows, lv, x, y, z));
    else sm.win[i] = T(0);
  }
  copy_async_commit();
  // Level-0 codes by window rows r = z*17 + y: a row with y or z odd holds
  // 17 level-0 points at consecutive slots rows[r] + x, a row with both even
  // its 8 odd-x points at rows[r] + x/2.
  // Interior tiles with 16-byte aligned codes load them in 16-byte chunks
  // (fetch_level0_vec): a third of the instructions of one copy per code, but
  // the codes are stored from registers, so the loads must have arrived.
  // Float tiles (seven per SM) do that before the coarse levels; double
  // tiles (five per SM, which hide less of that wait) bring the rows into L2
  // now and load them after the coarse levels (1-3% faster than copies
  // landing during the coarse levels; loading before them was 3% slower).
  const bool late = sizeof(T) == 8 && !EDGE && maxlevel >= 0 && (reinterpret_cast<uintptr_t>(qc) & 15) == 0;
  if (late) {
    for (int r = tid; r < kWin * kWin; r += kPredThreads) {
      const int y = r % kWin, z = r / kWin, n = ((y | z) & 1) ? kWin : 8;
      const int32_t* p = qc + sm.rows[r];
      prefetch_l2(p);
      prefetch_l2(p + n - 1);
    }
  } else if (sizeof(T) == 4 && !EDGE && maxlevel >= 0 && (reinterpret_cast<uintptr_t>(qc) & 15) == 0) {
    fetch_level0_vec<T>(sm, qc, tid);  // 2.5-9% faster than the copies below
  } else {
    // Each half-warp takes x = 0..15 of one row (the row's slot base is one
    // shared broadcast), then x = 16.
    static_assert(2 * (kPredThreads / 32) == 16, "rows advance by 16: (y, z) -> (y - 1, z + 1) or (16, z)");
    const int lane = tid & 31, x = lane & 15;
    const bool codes = maxlevel >= 0;
    int r = (tid >> 5) * 2 + (lane >> 4), y = r, z = 0;  // r = 17 z + y
    for (; r < kWin * kWin; r += 16) {
      const int ee = ((y | z) & 1) == 0;
      if (!ee || (x & 1)) {
        T* dst = &sm.win[Win<T>::at(x, y, z)];
        if (codes && L.in_data(x, y, z)) copy_async<4>(dst, qc + (sm.rows[r] + (uint64_t)(x >> ee)));
        else *dst = T(0);
      }
      if (y == 0) {
        y = 16;
      } else {
        --y;
        ++z;
      }
    }
    for (int r = tid; r < kWin * kWin; r += kPredThreads) {
      const int y = r % kWin, z = r / kWin;
      if (((y | z) & 1) == 0) continue;
      T* dst = &sm.win[Win<T>::at(16, y, z)];
      if (maxlevel >= 0 && L.in_data(16, y, z)) copy_async<4>(dst, qc + (sm.rows[r] + 16));
      else *dst = T(0);
    }
  }
  copy_async_commit();
  copy_async_wait_group<1>();
  __syncthreads();
  if (tid < 8) {  // x_reset_scratch_data (:1027-1067): anchors at the corners
    int x = (tid & 1) * 16, y = ((tid >> 1) & 1) * 16, z = (tid >> 2) * 16;
    uint32_t ax = x / 16 + bi[0], ay = y / 16 + bi[1], az = z / 16 + bi[2];
    if (ax < g.ax && ay < g.ay && az < g.az)
      sm.win[Win<T>::at(x, y, z)] = anchors[ax + (uint64_t)ay * g.ax + (uint64_t)az * g.ax * g.ay];
  }
  __syncthreads();
  sweep_coarse<T, false, EDGE>(sm.win, nullptr, f.lim, f.last[2], sm.p);
  if (late) fetch_level0_vec<T>(sm, qc, tid);
  copy_async_wait_group<0>();
  __syncthreads();
  sweep_fine<T, false, EDGE>(sm.win, nullptr, f.lim, f.last[2], sm.p);
  if constexpr (!EDGE) {
    // An interior tile writes 256 full rows of 16 values.  When every row
    // start is aligned to a pair of values (even row stride, aligned
    // buffers), pairs move as one vector: 2048 pairs, four in flight per
    // thread, pair q at x = 2 (q % 8), y = q / 8 % 16, z = q / 128.
    using V = typename PairOf<T>::type;
    const uintptr_t ends = reinterpret_cast<uintptr_t>(out + base) | (PROG ? reinterpret_cast<uintptr_t>(old + base) : 0);
    const bool pairs = (sy & 1) == 0 && ends % sizeof(V) == 0;
    if (pairs) {
      for (int b = tid; b < 2048; b += 4 * kPredThreads) {
        V o[4];
        if (PROG) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int q = b + k * kPredThreads, x = 2 * (q & 7), y = (q >> 3) & 15, z = q >> 7;
            o[k] = *reinterpret_cast<const V*>(old + base + x + (uint64_t)y * sy + (uint64_t)z * sz);
          }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int q = b + k * kPredThreads, x = 2 * (q & 7), y = (q >> 3) & 15, z = q >> 7;
          const int wi = Win<T>::at(x, y, z);
          V v;
          v.x = sm.win[wi];
          v.y = sm.win[wi + 1];
          if (PROG) {
            v.x = Fp<T>::add(v.x, o[k].x);
            v.y = Fp<T>::add(v.y, o[k].y);
          }
          *reinterpret_cast<V*>(out + base + x + (uint64_t)y * sy + (uint64_t)z * sz) = v;
        }
      }
      return;
    }
  }
  // The tile's points (16 per axis, plus the plane at 16 on the field's last
  // slab along that axis), enumerated over a fixed box so the coordinates
  // come from constant divisors.
  constexpr int kB = EDGE ? kWin : 16, kBox = kB * kB * kB;
  const int xs = 16 + (EDGE && f.last[0]), ys = 16 + (EDGE && f.last[1]), zs = 16 + (EDGE && f.last[2]);
  for (int b = tid; b < kBox; b += kPrefetch * kPredThreads) {
    T o[kPrefetch];
    if (PROG) {
#pragma unroll
      for (int k = 0; k < kPrefetch; ++k) {
        const int i = b + k * kPredThreads, x = i % kB, y = (i / kB) % kB, z = i / (kB * kB);
        o[k] = T(0);
        if (i < kBox && x < xs && y < ys && z < zs && L.in_data(x, y, z))
          o[k] = old[base + x + (uint64_t)y * sy + (uint64_t)z * sz];
      }
    }
#pragma unroll
    for (int k = 0; k < kPrefetch; ++k) {
      const int i = b + k * kPredThreads, x = i % kB, y = (i / kB) % kB, z = i / (kB * kB);
      if (i >= kBox || x >= xs || y >= ys || z >= zs || !L.in_data(x, y, z)) continue;
      T v = sm.win[Win<T>::at(x, y, z)];
      out[base + x + (uint64_t)y * sy + (uint64_t)z * sz] = PROG ? Fp<T>::add(v, o[k]) : v;
    }
  }
}

template <class T, bool PROG, int PART>
__global__ void __launch_bounds__(kPredThreads, reconstruct_min_ctas<T, PART>())
reconstruct_kernel(const int32_t* __restrict__ qc, const T* __restrict__ anchors, Geometry g,
                   const PredParams<T>* __restrict__ pp, const T* old, T* out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint32_t bi[3];
  tile_of_block<PART>(g, bi);
  reconstruct_tile<T, PROG, PART == 1>(*reinterpret_cast<ReconSmem<T>*>(smem_raw), qc, anchors, g, bi, pp, old, out);
}

// Both parts in one launch, as predict_compress_both_kernel.  A whole
// decompression with two launches and with one, just below the limit (740 tiles,
// 64x80x592): float 85 -> 76 us (61x77x590: 105 -> 80), double level (82-87
// either way; its two progressive steps 171 -> 168).  Above it, one launch would
// take 3-18 us less up to 1536 tiles and as much at 2304.
constexpr int kReconBothCtas = 5;
template <class T, bool PROG>
__global__ void __launch_bounds__(kPredThreads, kReconBothCtas)
reconstruct_both_kernel(const int32_t* __restrict__ qc, const T* __restrict__ anchors, Geometry g,
                        const PredParams<T>* __restrict__ pp, const T* old, T* out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ReconSmem<T>& sm = *reinterpret_cast<ReconSmem<T>*>(smem_raw);
  const uint32_t edge = (uint32_t)tiles_in_part(g, 1);
  uint32_t bi[3];
  if (blockIdx.x < edge) {
    tile_of_index<1>(g, blockIdx.x, bi);
    reconstruct_tile<T, PROG, true>(sm, qc, anchors, g, bi, pp, old, out);
  } else {
    tile_of_index<0>(g, blockIdx.x - edge, bi);
    reconstruct_tile<T, PROG, false>(sm, qc, anchors, g, bi, pp, old, out);
  }
}

// Trailer of a container (compress_merge, compressor.cu:139-151): use_md[4],
// reverse[4], double range, size_t comp_size_bp[4][32], anchors.  Words w,
// w + step, ... below `limit` (every field is a multiple of 4 bytes); stored
// as words where the trailer is aligned for it.
template <class T>
__device__ __forceinline__ void write_trailer(uint8_t* tr, const PredParams<T>* p, const double* range,
                                              const uint64_t* csbp, const T* anchors, uint64_t nanchors, uint64_t w,
                                              uint64_t step, uint64_t limit) {
  const uint64_t total = (1040 + nanchors * sizeof(T)) / 4;
  const bool aligned = (reinterpret_cast<uintptr_t>(tr) & 3) == 0;
  for (; w < total && w < limit; w += step) {
    uint32_t v;
    if (w == 0) v = p->use_md[0] | p->use_md[1] << 8 | p->use_md[2] << 16 | (uint32_t)p->use_md[3] << 24;
    else if (w == 1) v = p->reverse[0] | p->reverse[1] << 8 | p->reverse[2] << 16 | (uint32_t)p->reverse[3] << 24;
    else if (w < 4) v = reinterpret_cast<const uint32_t*>(range)[w - 2];
    else if (w < 260) v = reinterpret_cast<const uint32_t*>(csbp)[w - 4];
    else v = reinterpret_cast<const uint32_t*>(anchors)[w - 260];
    if (aligned) {
      reinterpret_cast<uint32_t*>(tr)[w] = v;
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) tr[4 * w + k] = (uint8_t)(v >> (8 * k));
    }
  }
}

template <class T>
constexpr int compress_smem_bytes() { return (int)sizeof(CompressSmem<T>); }
template <class T>
constexpr int recon_smem_bytes() { return (int)sizeof(ReconSmem<T>); }

}  // namespace prism_b200
