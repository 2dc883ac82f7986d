// sg4_fixed.cuh -- the H.psi work items in block fixed point.
//
// GB300 runs two FP64 multiply-adds a clock and SM, but nine to ten of these in
// fixed point (evr_probe_fp64_peak: 1.25 TFLOP/s, evr_probe_fixed_peak: 5.8), so
// the items' contractions -- the 1-D passes, the derivatives, the metric -- run
// on the integer pipe: a value is a 60-bit integer in two limbs,
//   value = (h 2^29 + l) 2^e,  |l| <= 2^28,  |h| <= 2^30,
// with one exponent e per right-hand side of an item and stage, and a
// multiply-add is three 32 x 32 + 64-bit ones into two 64-bit accumulators,
//   hh += xh mh,  mid += xh ml + xl mh
// (the xl ml product is below 2^-60 of full scale).  Matrices are scaled so
// that the absolute sum of every row is at most 2^58, so a pass cannot
// overflow; every pass ORs the magnitudes of what it stores per right-hand
// side, and the next pass shifts the headroom it finds there into its result,
// so each pass loses only the bits by which its own row-sum bound exceeds its
// result (two to four), not the product of all of them.  That keeps 55 to 57
// bits of each stage's largest value, at every point alike; a double has 53 of
// each value.
//
// A right-hand side whose largest entry in a term lies outside 2^+-300 (all
// subnormal, for instance), or is not finite, and one whose result is small
// against what the scheme's errors could make of it (fx_grid: a potential so
// steep that the tails of x carry it, say), goes through the FP64 code instead,
// that column alone.  Operators the scheme does not suit (see fx_prepare in
// sg4_device.cu) never come here.
#pragma once
#include "sg4_items.cuh"

namespace evr {

enum {
  FX_MAXR = 2,                  // right-hand sides per item
  FX_MAXD = 12,                 // modes
  FX_STAGES = 2 * FX_MAXD + 3,  // recorded magnitudes: gather, B->G passes, U, O, G->B passes
  FX_FLUSH = 24,                // products |xh ml| <= 2^58 an accumulator takes before it is folded
  FX_TILE = 32,                 // points per tile of the fixed-point metric
  FX_AHEAD = 4,                 // loads ahead of their products from global scratch
  FX_NONE = -(1 << 30),         // exponent of a type-1 mode without a derivative term
  FX_MARGIN_V = 5,              // bits by which a result may stay below its bound (fx_grid)
  FX_MARGIN_1 = 5,
  FX_MARGIN_10 = 9
};

// int2 values of one tile of the fixed-point metric: its D*D elements, rounded
// up to whole pairs, of 32 points; element ij of point q of the tile sits at
// (ij/2)*64 + 2 q + (ij & 1), so that a warp reads two elements of its 32
// points as one 512-byte access, at fixed offsets from the tile's start.
__host__ __device__ __forceinline__ int fx_tile_size(int D) { return (D * D + 1) / 2 * 2 * FX_TILE; }
__device__ __forceinline__ long long fx_g_index(int D, long long tile0, int q, int ij) {
  return (tile0 + q / FX_TILE) * fx_tile_size(D) + (ij >> 1) * (2 * FX_TILE) + 2 * (q % FX_TILE) + (ij & 1);
}

struct FxPass {  // a basis<->grid pass: mode of rank k in the mode order
  int nb, nq;
  int S, nf;            // stride of the mode, fibres
  unsigned mgS, mgF;    // ceil(2^31 / S), ceil(2^31 / nf), or 0: divide
  int mB, mG;           // its two matrices (int2 index into shared memory)
  int recB, recG;       // whether the pass records magnitudes
};

struct FxShared {
  FxPass ps[FX_MAXD];
  int4 md[FX_MAXD];               // per mode: nq, grid stride, derivative matrix (-1: none), magic of nq
  int moff[FX_MAXD];              // where the mode's matrices start in shared memory
  unsigned mx[FX_STAGES][FX_MAXR];  // OR of |h| of what stage s stored, per right-hand side (0: see fx_grid)
  int em[FX_MAXR];                // largest biased exponent of the gathered column
  int mv[FX_MAXR];                // largest bits(|h|) + biased exponent of V over the points
  int evmax;                      // largest biased exponent of V
  int e[FX_MAXR], eo[FX_MAXR];    // exponents of the running stage and of the grid result
  int deriv;                      // type 1: some mode has a derivative term
  int bad;                        // columns left to the FP64 code
  int msz;                        // int2 values of the term's matrices
  long long tile;                 // the term's first tile of the metric
  double wf, wl;                  // weight times the matrices' scales, in two parts
};

// The item's matrices, then its work arrays x and U_1..U_D (type 10) or O.
extern __shared__ __align__(16) int4 fx_sm[];

// The accumulators of one sum of products: its value is
// (hh 2^29 + m1 + m2) 2^29.
struct FxAcc {
  long long hh, m1, m2;
};
// mul.wide by name, the sum in C++: of (long long)a * b the compiler may form
// 64-bit products, and of mad.wide by name sums of pairs with extra adds.
__device__ __forceinline__ long long fx_mul(int a, int b) {
  long long r;
  asm("mul.wide.s32 %0, %1, %2;" : "=l"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ void fx_mac(FxAcc& s, int xh, int xl, int2 m) {
  s.hh += fx_mul(xh, m.x);
  s.m1 += fx_mul(xh, m.y);
  s.m2 += fx_mul(xl, m.x);
}

// A value and its limbs.  The sums that are stored carry an offset of 2^28
// from their start constant (fx_start): then the limbs are a shift and a mask.
__device__ __forceinline__ int2 fx_split(long long y) {  // y = value + 2^28
  return make_int2((int)(y >> 29), (int)((unsigned)y & 0x1fffffffu) - 0x10000000);
}
__device__ __forceinline__ int2 fx_pack(long long y) { return fx_split(y + (1 << 28)); }

// Start of a sum whose inputs left a bits of headroom, and its full-scale
// result shifted up by those bits, plus 2^28: the constant rounds the shift
// and adds the offset of fx_split.
__device__ __forceinline__ FxAcc fx_start(int a) { return FxAcc{0, ((1LL << 29) + 1) << (28 - a), 0}; }
__device__ __forceinline__ long long fx_sum(const FxAcc& s, int a) {
  return (s.hh << a) + ((s.m1 + s.m2) >> (29 - a));
}

// bits by which the recorded magnitudes stay below full scale
__device__ __forceinline__ int fx_head(unsigned m) { return m ? min(max(__clz((int)m) - 2, 0), 28) : 0; }

// u / n with mg = ceil(2^31 / n) (exact for u n < 2^31), or mg = 0: divide
template <bool FAST>
__device__ __forceinline__ int fx_div(int u, int n, unsigned mg) {
  if (FAST || mg) return (int)(((unsigned long long)(unsigned)u * mg) >> 31);
  return u / n;
}

// floor((t 2^29 + f) / 2^s), f in [0, 2^29), s >= 0, for results within 64 bits
__device__ __forceinline__ long long fx_shr(long long t, unsigned f, int s) {
  const unsigned tl = (unsigned)t, th = (unsigned)((unsigned long long)t >> 32);
  const unsigned k = (unsigned)s + 3;
  const long long far = t >> min(max(s - 29, 0), 63);
  const unsigned lo = __funnelshift_r(f << 3, tl, k), hi = __funnelshift_r(tl, th, k);
  return k < 32 ? (long long)(((unsigned long long)hi << 32) | lo) : far;
}

// the C right-hand sides of one element
template <int C>
struct FxVal {
  int h[C], l[C];
};

// A work array of C columns, the columns of an element side by side (one
// 16-byte access for both).  SM: in shared memory.
template <int C, bool SM>
struct FxArr;
template <int C>
struct FxArr<C, true> {
  int b;
  __device__ __forceinline__ FxArr(int start) : b(start / C) {}
  __device__ __forceinline__ FxVal<C> load(int i) const {
    if constexpr (C == 1) {
      const int2 t = reinterpret_cast<const int2*>(fx_sm)[b + i];
      return FxVal<1>{{t.x}, {t.y}};
    } else {
      const int4 t = fx_sm[b + i];
      return FxVal<2>{{t.x, t.z}, {t.y, t.w}};
    }
  }
  __device__ __forceinline__ void store(int i, const FxVal<C>& v) const {
    if constexpr (C == 1) reinterpret_cast<int2*>(fx_sm)[b + i] = make_int2(v.h[0], v.l[0]);
    else fx_sm[b + i] = make_int4(v.h[0], v.l[0], v.h[1], v.l[1]);
  }
  __device__ __forceinline__ long long* raw(int i, int w) const {  // the eight bytes of one value
    return reinterpret_cast<long long*>(fx_sm) + (b + i) * C + w;
  }
};
template <int C>
struct FxArr<C, false> {
  int2* b;
  __device__ __forceinline__ FxArr(int2* start) : b(start) {}
  __device__ __forceinline__ FxVal<C> load(int i) const {
    if constexpr (C == 1) {
      const int2 t = b[i];
      return FxVal<1>{{t.x}, {t.y}};
    } else {
      const int4 t = reinterpret_cast<const int4*>(b)[i];
      return FxVal<2>{{t.x, t.z}, {t.y, t.w}};
    }
  }
  __device__ __forceinline__ void store(int i, const FxVal<C>& v) const {
    if constexpr (C == 1) b[i] = make_int2(v.h[0], v.l[0]);
    else reinterpret_cast<int4*>(b)[i] = make_int4(v.h[0], v.l[0], v.h[1], v.l[1]);
  }
  __device__ __forceinline__ long long* raw(int i, int w) const { return reinterpret_cast<long long*>(b) + i * C + w; }
};

// Where an item's arrays are: x, T, and U_1..U_D at T, of which the first nfit
// lie there and the rest at U2 (only outside shared memory).
template <int C, bool SM>
struct FxBufs;
template <int C>
struct FxBufs<C, true> {
  int X, T, NQR;
  __device__ __forceinline__ FxArr<C, true> x() const { return FxArr<C, true>(X); }
  __device__ __forceinline__ FxArr<C, true> t() const { return FxArr<C, true>(T); }
  __device__ __forceinline__ FxArr<C, true> u(int i) const { return FxArr<C, true>(T + i * NQR); }
};
template <int C>
struct FxBufs<C, false> {
  int2 *X, *T, *U2;
  int nfit, NQR;
  __device__ __forceinline__ FxArr<C, false> x() const { return FxArr<C, false>(X); }
  __device__ __forceinline__ FxArr<C, false> t() const { return FxArr<C, false>(T); }
  __device__ __forceinline__ FxArr<C, false> u(int i) const {
    return FxArr<C, false>(i < nfit ? T + (long long)i * NQR : U2 + (long long)(i - nfit) * NQR);
  }
};

// ORs a warp's magnitudes of one column into the stage's record
__device__ __forceinline__ void fx_record(unsigned* slot, unsigned m) {
  m = __reduce_or_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0 && m) atomicOr(slot, m);
}

__device__ __forceinline__ int fx_bad_exp(int em) { return em > 1323 || (em && em < 723); }

// One basis->grid or grid->basis pass, one thread per output element of all C
// columns.  kind 0 stores; 1 stores the grid values of the last basis->grid
// pass and records the largest |V x|; 2 writes the weighted contributions of
// the last grid->basis pass.  NIN 0: nin at run time.
template <int NIN, int C, bool SM>
__device__ __forceinline__ void fx_pass_n(const KParams& p, const ItemShared& it, FxShared& fs, const FxPass& ps,
                                          int nin, int nout, int M, int si, int so, const FxArr<C, SM> in,
                                          const FxArr<C, SM> out, int kind) {
  const int S = ps.S, nf = ps.nf, tot = nf * nout;
  if ((int)(threadIdx.x & ~31u) >= tot) return;  // a warp without an output
  const unsigned mgF = ps.mgF, mgS = ps.mgS;
  int a[C];
  unsigned m[C];
  int mv[C], ev = 0;
#pragma unroll
  for (int w = 0; w < C; ++w) {
    a[w] = si > 0 ? fx_head(fs.mx[si][w]) : 0;
    m[w] = 0;
    mv[w] = 0;
  }
  for (int u = threadIdx.x; u < tot; u += blockDim.x) {
    const int k = fx_div<SM>(u, nf, mgF), f = u - k * nf;
    const int b = fx_div<SM>(f, S, mgS), c = f - b * S;
    const int i0 = c + S * nin * b, row = M + k * nin;
    FxAcc s[C];
#pragma unroll
    for (int w = 0; w < C; ++w) s[w] = fx_start(a[w]);
    const int2* Ms = reinterpret_cast<const int2*>(fx_sm);
    if constexpr (NIN > 0) {
#pragma unroll
      for (int i = 0; i < NIN; ++i) {
        const int2 mm = Ms[row + i];
        const FxVal<C> v = in.load(i0 + S * i);
#pragma unroll
        for (int w = 0; w < C; ++w) fx_mac(s[w], v.h[w], v.l[w], mm);
      }
    } else {
      for (int i = 0; i < nin; ++i) {
        const int2 mm = Ms[row + i];
        const FxVal<C> v = in.load(i0 + S * i);
#pragma unroll
        for (int w = 0; w < C; ++w) fx_mac(s[w], v.h[w], v.l[w], mm);
      }
    }
    const int o = c + S * (k + nout * b);
    if (kind == 2) {
      if (__ldg(p.map + it.off_nb + o) > 0) {
        double* cb = p.contrib + (it.off_nb + o) * p.nrhs_v + it.rhs0;
#pragma unroll
        for (int w = 0; w < C; ++w) {
          const double y = (double)(fx_sum(s[w], a[w]) - (1 << 28)) *
                           __hiloint2double((1023 + fs.eo[w] - a[w]) << 20, 0);
          cb[w] = fma(y, fs.wf, y * fs.wl);
        }
      }
    } else {
      FxVal<C> y;
#pragma unroll
      for (int w = 0; w < C; ++w) {
        const int2 t = fx_split(fx_sum(s[w], a[w]));
        y.h[w] = t.x;
        y.l[w] = t.y;
        m[w] |= (unsigned)(t.x ^ (t.x >> 31));
      }
      out.store(o, y);
      if (kind == 1) {
        const int e = (__double2hiint(__ldg(p.V + it.off_nq + o)) >> 20) & 0x7ff;
        ev = max(ev, e);
#pragma unroll
        for (int w = 0; w < C; ++w) mv[w] = max(mv[w], 32 - __clz(y.h[w] ^ (y.h[w] >> 31)) + e);
      }
    }
  }
  if (so > 0) {
#pragma unroll
    for (int w = 0; w < C; ++w) fx_record(&fs.mx[so][w], m[w]);
  }
  if (kind == 1) {
#pragma unroll
    for (int w = 0; w < C; ++w) {
      mv[w] = __reduce_max_sync(0xffffffffu, mv[w]);
      if ((threadIdx.x & 31) == 0) atomicMax(&fs.mv[w], mv[w]);
    }
    ev = __reduce_max_sync(0xffffffffu, ev);
    if ((threadIdx.x & 31) == 0) atomicMax(&fs.evmax, ev);
  }
}

template <int C, bool SM>
__device__ __noinline__ void fx_pass(const KParams& p, const ItemShared& it, FxShared& fs, int rank, bool to_grid,
                                     int si, int so, const FxArr<C, SM> in, const FxArr<C, SM> out, int kind) {
  const FxPass& ps = fs.ps[rank];
  const int nin = to_grid ? ps.nb : ps.nq, nout = to_grid ? ps.nq : ps.nb;
  const int M = to_grid ? ps.mB : ps.mG;
  if constexpr (SM) {
    switch (nin) {
#define EVR_CASE(n) \
  case n:           \
    fx_pass_n<n, C, SM>(p, it, fs, ps, n, nout, M, si, so, in, out, kind); return;
      EVR_CASE(1) EVR_CASE(2) EVR_CASE(3) EVR_CASE(4) EVR_CASE(5)
#undef EVR_CASE
      default: break;
    }
  }
  fx_pass_n<0, C, SM>(p, it, fs, ps, nin, nout, M, si, so, in, out, kind);
}

// sum over a fibre: n products of a matrix row with the fibre's values.  Two
// values are loaded ahead of their products, or four where they come from
// global scratch (L2 latency): with four 2.82 ms on the 6-D benchmark, three
// 2.87, two 3.00.
template <int C, bool SM>
__device__ __forceinline__ void fx_fibre(FxAcc (&s)[C], int row, const FxArr<C, SM>& a, int i0, int n, int sd) {
  constexpr int U = SM ? 2 : FX_AHEAD;
  const int2* Ms = reinterpret_cast<const int2*>(fx_sm);
  int m = 0;
  for (; m + U <= n; m += U, row += U, i0 += U * sd) {
    FxVal<C> v[U];
#pragma unroll
    for (int k = 0; k < U; ++k) v[k] = a.load(i0 + k * sd);
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const int2 mm = Ms[row + k];
#pragma unroll
      for (int w = 0; w < C; ++w) fx_mac(s[w], v[k].h[w], v[k].l[w], mm);
    }
  }
  if (U == 2) {
    if (m < n) {
      const int2 m0 = Ms[row];
      const FxVal<C> v0 = a.load(i0);
#pragma unroll
      for (int w = 0; w < C; ++w) fx_mac(s[w], v0.h[w], v0.l[w], m0);
    }
  } else if (m < n) {  // one to U - 1 left
    FxVal<C> v[U - 1];
#pragma unroll
    for (int k = 0; k < U - 1; ++k) v[k] = a.load(m + k < n ? i0 + k * sd : i0);
#pragma unroll
    for (int k = 0; k < U - 1; ++k)
      if (m + k < n) {
        const int2 mm = Ms[row + k];
#pragma unroll
        for (int w = 0; w < C; ++w) fx_mac(s[w], v[k].h[w], v[k].l[w], mm);
      }
  }
}

// Type 10, pass A: phi_j = d_j x at every point, then U_i = sum_j G_ji phi_j.
template <int DD, int C, bool SM>
__device__ __forceinline__ void fx_type10_a(const KParams& p, const ItemShared& it, FxShared& fs,
                                            const FxBufs<C, SM>& B) {
  const int nqt = it.nq_t;
  int a[C];
  unsigned m[C];
#pragma unroll
  for (int w = 0; w < C; ++w) {
    a[w] = fx_head(fs.mx[DD][w]);
    m[w] = 0;
  }
  const FxArr<C, SM> x = B.x();
  const int2* G0 = p.Gfx + fs.tile * fx_tile_size(DD) + 2 * (threadIdx.x & 31);
  for (int q = threadIdx.x; q < nqt; q += blockDim.x) {
    FxVal<C> phi[DD];
    unsigned rem = (unsigned)q;
#pragma unroll
    for (int j = 0; j < DD; ++j) {
      const int4 md = fs.md[j];
      const unsigned quo = md.w ? __umulhi(rem, (unsigned)md.w) : rem;
      const int idx = (int)(rem - quo * (unsigned)md.x);
      rem = quo;
      FxAcc s[C];
#pragma unroll
      for (int w = 0; w < C; ++w) s[w] = fx_start(a[w]);
      fx_fibre<C, SM>(s, md.z + idx * md.x, x, q - idx * md.y, md.x, md.y);
#pragma unroll
      for (int w = 0; w < C; ++w) {
        const int2 t = fx_split(fx_sum(s[w], a[w]));
        phi[j].h[w] = t.x;
        phi[j].l[w] = t.y;
      }
    }
    // blockDim.x is a multiple of the tile, so q's place in its tile is the lane
    const int4* g = reinterpret_cast<const int4*>(G0 + (long long)(q / FX_TILE) * fx_tile_size(DD));
    int4 gg = make_int4(0, 0, 0, 0);
#pragma unroll
    for (int i = 0; i < DD; ++i) {
      FxAcc s[C];
#pragma unroll
      for (int w = 0; w < C; ++w) s[w] = fx_start(0);
#pragma unroll
      for (int j = 0; j < DD; ++j) {
        const int ij = i * DD + j;
        if (ij % 2 == 0) gg = __ldg(g + (ij / 2) * FX_TILE);
        const int2 ge = ij % 2 == 0 ? make_int2(gg.x, gg.y) : make_int2(gg.z, gg.w);
#pragma unroll
        for (int w = 0; w < C; ++w) fx_mac(s[w], phi[j].h[w], phi[j].l[w], ge);
      }
      FxVal<C> u;
#pragma unroll
      for (int w = 0; w < C; ++w) {
        const int2 t = fx_split(fx_sum(s[w], 0));
        u.h[w] = t.x;
        u.l[w] = t.y;
        m[w] |= (unsigned)(t.x ^ (t.x >> 31));
      }
      B.u(i).store(q, u);
    }
  }
#pragma unroll
  for (int w = 0; w < C; ++w) fx_record(&fs.mx[DD + 1][w], m[w]);
}

template <int C, bool SM>
__device__ __noinline__ void fx_type10_a_dispatch(const KParams& p, const ItemShared& it, FxShared& fs,
                                                  const FxBufs<C, SM> B) {
  switch (p.D) {
#define EVR_T10(n) \
  case n:          \
    fx_type10_a<n, C, SM>(p, it, fs, B); break;
    EVR_T10(1) EVR_T10(2) EVR_T10(3) EVR_T10(4) EVR_T10(5) EVR_T10(6) EVR_T10(7) EVR_T10(8) EVR_T10(9)
    EVR_T10(10) EVR_T10(11) EVR_T10(12)
#undef EVR_T10
    default: break;
  }
}

// The grid result O, per point: V x - 1/2 sum_i (d_i U_i) for type 10 (over x),
// V x + sum_i F2_ii (d2_i x) for type 1, V x for type 0 (both into T).  Its
// exponent bounds both parts: the derivative part from the recorded magnitudes
// and the row sums, V x from its recorded maximum.
//
// x is good to some 2^-57 of its largest value, at every point alike, where an
// FP64 item keeps 53 bits of each value, so the error of the result is some
// 2^-57 of max|V| max|x| and of the derivative part's row-sum bound.  An FP64
// item loses about 2^-53 of the larger part of the result itself.  A column
// whose result, or V x, stays more than a margin below those bounds is left to
// the FP64 code: a potential that is large where x is small, derivatives that
// cancel.  The margins are where errors in units of the FP64 items' reach about
// one (long-double oracle, columns from N(0, 1) to the lowest function): V x 5
// bits (4: harmonic vectors on 14 points would go too; 6: twice the error on
// walls), type 1 5, type 10 9 (its bound takes row sums twice); one less on a
// basis of a single term, whose FP64 errors no alternating sum adds up.  With
// the margins 2-D L=13 Morse and wall potentials give 0.4-1.3 times the FP64
// error (up to 500 times without), at 1 to 2 % of the time of the items.
template <int C, bool SM>
__device__ __noinline__ void fx_grid(const KParams& p, const ItemShared& it, FxShared& fs, const FxBufs<C, SM> B) {
  const int D = p.D, nqt = it.nq_t;
  const bool t10 = p.type == 10, hasT = t10 || fs.deriv;
  const int kD = D > 8 ? 4 : (D > 4 ? 3 : (D > 2 ? 2 : D - 1));
  int a[C], h[C], sP[C];
  unsigned m[C];
#pragma unroll
  for (int w = 0; w < C; ++w) {
    const int eX = fs.e[w], aX = fx_head(fs.mx[D][w]);
    // the derivative sum, shifted up by a, has the exponent eT and at most bT bits
    int eT = eX, bT = -100000, aT = 0;
    if (t10) {
      const int aU = fx_head(fs.mx[D + 1][w]);
      aT = max(0, aU - kD);
      eT = eX - aX + p.geg[it.term] - 1 - aT;
      if (fs.mx[D + 1][w]) bT = 59 + max(0, kD - aU) + eT;
    } else if (hasT) {
      aT = aX;
      eT = eX + p.geg[it.term] - aT;
      if (fs.mx[D][w]) bT = 59 + eT;
    }
    const bool hasV = p.V && fs.mv[w] > 600;  // V x is there, and not below 2^-400
    const int bV = hasV ? fs.mv[w] + (29 - 1022) + eX : -100000;
    int eO = max(bT, bV + 1) - 58;
    if (bT < -90000 && !hasV) eO = eX;
    if (hasT) eO = max(eO, eT + 1);
    a[w] = aT;
    h[w] = min(eO - eT, 62);
    sP[w] = 1051 + eO - eX;
    m[w] = 0;
    if (threadIdx.x == blockDim.x - 32) {  // the last warp: idle on a small term
      fs.eo[w] = eO;
      const int bX = 59 - aX + eX;
      int need = -100000;
      if (fs.mx[D][w]) {
        if (t10) need = bX + kD + p.geg[it.term] - 1 - (FX_MARGIN_10 - p.strict);
        else if (hasT) need = bT - (FX_MARGIN_1 - p.strict);
        if (p.V && fs.evmax) need = max(need, hasV ? fs.evmax - 1022 + bX - (FX_MARGIN_V - p.strict) : 100000);
      }
      fs.mx[0][w] = (unsigned)(need > bV ? need : -100000);
    }
  }
  const FxArr<C, SM> x = B.x(), O = t10 ? B.x() : B.t();
  for (int q = threadIdx.x; q < nqt; q += blockDim.x) {
    long long r[C];
#pragma unroll
    for (int w = 0; w < C; ++w) r[w] = 0;
    if (hasT) {
      FxAcc s[C];
#pragma unroll
      for (int w = 0; w < C; ++w) s[w] = FxAcc{0, 0, 0};
      unsigned rem = (unsigned)q;
      int cnt = 0;
      for (int i = 0; i < D; ++i) {
        const int4 md = fs.md[i];
        const unsigned quo = md.w ? __umulhi(rem, (unsigned)md.w) : rem;
        const int idx = (int)(rem - quo * (unsigned)md.x);
        rem = quo;
        if (md.z < 0) continue;
        if ((cnt += md.x) > FX_FLUSH) {
          cnt = md.x;
#pragma unroll
          for (int w = 0; w < C; ++w) {
            const long long mid = s[w].m1 + s[w].m2;
            s[w] = FxAcc{s[w].hh + (mid >> 29), mid & ((1 << 29) - 1), 0};
          }
        }
        fx_fibre<C, SM>(s, md.z + idx * md.x, t10 ? B.u(i) : x, q - idx * md.y, md.x, md.y);
      }
#pragma unroll
      for (int w = 0; w < C; ++w) {
        const long long t = (fx_sum(s[w], a[w]) + ((1LL << h[w]) >> 1)) >> h[w];
        r[w] = t10 ? -t : t;
      }
    }
    if (p.V) {
      // V = +-(vh 2^29 + vl) 2^(ev - 1080), the 53-bit mantissa shifted up by five
      const long long vb = __double_as_longlong(__ldg(p.V + it.off_nq + q));
      const int ev = (int)(vb >> 52) & 0x7ff;
      long long vm = (vb & 0xFFFFFFFFFFFFFLL) | (ev ? 0x10000000000000LL : 0);
      vm <<= 5;
      if (vb < 0) vm = -vm;
      const int2 vv = fx_pack(vm);
      const FxVal<C> xv = x.load(q);
#pragma unroll
      for (int w = 0; w < C; ++w) {
        FxAcc s = {0, 0, 0};
        fx_mac(s, xv.h[w], xv.l[w], vv);
        const long long mid = s.m1 + s.m2;
        r[w] += (fx_shr(s.hh + (mid >> 29), (unsigned)mid & ((1u << 29) - 1), max(sP[w] - ev, 1) - 1) + 1) >> 1;
      }
    }
    FxVal<C> y;
#pragma unroll
    for (int w = 0; w < C; ++w) {
      const int2 t = fx_pack(r[w]);
      y.h[w] = t.x;
      y.l[w] = t.y;
      m[w] |= (unsigned)(t.x ^ (t.x >> 31));
    }
    O.store(q, y);
  }
#pragma unroll
  for (int w = 0; w < C; ++w) fx_record(&fs.mx[D + 2][w], m[w]);
}

template <int C, bool SM>
__device__ __forceinline__ void fx_body(const KParams& p, const ItemShared& it, FxShared& fs,
                                        const FxBufs<C, SM>& B) {
  const int D = p.D, nbt = it.nb_t, tid = threadIdx.x;
  {  // the term's matrices, one warp per mode
    int2* Ms = reinterpret_cast<int2*>(fx_sm);
    for (int i = tid >> 5; i < D; i += blockDim.x >> 5) {
      const int nbq = 2 * it.nb[i] * it.nq[i], nqq = it.nq[i] * it.nq[i];
      const int2 *s1 = p.fxm + it.mo[i][M_BG], *s2 = p.fxm + it.mo[i][p.type == 10 ? M_D1 : M_D2];
      // type 1: the modes' derivative matrices, each kept on its own scale, go
      // into one sum: onto the term's
      const int sh = fs.md[i].z >= 0 ? it.st[i] : 0;
      for (int e = tid & 31; e < nbq + nqq; e += 32) {
        int2 m = __ldg(e < nbq ? s1 + e : s2 + (e - nbq));
        if (sh > 0 && e >= nbq) m = fx_pack((((((long long)m.x << 29) + m.y) >> (sh - 1)) + 1) >> 1);
        Ms[fs.moff[i] + e] = m;
      }
    }
  }
  // gather (tabPackedBasis_TO_tabR_AT_iG) into the buffer from which the D
  // ping-pong passes of basis->grid end in x: the doubles, then, with the
  // column's largest exponent known, its fixed-point values in their place
  const FxArr<C, SM> G0 = (D & 1) ? B.t() : B.x(), G1 = (D & 1) ? B.x() : B.t();
  const int* map = p.map + it.off_nb;
  int em[C];
#pragma unroll
  for (int w = 0; w < C; ++w) em[w] = 0;
  for (int k = tid; k < nbt; k += blockDim.x) {
    const int n = __ldg(map + k) - 1;
#pragma unroll
    for (int w = 0; w < C; ++w) {
      const int v = it.rhs0 + w;
      const double d =
          n >= 0 ? p.psi[(long long)(v >> p.cshift) * p.ldpsi + (((long long)n << p.cshift) | (v & p.cshift))] : 0.0;
      *G0.raw(k, w) = __double_as_longlong(d);
      em[w] = max(em[w], (__double2hiint(d) >> 20) & 0x7ff);
    }
  }
#pragma unroll
  for (int w = 0; w < C; ++w) {
    em[w] = __reduce_max_sync(0xffffffffu, em[w]);
    if ((tid & 31) == 0) atomicMax(&fs.em[w], em[w]);
  }
  __syncthreads();
#pragma unroll
  for (int w = 0; w < C; ++w) em[w] = fs.em[w];
  for (int k = tid; k < nbt; k += blockDim.x) {
    FxVal<C> f;
#pragma unroll
    for (int w = 0; w < C; ++w) {
      const long long b = *G0.raw(k, w);
      if (em[w] == 0 && (b << 1) != 0) atomicOr(&fs.bad, 1 << w);  // subnormal entries alone
      const int e = (int)(b >> 52) & 0x7ff, s = em[w] - e;
      long long y = ((b & 0xFFFFFFFFFFFFFLL) | (e ? 0x10000000000000LL : 0)) << 6;
      y = s > 60 || em[w] == 0 || fx_bad_exp(em[w]) ? 0 : (s ? ((y >> (s - 1)) + 1) >> 1 : y);
      const int2 t = fx_pack(b < 0 ? -y : y);
      f.h[w] = t.x;
      f.l[w] = t.y;
    }
    G0.store(k, f);
  }
  if (tid < C) {
    const bool bad = fx_bad_exp(fs.em[tid]);
    fs.e[tid] = fs.em[tid] && !bad ? fs.em[tid] - 1081 : 0;
    if (bad) atomicOr(&fs.bad, 1 << tid);
  }
  __syncthreads();
  for (int k = 0; k < D; ++k) {
    const int si = k && fs.ps[k - 1].recB ? k : 0;
    if (si && tid < C) fs.e[tid] -= fx_head(fs.mx[k][tid]);
    fx_pass<C, SM>(p, it, fs, k, true, si, fs.ps[k].recB ? k + 1 : 0, (k & 1) ? G1 : G0, (k & 1) ? G0 : G1,
                   k == D - 1 && p.V ? 1 : 0);
    __syncthreads();
  }
  if (p.type == 10) {
    fx_type10_a_dispatch<C, SM>(p, it, fs, B);
    __syncthreads();
  }
  fx_grid<C, SM>(p, it, fs, B);
  __syncthreads();
  const int lw = tid - ((int)blockDim.x - 32);
  if (lw >= 0 && lw < C &&
      (int)fs.mx[0][lw] > (fs.mx[D + 2][lw] ? fs.eo[lw] + 61 - __clz((int)fs.mx[D + 2][lw]) : -90000))
    atomicOr(&fs.bad, 1 << lw);
  const FxArr<C, SM> O0 = p.type == 10 ? B.x() : B.t(), O1 = p.type == 10 ? B.t() : B.x();
  for (int k = 0; k < D; ++k) {
    const bool last = k == D - 1;
    const int si = !k || fs.ps[D - k].recG ? D + 2 + k : 0;
    fx_pass<C, SM>(p, it, fs, D - 1 - k, false, si, !last && fs.ps[D - 1 - k].recG ? D + 3 + k : 0,
                   (k & 1) ? O1 : O0, (k & 1) ? O0 : O1, last ? 2 : 0);
    if (!last && si && lw >= 0 && lw < C) fs.eo[lw] -= fx_head(fs.mx[si][lw]);
    __syncthreads();
  }
}

// element (output i, input j) of the fixed-point metric as a double
__device__ __forceinline__ double gfx_value(const KParams& p, const ItemShared& it, int2 g, int i, int j) {
  const unsigned char* l = p.terms[it.term].l;
  const int e = p.geg[it.term] - 58 - p.ed[i * p.Lp1 + l[i]] - p.ed[j * p.Lp1 + l[j]];
  return (double)(((long long)g.x << 29) + g.y) * __hiloint2double((1023 + e) << 20, 0);
}

// a matrix row's products with the fibre through a point, added to s in FP64
__device__ __forceinline__ double fibre_fp64(const double* __restrict__ M, const double* a, int n, int sd, double s) {
  for (int m = 0; m < n; ++m) s = fma(__ldg(M + m), a[m * sd], s);
  return s;
}

// Columns of an item in FP64 (the exceptional ones, r of them from rhs on),
// with the operators that the fixed-point items take: x in A, then U_1..U_D or
// O, each column after column.  The sums are those of the FP64 items, in their
// order (type10_fused, type1_fused).
static __device__ __noinline__ void fx_item_fp64(const KParams& p, ItemShared& it, double* A, int rhs0, int bad,
                                                 long long tile) {
  const int r = __popc(bad), rhs = rhs0 + (bad == 2);
  const int D = p.D, nqt = it.nq_t, nbt = it.nb_t, NQR = nqt * r;
  const long long oq = it.off_nq;
  double* B = A + NQR;
  if (threadIdx.x == 0) {
    it.rhs0 = rhs;
    it.r = r;
  }
  if (threadIdx.x < D) {
    int rank = 0, st = 1;
    const int i = threadIdx.x, ni = it.nq[i] - it.nb[i], di = it.nb[i] * it.nq[i];
    for (int j = 0; j < D; ++j) {
      const int kj = (it.nq[j] - it.nb[j]) * di, ki = ni * (it.nb[j] * it.nq[j]);
      rank += j != i && (kj < ki || (kj == ki && j < i));
      if (j < i) st *= it.nq[j];
    }
    it.ord[rank] = i;
    it.pos[i] = rank;
    it.st[i] = st;
  }
  double* G0 = (D & 1) ? B : A;
  for (int e = threadIdx.x; e < nbt * r; e += blockDim.x) {
    const int w = e / nbt, n = __ldg(p.map + it.off_nb + e - w * nbt);
    G0[e] = n > 0 ? p.psi[vaddr(p, rhs + w, n - 1, p.ldpsi)] : 0.0;
  }
  __syncthreads();
  double* x = transform(p, it, true, G0, G0 == A ? B : A);  // == A
  double* y = p.type == 10 ? x : B;
  if (p.type == 10) {
    for (int e = threadIdx.x; e < NQR; e += blockDim.x) {
      const int q = e % nqt;
      double phi[FX_MAXD];
      int rem = q;
      for (int j = 0; j < D; ++j) {
        const int n = it.nq[j], st = it.st[j], idx = rem % n;
        rem /= n;
        phi[j] = fibre_fp64(p.mats + it.mo[j][M_D1] + idx * n, x + e - idx * st, n, st, 0.0);
      }
      for (int i = 0; i < D; ++i) {
        double u = 0.0;
        for (int j = 0; j < D; ++j)
          u = fma(gfx_value(p, it, __ldg(p.Gfx + fx_g_index(D, tile, q, i * D + j)), i, j), phi[j], u);
        B[(long long)i * NQR + e] = u;
      }
    }
    __syncthreads();
  }
  for (int e = threadIdx.x; e < NQR; e += blockDim.x) {
    const int q = e % nqt;
    double s = 0.0, o = p.V ? __ldg(p.V + oq + q) * x[e] : 0.0;
    int rem = q;
    for (int i = 0; i < D && p.type != 0; ++i) {
      const int n = it.nq[i], st = it.st[i], idx = rem % n;
      rem /= n;
      if (p.type == 10) {
        s = fibre_fp64(p.mats + it.mo[i][M_D1] + idx * n, B + (long long)i * NQR + e - idx * st, n, st, s);
      } else if (__ldg(p.F2 + i * D + i) != 0.0) {
        s = fibre_fp64(p.mats + it.mo[i][M_D2] + idx * n, x + e - idx * st, n, st, 0.0);
        o = fma(__ldg(p.F2 + i * D + i), s, o);
      }
    }
    y[e] = p.type == 10 ? fma(-0.5, s, o) : o;
  }
  __syncthreads();
  const double* yb = transform(p, it, false, y, y == A ? B : A);
  store_contrib(p, it, yb);
}

// One work item in fixed point (one or two columns), then its exceptional
// columns, if any, through the FP64 code.
__device__ __forceinline__ void run_item_fx(const KParams& p, ItemShared& it, FxShared& fs, int term, int rhs0, int r) {
  const int tid = threadIdx.x, D = p.D;
  if (tid == 0) {
    const TermInfo& T = p.terms[term];
    it.term = term;
    it.rhs0 = rhs0;
    it.r = r;
    it.off_nb = T.off_nb;
    it.off_nq = T.off_nq - p.fbase;
    fs.tile = p.fxterms[term].tile - p.tbase;
    it.nb_t = T.nb;
    it.nq_t = T.nq;
    it.w = T.w;
    fs.wf = p.fxterms[term].wf[p.transpose];
    fs.wl = p.fxterms[term].wl[p.transpose];
    fs.bad = 0;
    fs.evmax = 0;
    fs.deriv = 0;
  }
  if (tid < D) {
    const int l = p.terms[term].l[tid];
    const int k = tid * p.Lp1 + l;
    it.nb[tid] = p.nb_of_l[k];
    it.nq[tid] = p.nq_of_l[k];
    it.mg[tid] = it.nq[tid] > 1 ? 0xFFFFFFFFu / (unsigned)it.nq[tid] + 1u : 0u;
    for (int q = 0; q < 4; ++q) it.mo[tid][q] = p.mat_off[k * 8 + 4 * p.transpose + q];
    // the shift of the mode's type-1 matrix (the FP64 code keeps strides here)
    const int e1 = p.type == 1 ? __ldg(p.e1 + k) : FX_NONE;
    it.st[tid] = e1 == FX_NONE ? (p.type == 10 ? 0 : FX_NONE) : min(__ldg(p.geg + term) - e1, 62);
  }
  for (int e = tid; e < FX_STAGES * FX_MAXR; e += blockDim.x) (&fs.mx[0][0])[e] = 0;
  if (tid < FX_MAXR) {
    fs.em[tid] = 0;
    fs.mv[tid] = 0;
  }
  __syncthreads();
  if (tid < D) {  // each mode's rank (mode_order), and the extents of its passes
    const int i = tid, ni = it.nq[i] - it.nb[i], di = it.nb[i] * it.nq[i];
    int rank = 0, S = 1, R = 1, st = 1, mo = 0;
    for (int j = 0; j < D; ++j) {
      if (j == i) continue;
      if (j < i) mo += it.nq[j] * (2 * it.nb[j] + it.nq[j]);
      const int kj = (it.nq[j] - it.nb[j]) * di, ki = ni * (it.nb[j] * it.nq[j]);
      const bool before = kj < ki || (kj == ki && j < i);
      rank += before;
      const int c = before ? it.nq[j] : it.nb[j];
      if (j < i) {
        S *= c;
        st *= it.nq[j];
      } else {
        R *= c;
      }
    }
    FxPass ps;
    ps.nb = it.nb[i];
    ps.nq = it.nq[i];
    ps.S = S;
    ps.nf = S * R;
    // (in shared memory nf and nf nq are below 2^15: always exact)
    const bool fast = (unsigned long long)ps.nf * ps.nf * (unsigned)it.nq[i] < (1ull << 31);
    ps.mgS = fast ? ((1u << 31) + S - 1) / S : 0u;
    ps.mgF = fast ? ((1u << 31) + ps.nf - 1) / ps.nf : 0u;
    ps.mB = mo;  // the mode's matrices follow each other: B->G, G->B, derivative
    ps.mG = mo + di;
    fs.ps[rank] = ps;
    fs.moff[i] = mo;
    int md = mo + 2 * di;
    if (i == D - 1) fs.msz = (md + it.nq[i] * it.nq[i] + 1) & ~1;
    if (p.type != 10) {
      if (it.st[i] != FX_NONE) fs.deriv = 1;
      else md = -1;
    }
    fs.md[i] = make_int4(it.nq[i], st, md, (int)it.mg[i]);
  }
  __syncthreads();
  if (tid == 0) {
    // A pass over n inputs loses at most log2(n) bits and a little against its
    // row-sum bound; magnitudes are recorded, and the headroom used, whenever
    // the passes since the last record could lose two, and on the grid (four
    // saved 0.3 % of the time at most and cost up to two bits).
    int n = 1;
    for (int k = 0; k < D; ++k) {
      n *= fs.ps[k].nb;
      fs.ps[k].recB = n > 4 || k == D - 1;
      if (n > 4) n = 1;
    }
    n = 1;
    for (int k = D - 1; k >= 0; --k) {
      n *= fs.ps[k].nq;
      fs.ps[k].recG = n > 4;
      if (n > 4) n = 1;
    }
  }
  // work arrays x, then U_1..U_D (type 10) or O, behind the matrices: all in
  // shared memory, or as many whole ones as fit and the rest in this CTA's slab
  const int nq = it.nq_t, NQR = nq * r, msz = fs.msz;
  const int narr = p.type == 10 ? D + 1 : 2;
  const int fit = min(narr, (p.smem_doubles - msz) / NQR);
  int2* slab = reinterpret_cast<int2*>(p.gscratch + (long long)blockIdx.x * p.scratch_per_cta);
  if (fit == narr) {
    if (r == 1) fx_body<1, true>(p, it, fs, FxBufs<1, true>{msz, msz + NQR, NQR});
    else fx_body<2, true>(p, it, fs, FxBufs<2, true>{msz, msz + NQR, NQR});
  } else {
    int2* sm = reinterpret_cast<int2*>(fx_sm) + msz;
    int2* X = fit ? sm : slab;
    int2* Tb = fit >= 2 ? sm + NQR : (fit ? slab : slab + NQR);
    const int nfit = fit >= 2 ? fit - 1 : D;
    if (r == 1) fx_body<1, false>(p, it, fs, FxBufs<1, false>{X, Tb, slab, nfit, NQR});
    else fx_body<2, false>(p, it, fs, FxBufs<2, false>{X, Tb, slab, nfit, NQR});
  }
  if (fs.bad) {
    // the arrays of the item's columns, in the plan's slab where they exceed shared memory
    const bool in = (p.type == 10 ? D + 1LL : 2LL) * it.nq_t * r <= p.smem_doubles;
    double* A = in ? reinterpret_cast<double*>(fx_sm) : p.gscratch + (long long)blockIdx.x * p.scratch_per_cta;
    fx_item_fp64(p, it, A, rhs0, fs.bad, fs.tile);
  }
}

}  // namespace evr
