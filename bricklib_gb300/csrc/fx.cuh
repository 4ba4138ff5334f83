// FP64 stencil sums in fixed point on the integer multipliers.
//
// GB300 executes 2 FP64 operations per clock and SM, but 32 integer multiply-adds with a 32 x 32
// bit product and a 64-bit accumulator (mad.wide), so a 53-bit product is cheaper in four integer
// multiply-adds than in one DFMA, by a factor of four, and sums of input values in 64-bit integer
// additions are cheaper by a factor of sixteen (standalone probes: DFMA 2.0, mad.wide 32, 64-bit
// add 32 per clock and SM).
//
// Per brick: E is the largest biased exponent of the values the stencil reads around the brick
// (centre and faces / box of radius R).  Every value becomes an integer X = x * 2^(XB - 1 - (E - 1023)),
// |X| < 2^XB, XB = 60 (58 for the 125-point cube, whose classes add up to 24 values before they are
// multiplied): exact when its exponent is at least E - (XB - 53), else cut below 2^-XB of the largest.
// Coefficients are integers C = c * 2^q, with sum |C| <= 2^63 over the products of a point (host, fx_table).  With the halves
// X = xh 2^32 + xl and C = ch 2^32 + cl (xl, cl signed),
//   sum C X = 2^64 sum ch xh + 2^32 (sum ch xl + sum cl xh) + sum cl xl,
// whose first three sums are exact 64-bit integers and whose last (below 2^-61 of the largest total
// per product, with no preferred sign) is left out.  The total is rounded to units of 2^64 (2^-59
// of the largest possible one, less where values are added before they are multiplied) and then
// to a double.  Integer sums do not depend on their order: every kernel that sums a brick this way
// gives the same bits.
//
// A brick is computed this way only when the error bound is no larger than that of the chain of n
// FP64 multiply-adds, else its threads run FP64: E within the range where results
// are normal numbers (which leaves out infinities and NaNs), and every point has a term
// |c_t x_t| >= error / (n 2^-53) among its centre tap and, within its 2 x 2 x 2 block, its neighbour on
// each axis (cubes: all seven others).  error is the bound of what goes wrong here, in units of
// 2^(E - 1022): cut values 2^-XB sum |c|, rounded coefficients n 2^(-1 - q), one or two roundings of half
// a unit 2^(64 - q - XB), and 2^(31 - q - XB) sum |cl|.  It is then at most n 2^-53 max |c_t x_t|, the
// a-priori bound of the chain's own rounding errors; the rounding of the total to a double, half a
// unit of the result's last place, comes on top.  On uniform values the result is closer to the
// exact sum than the chain's; it need not be where a point has one large term and the others are
// next to nothing, since the chain then rounds once (half a unit of 2^-53; 1.07 of them were found
// here for a 7-point heat step on isolated values beside one 2^5 as large).  (Values that are all exact
// do not do instead of the check: where all but one of a point's values are zero, the chain is exact
// but for one rounding.)  Bricks that are zero throughout need no sums either way.
#pragma once

#include "bk_common.cuh"

namespace bk {

// Coefficients as fixed-point integers (filled by fx_table, sweep.cu).
constexpr int FX_TAPS = 27;
struct FxTab {
  int on;                        // 0: not usable; 1: per tap; 2: per class of equal coefficients
  int ch[FX_TAPS], cl[FX_TAPS];  // C = ch 2^32 + cl
  int w[8];                      // weights of the checked terms, by neighbour: 1 i, 2 j, 4 k
  int elo, ehi;                  // range of E
  int q;                         // C = c 2^q
  int zeros;                     // sums of +0 are +0 (they are -0 where all coefficients are negative)
};

bool fx_table(const double *c, int n, const int (*near)[9], int masks, int slots, const int *first, const int *count,
              int xb, bool one, FxTab *t);

// What a thread learns of its share of a brick's values, and after the exchange the whole brick's.
struct FxScan {
  unsigned top;  // largest high word without sign
  int term;      // smallest over points of the largest high word of a checked term
};

__device__ __forceinline__ unsigned fx_mag(double x) { return (unsigned)__double2hiint(x) & 0x7FFFFFFFu; }

// X of a value, for a brick whose largest biased exponent is E.
template <int XB>
__device__ __forceinline__ long long fx_of(double x, int E) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned mh = (hi & 0xFFFFFu) | 0x100000u;
  const unsigned long long v = ((unsigned long long)__funnelshift_l(lo, mh, 11) << 32) | (lo << 11);
  // 64 - XB for exponent E; 64 and more give 0 (shr clamps).  A biased exponent of 0 (zero, denormal)
  // is at least 72 below E: 0 whatever the implicit bit
  long long m;
  asm("{\n\t.reg .pred p;\n\t"
      "shr.u64 %0, %1, %2;\n\t"
      "setp.lt.s32 p, %3, 0;\n\t"
      "@p neg.s64 %0, %0;\n\t}\n"
      : "=l"(m)
      : "l"(v), "r"((unsigned)(64 - XB + E) - ((hi >> 20) & 0x7FFu)), "r"((int)hi));
  return m;
}
// The same by the FP64 unit: the exponent is shifted so that its conversion to integer, which cuts
// towards zero, gives X (values 2^70 below the largest become 0 first).  The unit converts 2 per
// clock and SM beside the integer pipes, which the 14 instructions above load; the centre of a brick
// is converted here and the values around it there (256^3, us, none / centre / all here: 7-point star
// 94.8 / 92.6 / 98.7, 125-point cube 301 / 298 / 390).
template <int XB>
__device__ __forceinline__ long long fx_of_unit(double x, int E) {
  const int hi = __double2hiint(x);
  const int h = (unsigned)(hi & 0x7FFFFFFF) >= (unsigned)(E - 70) << 20 ? hi + ((1022 + XB - E) << 20) : 0;
  long long r;
  asm("cvt.rzi.s64.f64 %0, %1;\n" : "=l"(r) : "d"(__hiloint2double(h, __double2loint(x))));
  return r;
}

// Signed halves of an integer: x = y * 2^32 + x, x in [-2^31, 2^31).
__device__ __forceinline__ int2 fx_split(long long x) {
  const int lo = (int)x;
  return make_int2(lo, (int)(x >> 32) + (int)((unsigned)lo >> 31));
}

// A sum of products.  ONE: sum ch xl (below 2^62 for any number of taps) and sum cl xh (2^59 a tap)
// in one accumulator, for up to 7 taps; else each its own (fx_table sees to |sum cl xh| < 2^63).
template <bool ONE>
struct FxAcc {
  long long a2, a1, b1;
  static constexpr long long HALF = 0x80000000ll;  // half a unit of sum()
  __device__ __forceinline__ void first(const FxTab &t, int q, int2 x) {
    a2 = (long long)t.ch[q] * x.y;
    a1 = (long long)t.ch[q] * x.x + HALF;
    if constexpr (ONE) a1 += (long long)t.cl[q] * x.y;
    else b1 = (long long)t.cl[q] * x.y + HALF;
  }
  __device__ __forceinline__ void add(const FxTab &t, int q, int2 x) {
    a2 += (long long)t.ch[q] * x.y;
    a1 += (long long)t.ch[q] * x.x;
    if constexpr (ONE) a1 += (long long)t.cl[q] * x.y;
    else b1 += (long long)t.cl[q] * x.y;
  }
  // the sum in units of 2^64
  __device__ __forceinline__ long long sum() const {
    if constexpr (ONE) return a2 + (a1 >> 32);
    return a2 + (a1 >> 32) + (b1 >> 32);
  }
};

// What turns a sum into the double of a brick of largest exponent E: added to its high word.
template <int XB>
__device__ __forceinline__ int fx_scale(int E, int q) { return (E + 64 - 1022 - XB - q) * (1 << 20); }
__device__ __forceinline__ double fx_result(long long y, int scale) {
  const double r = (double)y;
  const int hi = __double2hiint(r);
  return __hiloint2double(hi ? hi + scale : 0, __double2loint(r));
}

// Whether a brick with this scan is computed in fixed point.
__device__ __forceinline__ bool fx_ok(const FxTab &t, const FxScan &s) {
  const int E = (int)(s.top >> 20);
  return E >= t.elo && E <= t.ehi && s.term >= (int)(s.top & 0x7FF00000u);
}

// The scan of the brick's 64 threads from those of its two warps: each warp reduces and leaves
// its result in slot[warp]; the caller's barrier follows, then fx_gather.
__device__ __forceinline__ void fx_publish(FxScan s, int2 *slot, int lt) {
  s.top = __reduce_max_sync(0xFFFFFFFFu, s.top);
  s.term = __reduce_min_sync(0xFFFFFFFFu, s.term);
  if ((lt & 31) == 0) slot[lt >> 5] = make_int2((int)s.top, s.term);
}
__device__ __forceinline__ FxScan fx_gather(const int2 *slot) {
  const int2 a = slot[0], b = slot[1];
  return FxScan{max((unsigned)a.x, (unsigned)b.x), min(a.y, b.y)};
}

// Named barriers over the 64 threads of a brick: 1 for a CTA's first brick, 2 for its second.  The
// numbers are constants, since a barrier number in a register reserves all sixteen for the CTA,
// which leaves four resident CTAs per SM.
template <int ID>
__device__ __forceinline__ bool fx_bar_or_id(bool pred) {
  unsigned r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "bar.red.or.pred q, %2, 64, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}\n"
      : "=r"(r)
      : "r"((unsigned)pred), "n"(ID)
      : "memory");
  return r != 0;
}
__device__ __forceinline__ bool fx_bar_or(int brick, bool pred) {
  return brick == 0 ? fx_bar_or_id<1>(pred) : fx_bar_or_id<2>(pred);
}
__device__ __forceinline__ void fx_bar(int brick) {
  if (brick == 0) asm volatile("bar.sync 1, 64;\n" ::: "memory");
  else asm volatile("bar.sync 2, 64;\n" ::: "memory");
}

// A thread's share of a brick's values: its 2 x 2 x 2 block of the centre and its part of the values
// around it, read where From has them and stored as integers where To has them (the same place, or
// a tile of their own).  A place has block(k, j, i), the position of centre value (k, j, i), and
// for the others NP aligned pairs at pair(p) and NS single values at one(p) (where has(p)).  PAIR:
// values (i, i + 1) of an even i sit in one aligned 16-byte unit.  SWAP: the two rows of a block
// are taken in an order that differs between the lanes of a quarter warp, so that its 16-byte
// accesses fall in different banks where rows are 64 bytes apart.  SUM: integers are kept whole, to
// be added; else as their halves.  BOX: all eight values of a block are checked terms of each point.
template <bool PAIR, bool SWAP, bool SUM, bool BOX, int XB, class From, class To>
struct FxShare {
  static constexpr int NV = 8 + 2 * From::NP + From::NS;
  // values kept in registers between the scan and the conversion, or loaded again
  static constexpr bool HOLD = NV <= 20, STAR = !BOX;
  int lt;
  From from;
  To to;
  template <class Place>
  __device__ __forceinline__ int block(const Place &pl, int q) const {
    const int dj = q & 1;
    return pl.block(2 * (lt >> 4) + (q >> 1), 2 * ((lt >> 2) & 3) + (SWAP ? dj ^ ((lt >> 2) & 1) : dj), 2 * (lt & 3));
  }
  static __device__ __forceinline__ void ld2(const double *c, double &a, double &b) {
    if constexpr (PAIR) {
      const double2 x = *reinterpret_cast<const double2 *>(c);
      a = x.x;
      b = x.y;
    } else {
      a = c[0];
      b = c[1];
    }
  }
  static __device__ __forceinline__ void st2(double *c, double a, double b) {
    if constexpr (PAIR) *reinterpret_cast<double2 *>(c) = make_double2(a, b);
    else {
      c[0] = a;
      c[1] = b;
    }
  }
  // v: the block ([dk][dj][di]), the pairs, the single values (0 where there is none)
  __device__ __forceinline__ void load(const double *t, double (&v)[NV]) const {
#pragma unroll
    for (int q = 0; q < 4; ++q) ld2(t + block(from, q), v[2 * q], v[2 * q + 1]);
#pragma unroll
    for (int p = 0; p < From::NP; ++p) ld2(t + from.pair(p), v[8 + 2 * p], v[9 + 2 * p]);
#pragma unroll
    for (int p = 0; p < From::NS; ++p) v[8 + 2 * From::NP + p] = from.has(p) ? t[from.one(p)] : 0.0;
  }
  static __device__ __forceinline__ FxScan scan(const double (&v)[NV], const FxTab &tab) {
    FxScan s{0u, 0x7FFFFFFF};
    int a[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) a[q] = (int)fx_mag(v[q]);
    // every point's checked terms: its own value, and its i, j and k neighbours inside the block
    // (whichever side they lie on: the weight is that of the smaller of the two coefficients)
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      int t = a[q] + tab.w[0];
#pragma unroll
      for (int m = 1; m < 8; ++m)
        if (BOX || (m & (m - 1)) == 0) t = __viaddmax_s32(a[q ^ m], tab.w[m], t);
      s.term = min(s.term, t);
    }
#pragma unroll
    for (int q = 0; q < NV; ++q) s.top = max(s.top, fx_mag(v[q]));
    return s;
  }
  template <bool UNIT>
  static __device__ __forceinline__ double conv(double x, int E) {
    const long long X = UNIT ? fx_of_unit<XB>(x, E) : fx_of<XB>(x, E);
    if constexpr (SUM) return __longlong_as_double(X);
    const int2 h = fx_split(X);
    return __hiloint2double(h.y, h.x);
  }
  __device__ __forceinline__ void convert(double *t, const double (&v)[NV], int E) const {
#pragma unroll
    for (int q = 0; q < 4; ++q) st2(t + block(to, q), conv<true>(v[2 * q], E), conv<true>(v[2 * q + 1], E));
#pragma unroll
    for (int p = 0; p < From::NP; ++p) st2(t + to.pair(p), conv<false>(v[8 + 2 * p], E), conv<false>(v[9 + 2 * p], E));
#pragma unroll
    for (int p = 0; p < From::NS; ++p)
      if (to.has(p)) t[to.one(p)] = conv<false>(v[8 + 2 * From::NP + p], E);
  }
};
template <bool PAIR, bool SWAP, bool SUM, bool BOX, int XB, class From, class To>
__device__ __forceinline__ FxShare<PAIR, SWAP, SUM, BOX, XB, From, To> fx_share(int lt, From from, To to) {
  return FxShare<PAIR, SWAP, SUM, BOX, XB, From, To>{lt, from, to};
}

// Stars in a tile with position at(k, j, i): R values of each face, one by one.
template <int R, class At>
struct FxFaces {
  static constexpr int NP = 0, NS = 6 * R;
  int lt;
  At at;
  __device__ __forceinline__ int block(int k, int j, int i) const { return at(k, j, i); }
  __device__ __forceinline__ bool has(int) const { return true; }
  __device__ __forceinline__ int pair(int) const { return 0; }
  __device__ __forceinline__ int one(int p) const {
    const int u = lt >> 3, v = lt & 7, d = p / 6;
    switch (p % 6) {
      case 0: return at(-1 - d, u, v);
      case 1: return at(8 + d, u, v);
      case 2: return at(u, -1 - d, v);
      case 3: return at(u, 8 + d, v);
      case 4: return at(u, v, -1 - d);
      default: return at(u, v, 8 + d);
    }
  }
};
// Stars staged by bulk copies: the centre, then the six faces densely one after the other (k and j
// faces 64 R values each, i faces 64 rows of IW values).  The faces are taken as whole aligned
// pairs in order, except the i faces of radius 1, whose rows hold a value that the stencil does not
// read.
template <int R, int IW>
struct FxDense {
  static constexpr int NP = R == 1 ? 2 : 3 * R, NS = R == 1 ? 2 : 0;
  static_assert(R == 1 ? IW == 2 : IW == R, "i-face rows of whole 16-byte units");
  int lt;
  __device__ __forceinline__ int block(int k, int j, int i) const { return (k * 8 + j) * 8 + i; }
  __device__ __forceinline__ bool has(int) const { return true; }
  __device__ __forceinline__ int pair(int p) const { return 512 + 2 * (64 * p + lt); }
  __device__ __forceinline__ int one(int p) const { return 768 + 128 * p + 2 * lt + (p ? 0 : 1); }
};
// The same values in a tile of their own with one row and plane stride for all of them, so that
// a thread's taps lie at constant distances.  R = 2: rows of 12 (columns -2 .. 9); rows two apart are
// 192 bytes apart, so a quarter warp's pair loads from two such rows use all banks.  R = 1: rows of 10
// (columns -1 .. 8; the last one where the next row's column -2 would be), rows four apart likewise.
template <int R>
struct FxTile {
  static_assert(R <= 2, "two columns either side");
  static constexpr int EJ = 8 + 2 * R, SJ = R == 1 ? 10 : 12, SK = EJ * SJ, SIZE = ((8 + 2 * R) * SK + 15) / 16 * 16;
  // row of a thread's pair: two rows of a quarter warp in different banks
  static __device__ __forceinline__ int row(int lt) {
    const int q = (lt >> 2) & 7;
    return R == 1 ? (q >> 1) | ((q & 1) << 2) : (q & 4) | ((q & 1) << 1) | ((q >> 1) & 1);
  }
  int pk, pj, pi;  // positions of this thread's k-, j- and i-face values (low side)
  static __device__ __forceinline__ int at(int k, int j, int i) { return (k + R) * SK + (j + R) * SJ + i + 2; }
  __device__ __forceinline__ FxTile(int lt) {
    const int r = lt >> 2, i = 2 * (lt & 3);  // row of four pairs in the dense faces
    if constexpr (R == 1) {
      const int u = r & 7, hi = (r >> 3) * 9;  // 8 rows of the low face, 8 of the high one
      pk = at(hi - 1, u, i);
      pj = at(u, hi - 1, i);
      pi = at(lt >> 3, lt & 7, -1);
    } else {
      pk = at((r >> 3) - 2, r & 7, i);
      pj = at(r >> 1, (r & 1) - 2, i);
      pi = at(lt >> 3, lt & 7, -2);
    }
  }
  __device__ __forceinline__ int block(int k, int j, int i) const { return at(k, j, i); }
  __device__ __forceinline__ bool has(int) const { return true; }
  __device__ __forceinline__ int pair(int p) const {
    if constexpr (R == 1) return p ? pj : pk;
    return p < 2 ? pk + 10 * SK * p : p < 4 ? pj + 10 * SJ * (p - 2) : pi + 10 * (p - 4);
  }
  __device__ __forceinline__ int one(int p) const { return pi + 9 * p; }
  // position of this thread's (j, i) column at plane k of its four (k in -R .. 3 + R), its warp w
  __device__ __forceinline__ static void columns(int j, int i, int w, int (&c)[3]) {
    c[0] = c[1] = c[2] = at(4 * w, j, i);
  }
};
// Radius 4: planes 0 .. 7 of 16 rows (-4 .. 11) of 18 (columns -4 .. 11); the four corners of a plane,
// which a star does not read, hold the quarters of a k-face plane: plane -4 + q in plane q, plane 8 + q
// in plane 4 + q.  18 KB instead of 32 for the whole box.
template <>
struct FxTile<4> {
  static constexpr int SJ = 18, SK = 16 * SJ, SIZE = 8 * SK;
  static __device__ __forceinline__ int row(int lt) {
    const int q = (lt >> 2) & 7;
    return (q >> 1) | ((q & 1) << 2);
  }
  int pk, pj, pi;
  static __device__ __forceinline__ int at(int k, int j, int i) { return k * SK + (j + 4) * SJ + i + 4; }
  // row j or column i of a k-face plane, in the corners
  static __device__ __forceinline__ int corner(int x) { return x < 4 ? x - 4 : x + 4; }
  __device__ __forceinline__ FxTile(int lt) {
    const int i = 2 * (lt & 3);
    pk = at(lt >> 5, corner((lt >> 2) & 7), corner(i));
    pj = at(lt >> 4, ((lt >> 2) & 3) - 4, i);
    pi = at(lt >> 4, (lt >> 1) & 7, 2 * (lt & 1) - 4);
  }
  __device__ __forceinline__ int block(int k, int j, int i) const { return at(k, j, i); }
  __device__ __forceinline__ bool has(int) const { return true; }
  __device__ __forceinline__ int pair(int p) const {
    return p < 4 ? pk + 2 * SK * p : p < 8 ? pj + 4 * SK * (p & 1) + (p >= 6 ? 12 * SJ : 0)
                                           : pi + 4 * SK * (p & 1) + (p >= 10 ? 12 : 0);
  }
  __device__ __forceinline__ int one(int) const { return 0; }
  __device__ __forceinline__ static void columns(int j, int i, int w, int (&c)[3]) {
    const int centre = at(0, j, i), face = at(0, corner(j), corner(i));
    c[0] = (w ? centre : face) + 4 * SK;  // planes -4 .. -1 of the thread
    c[1] = centre + 4 * w * SK;           // 0 .. 3
    c[2] = w ? face : centre;             // 4 .. 7
  }
};

// Cubes: the (8 + 2R)^3 box without its centre, value n of the list to thread n mod 64; the
// positions are found once per thread (two to a register).
template <int R, class At>
struct FxBox {
  static constexpr int E = 8 + 2 * R, N = E * E * E - 512, PT = (N + 63) / 64;
  static constexpr int NP = 0, NS = PT;
  unsigned pos[(PT + 1) / 2];
  int lt;
  At at;
  __device__ __forceinline__ int block(int k, int j, int i) const { return at(k, j, i); }
  __device__ __forceinline__ FxBox(int lt_, At at_) : lt(lt_), at(at_) {
#pragma unroll
    for (int p = 0; p < (PT + 1) / 2; ++p) pos[p] = 0u;
#pragma unroll
    for (int p = 0; p < PT; ++p) {
      int n = p * 64 + lt, k, j, i;
      if (n >= N) n = 0;
      if (n < 2 * R * E * E) {  // whole planes below and above
        k = n / (E * E);
        j = n / E % E;
        i = n % E;
        k = k < R ? k - R : k - R + 8;
        j -= R;
        i -= R;
      } else if (n < 2 * R * E * E + 16 * R * E) {  // rows beside the centre planes
        n -= 2 * R * E * E;
        k = n / (2 * R * E);
        j = n / E % (2 * R);
        i = n % E - R;
        j = j < R ? j - R : j - R + 8;
      } else {  // the ends of the centre rows
        n -= 2 * R * E * E + 16 * R * E;
        k = n / (16 * R);
        j = n / (2 * R) % 8;
        i = n % (2 * R);
        i = i < R ? i - R : i - R + 8;
      }
      pos[p >> 1] |= (unsigned)at(k, j, i) << (16 * (p & 1));
    }
  }
  __device__ __forceinline__ bool has(int p) const { return (p + 1) * 64 <= N || p * 64 + lt < N; }
  __device__ __forceinline__ int pair(int) const { return 0; }
  __device__ __forceinline__ int one(int p) const { return (pos[p >> 1] >> (16 * (p & 1))) & 0xFFFFu; }
};

// Four planes of a column pair (j, i0), (j, i0 + 1) of a converted brick under a star: eight outputs
// per thread.  l2(k, dj, m): the aligned pair at the thread's plane k (-R .. 3 + R), row j + dj, columns
// i0 + 2m; l1(k, di): the value at column i0 + di (radius 1: di = -1, 2); st(k, y0, y1) stores.  With
// two adjacent points per thread a pair load serves both and the i taps of one are partly the
// other's: for radius 4, 60 16-byte loads instead of 144 8-byte ones.  SUM: the coefficients of
// each distance are one class (ring symmetric), whose six values are added first: |sum| < 6 2^60.
template <int R, bool SUM, class L2, class L1, class ST>
__device__ __forceinline__ void fx_star_pairs(L2 l2, L1 l1, ST st, const FxTab &tab, int scale) {
  double2 w[4 + 2 * R];
#pragma unroll
  for (int q = 0; q < 4 + 2 * R; ++q) w[q] = l2(q - R, 0, 0);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    double x[2 + 2 * R];  // columns i0 - R .. i0 + 1 + R
    x[R] = w[k + R].x;
    x[R + 1] = w[k + R].y;
    if constexpr (R == 1) {
      x[0] = l1(k, -1);
      x[3] = l1(k, 2);
    } else {
#pragma unroll
      for (int m = 1; m <= R / 2; ++m) {
        const double2 lo = l2(k, 0, -m), hi = l2(k, 0, m);
        x[R - 2 * m] = lo.x;
        x[R - 2 * m + 1] = lo.y;
        x[R + 2 * m] = hi.x;
        x[R + 2 * m + 1] = hi.y;
      }
    }
    FxAcc<R == 1> acc[2];
    auto whole = [](double v) { return __double_as_longlong(v); };
    auto half = [](double v) { return make_int2(__double2loint(v), __double2hiint(v)); };
#pragma unroll
    for (int o = 0; o < 2; ++o) acc[o].first(tab, 0, SUM ? fx_split(whole(x[R + o])) : half(x[R + o]));
#pragma unroll
    for (int d = 1; d <= R; ++d) {
      const double2 jp = l2(k, d, 0), jm = l2(k, -d, 0);
#pragma unroll
      for (int o = 0; o < 2; ++o) {
        const double a = x[R + o + d], b = x[R + o - d], c = o ? jp.y : jp.x, e = o ? jm.y : jm.x;
        const double f = o ? w[k + R + d].y : w[k + R + d].x, g = o ? w[k + R - d].y : w[k + R - d].x;
        if constexpr (SUM) {
          long long y = whole(a) + whole(b) + whole(c);  // three at a time: one carry chain each
          y = y + whole(e) + whole(f);
          acc[o].add(tab, d, fx_split(y + whole(g)));
        } else {
          const int t = 1 + 6 * (d - 1);
          acc[o].add(tab, t + 0, half(a));
          acc[o].add(tab, t + 1, half(b));
          acc[o].add(tab, t + 2, half(c));
          acc[o].add(tab, t + 3, half(e));
          acc[o].add(tab, t + 4, half(f));
          acc[o].add(tab, t + 5, half(g));
        }
      }
    }
    st(k, fx_result(acc[0].sum(), scale), fx_result(acc[1].sum(), scale));
  }
}

// Four planes of a column pair under a radius-1 cube: l2(k, dj): the pair at the thread's plane k
// (-1 .. 4), row j + dj; l1(k, dj, di): the value at column i0 + di (-1, 2).  A row's four values serve
// up to 18 products: 18 16-byte and 36 8-byte loads for eight points (216 for one tap at a time).
template <class L2, class L1, class ST>
__device__ __forceinline__ void fx_cube_pairs(L2 l2, L1 l1, ST st, const FxTab &tab, int scale) {
  auto half = [](double v) { return make_int2(__double2loint(v), __double2hiint(v)); };
  FxAcc<false> acc[4][2];
#pragma unroll
  for (int p = 0; p < 6; ++p) {
#pragma unroll
    for (int dj = -1; dj <= 1; ++dj) {
      const double2 c = l2(p - 1, dj);
      const int2 x[4] = {half(l1(p - 1, dj, -1)), half(c.x), half(c.y), half(l1(p - 1, dj, 2))};
#pragma unroll
      for (int k = p - 2; k <= p; ++k)
        if (k >= 0 && k < 4)
#pragma unroll
          for (int di = 0; di < 3; ++di)
#pragma unroll
            for (int o = 0; o < 2; ++o) {
              const int t = ((p - k) * 3 + dj + 1) * 3 + di;
              if (t == 0) acc[k][o].first(tab, t, x[o + di]);
              else acc[k][o].add(tab, t, x[o + di]);
            }
    }
    if (p >= 2) st(p - 2, fx_result(acc[p - 2][0].sum(), scale), fx_result(acc[p - 2][1].sum(), scale));
  }
}

// One row (k, j) of a converted brick under the 125-point cube with one coefficient per sorted
// distance (ten classes).  l2(dk, dj, c): the row's columns 2c - 2, 2c - 1 (c = 0 .. 5) at plane k + dk, row
// j + dj.  Column by column the 25 values around the row are added to six sums q (k and j distances
// sorted: 00, 01, 11, 02, 12, 22); of five columns' sums a point's ten class sums take 20 more additions
// (integer, 64 bits, two instructions each and three operands where they chain) and 30 products,
// where products per column would take 54 per point.  st(c, y0, y1) stores columns 2c, 2c + 1.
template <class L2, class ST>
__device__ __forceinline__ void fx_cube125_row(L2 l2, ST st, const FxTab &tab, int scale) {
  auto whole = [](double v) { return __double_as_longlong(v); };
  long long q[6][6];  // [class][column]: the newest pair of columns at 4, 5
#pragma unroll
  for (int c = 0; c < 6; ++c) {
    long long s[3][3][2];  // [|dk|][|dj|][column]
#pragma unroll
    for (int d = 0; d < 5; ++d) {
      const int dk = d == 0 ? 0 : d == 1 ? -1 : d == 2 ? 1 : d == 3 ? -2 : 2, a = (d + 1) / 2;
      double2 x[5];
#pragma unroll
      for (int r = 0; r < 5; ++r) x[r] = l2(dk, r - 2, c);
#pragma unroll
      for (int o = 0; o < 2; ++o) {
        auto v = [&](int r) { return whole(o ? x[r].y : x[r].x); };
        if (d == 0 || dk < 0) {
          s[a][0][o] = v(2);
          s[a][1][o] = v(1) + v(3);
          s[a][2][o] = v(0) + v(4);
        } else {
          s[a][0][o] += v(2);
          s[a][1][o] = s[a][1][o] + v(1) + v(3);
          s[a][2][o] = s[a][2][o] + v(0) + v(4);
        }
      }
    }
#pragma unroll
    for (int m = 0; m < 6; ++m)
#pragma unroll
      for (int h = 0; h < 4; ++h) q[m][h] = q[m][h + 2];
#pragma unroll
    for (int o = 0; o < 2; ++o) {
      q[0][4 + o] = s[0][0][o];
      q[1][4 + o] = s[0][1][o] + s[1][0][o];
      q[2][4 + o] = s[1][1][o];
      q[3][4 + o] = s[0][2][o] + s[2][0][o];
      q[4][4 + o] = s[1][2][o] + s[2][1][o];
      q[5][4 + o] = s[2][2][o];
    }
    if (c < 2) continue;
    double y[2];
#pragma unroll
    for (int o = 0; o < 2; ++o) {  // output column 2c - 4 + o, its window q[.][o .. o + 4]
      auto t0 = [&](int m) { return q[m][o + 2]; };
      auto t1 = [&](int m) { return q[m][o + 1] + q[m][o + 3]; };
      auto t2 = [&](int m) { return q[m][o] + q[m][o + 4]; };
      FxAcc<false> acc;
      acc.first(tab, 0, fx_split(t0(0)));
      acc.add(tab, 1, fx_split(t1(0) + t0(1)));
      acc.add(tab, 2, fx_split(t2(0) + t0(3)));
      acc.add(tab, 3, fx_split(t1(1) + t0(2)));
      acc.add(tab, 4, fx_split(t2(1) + t0(4) + t1(3)));
      acc.add(tab, 5, fx_split(t2(3) + t0(5)));
      acc.add(tab, 6, fx_split(t1(2)));
      acc.add(tab, 7, fx_split(t2(2) + t1(4)));
      acc.add(tab, 8, fx_split(t2(4) + t1(5)));
      acc.add(tab, 9, fx_split(t2(5)));
      y[o] = fx_result(acc.sum(), scale);
    }
    st(c - 2, y[0], y[1]);
  }
}

// Scan, agree, convert: true when the brick's values are now integers in `to`, false when the brick
// is to be computed in FP64 (nothing was written).  Called by all 64 threads of a brick; on: the
// brick is to be computed (the same for all of them unless some thread gives up: stop, whose answer
// every thread gets in `stopped`).  slot: int2[2] of this brick and of this call's parity (a later
// call on the same slot follows a barrier of all 64 threads).  brick: 0 or 1, its place in the
// CTA.  When a thread passes the first barrier the brick's threads are done with what they read from
// `to` before the call.
// taken(): called once the values are in registers for good (HOLD) and `from` is not read again.
template <class Share, class Taken>
__device__ __forceinline__ bool fx_prepare(const Share &sh, const double *from, double *to, const FxTab &tab, int2 *slot,
                                           int brick, int &E, bool on, bool stop, bool &stopped, Taken taken) {
  double v[Share::NV];
  if (on) {
    sh.load(from, v);
    fx_publish(Share::scan(v, tab), slot, sh.lt);
  }
  stopped = fx_bar_or(brick, stop);
  if (stopped || !on) return false;
  const FxScan s = fx_gather(slot);
  E = (int)(s.top >> 20);
  // a star on zeros, or numbers below 2^-1042: where all are +0, so are the sums, on any scale (256^3
  // zeros, us, in FP64 / so: 7-point 197 / 89, 13-point 359 / 104, 25-point 689 / 162; the cubes
  // write their zeros themselves, sweep2_kernel)
  if (Share::STAR && s.top == 0 && tab.zeros) {
    if constexpr (!Share::HOLD) sh.load(from, v);
    bool some = false;
#pragma unroll
    for (int q = 0; q < Share::NV; ++q) some = some || __double_as_longlong(v[q]) != 0;
    if (fx_bar_or(brick, some)) return false;
    E = tab.elo;
  } else if (!fx_ok(tab, s)) {
    return false;
  }
  if constexpr (!Share::HOLD) sh.load(from, v);
  taken();
  sh.convert(to, v, E);
  fx_bar(brick);
  return true;
}

}  // namespace bk
