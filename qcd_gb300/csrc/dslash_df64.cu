// dslash_df64.cu -- the Wilson-TM operator on FP64 fields in float-float
// arithmetic.
//
// GB300 executes FP64 fused multiply-adds at about 1/60 of its FP32 rate
// (measured: 0.60 T DFMA/s against 35 T FFMA/s), so the FP64 operator
// computed natively is bound by the FP64 pipe, not by HBM. This kernel keeps
// FP64 storage for the spinors (read and written as doubles) and computes on
// the FP32 pipes with unevaluated float pairs (hi + lo, ~47 significant bits):
//   * products: Dekker's exact product of the high words via FMA plus the two
//     cross terms (T. J. Dekker, Numer. Math. 18 (1971) 224);
//   * sums: Knuth's TwoSum (TAOCP vol. 2) into lazy accumulators (s, e) whose
//     error word collects the rounding errors in FP32; an accumulator is
//     renormalised (Fast2Sum) only when its value is consumed.
// Every operation uses the explicitly rounded intrinsics, so the compiler can
// neither contract nor reorder them. The double -> float-pair splits of the
// spinors (four per hop and thread) and the widenings of the results use
// integer bit operations, because the hardware conversions run on the FP64
// pipe. The links come from a copy of the gauge field stored as float pairs,
// made once per field, with the boundary phase e^{i th/L} multiplied into the
// links of twisted directions (U' h for the forward hop,
// U'^+ h = e^{-i th/L} U^+ h for the backward one, as qcd_wilson.c applies it).
// The result differs from FP64 by a few 2^-46 relative, within the 1e-13
// per-site parity bar. Spinor values must lie in [2^-74, 2^127) in magnitude
// for the fast conversion; other values take an exact slower path, and
// doubles below 2^-1022 (denormals) count as zero.
#include "dslash_args.h"

namespace qg {

using namespace qgd;

struct F2 {  // h + l
  float h, l;
};

// double -> float pair, any value
__device__ F2 split_any(double d)
{
  const unsigned e = ((unsigned)__double2hiint(d) >> 20) & 0x7ffu;
  F2 r;
  if (e == 0u) {
    r.h = __uint_as_float((unsigned)__double2hiint(d) & 0x80000000u);
    r.l = 0.0f;
  } else {
    r.h = __double2float_rn(d);
    r.l = __double2float_rn(__dsub_rn(d, (double)r.h));
  }
  return r;
}

// In range (|d| in [2^-74, 2^127)) with integer bit operations: hi takes the
// leading 24 significand bits and lo the next 23 (both truncated; the pair
// keeps 47 bits, relative error below 2^-46).
__device__ __forceinline__ F2 split_d(double d)
{
  const unsigned lo32 = (unsigned)__double2loint(d), hi32 = (unsigned)__double2hiint(d);
  F2 r;
  // (hi32:lo32) << 3 holds the exponent's low 9 bits and the top 23
  // significand bits in float position; e - 896 = (e mod 512) - 384 here,
  // so one subtraction rebiases the exponent, and the sign goes back in
  const unsigned hb = (__funnelshift_l(lo32, hi32, 3) - (384u << 23)) | (hi32 & 0x80000000u);
  r.h = __uint_as_float(hb);
  // the 23 bits below hi as an exact integer-valued float, scaled by
  // 2^(e - 1069) with hi's sign: hi's sign and exponent field less 46
  const float f1 = __fsub_rn(__uint_as_float(0x4B000000u | ((lo32 >> 6) & 0x7fffffu)), 8388608.0f);
  r.l = __fmul_rn(f1, __uint_as_float((hb & 0xff800000u) - (46u << 23)));
  return r;
}

struct F2Quad {
  F2 ar, ai, br, bi;
};
// a zero or a value out of range among the four: out of line
__device__ __noinline__ F2Quad split_slow(double2 a, double2 b)
{
  auto one = [](double d) {
    const unsigned e = ((unsigned)__double2hiint(d) >> 20) & 0x7ffu;
    return e - 949u <= 201u ? split_d(d) : split_any(d);
  };
  return F2Quad{one(a.x), one(a.y), one(b.x), one(b.y)};
}
__device__ __forceinline__ bool is_zero(double2 a)
{
  return (((__double2hiint(a.x) | __double2hiint(a.y)) & 0x7fffffff) | __double2loint(a.x) | __double2loint(a.y)) == 0;
}
// exponent distance above 2^-74 (in units of the exponent field)
__device__ __forceinline__ unsigned split_range(double d)
{
  return ((unsigned)__double2hiint(d) & 0x7ff00000u) - (949u << 20);
}

// h + l -> double: two exact widenings and one FP64 add, rounded to nearest
__device__ __forceinline__ double join_d(F2 x) { return __dadd_rn((double)x.h, (double)x.l); }
// the same with the widenings as integer operations (the conversions run on
// the FP64 pipe), for normal h and l
__device__ __forceinline__ double widen(float f)
{
  const unsigned b = __float_as_uint(f);
  return __hiloint2double((int)((((b & 0x7fffffffu) >> 3) + 0x38000000u) | (b & 0x80000000u)), (int)(b << 29));
}
__device__ __forceinline__ double join_fast(float h, float l) { return __dadd_rn(widen(h), widen(l)); }
// below 0x7f000000 for normal f
__device__ __forceinline__ unsigned widen_range(float f) { return (__float_as_uint(f) & 0x7fffffffu) - 0x00800000u; }

// Two pairs at once, in the halves of sm_103a's packed FP32 operations (one
// issue slot for two results; each half rounds as the scalar operation does).
struct F2x2 {
  float2 h, l;
};
struct FAx2 {  // accumulator: values s + e, not normalised
  float2 s, e;
};
struct CAx2 {
  FAx2 re, im;
};
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
// a - b: a multiply-add by -1 rounds the same, and a negated operand of a
// packed add costs instructions of its own (24^3 x 48: 0.336 against 0.306 ms)
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }
__device__ __forceinline__ float2 dup2(float a) { return make_float2(a, a); }
__device__ __forceinline__ void two_sum2(float2 a, float2 b, float2 &s, float2 &q)
{
  s = __fadd2_rn(a, b);
  const float2 bb = sub2(s, a);
  q = __fadd2_rn(sub2(a, sub2(s, bb)), sub2(b, bb));
}
// acc += a * b; nah = -a.h (t is the product's error, negated: a negated
// operand of a packed operation costs an instruction of its own)
__device__ __forceinline__ void mac2(FAx2 &acc, F2x2 a, float2 nah, F2x2 b)
{
  const float2 p = __fmul2_rn(a.h, b.h);
  const float2 t = __ffma2_rn(nah, b.h, p);
  float2 s, q;
  two_sum2(acc.s, p, s, q);
  float2 e = __fadd2_rn(acc.e, sub2(q, t));
  e = __ffma2_rn(a.h, b.l, e);
  acc.e = __ffma2_rn(a.l, b.h, e);
  acc.s = s;
}
// acc = a * b into an empty accumulator: no error-free sum needed
__device__ __forceinline__ FAx2 mac02(F2x2 a, float2 nah, F2x2 b)
{
  const float2 p = __fmul2_rn(a.h, b.h);
  float2 e = __ffma2_rn(a.h, b.h, __fmul2_rn(nah, b.h));
  e = __ffma2_rn(a.h, b.l, e);
  return FAx2{p, __ffma2_rn(a.l, b.h, e)};
}
// acc += x for an unnormalised x
__device__ __forceinline__ void acc_add2(FAx2 &acc, FAx2 x)
{
  float2 s, q;
  two_sum2(acc.s, x.s, s, q);
  acc.e = __fadd2_rn(acc.e, __fadd2_rn(q, x.e));
  acc.s = s;
}
// (a, b) and their imaginary parts as pairs: one range test for the four values
__device__ __forceinline__ void split_pair(double2 a, double2 b, F2x2 &re, F2x2 &im)
{
  F2Quad q;
  if (max(max(split_range(a.x), split_range(a.y)), max(split_range(b.x), split_range(b.y))) <= (201u << 20))
    q = F2Quad{split_d(a.x), split_d(a.y), split_d(b.x), split_d(b.y)};
  else if (is_zero(a) && is_zero(b))  // empty sites of sources and first iterates
    q = F2Quad{};
  else
    q = split_slow(a, b);
  re = F2x2{make_float2(q.ar.h, q.br.h), make_float2(q.ar.l, q.br.l)};
  im = F2x2{make_float2(q.ai.h, q.bi.h), make_float2(q.ai.l, q.bi.l)};
}
// re + i im of both halves
__device__ __forceinline__ void join_pair(F2x2 re, F2x2 im, double2 &a, double2 &b)
{
  const unsigned m0 = max(max(widen_range(re.h.x), widen_range(re.l.x)), max(widen_range(im.h.x), widen_range(im.l.x)));
  const unsigned m1 = max(max(widen_range(re.h.y), widen_range(re.l.y)), max(widen_range(im.h.y), widen_range(im.l.y)));
  if (max(m0, m1) < 0x7f000000u) {
    a = make_double2(join_fast(re.h.x, re.l.x), join_fast(im.h.x, im.l.x));
    b = make_double2(join_fast(re.h.y, re.l.y), join_fast(im.h.y, im.l.y));
  } else {
    a = make_double2(join_d(F2{re.h.x, re.l.x}), join_d(F2{im.h.x, im.l.x}));
    b = make_double2(join_d(F2{re.h.y, re.l.y}), join_d(F2{im.h.y, im.l.y}));
  }
}
// the two halves exchanged
__device__ __forceinline__ FAx2 flip2(FAx2 v)
{
  return FAx2{make_float2(v.s.y, v.s.x), make_float2(v.e.y, v.e.x)};
}

// Thread layout: a block of three warps covers 32 sites; warp w owns colour
// row i = w and the four accumulators (spins 0..3) of that colour. Per hop
// each warp projects the neighbour spinor of its colour, the three warps share
// the half spinors through shared memory, and each multiplies its link row.
// With S the projector sign, (1 + S g_mu) in the chiral basis is
//   h0 = p0 + c0 p_b0, h1 = p1 + c1 p_b1            (upper half)
//   b0 = 2 (mu 0,3) or 3 (mu 1,2), b1 = 5 - b0, c = +-1 (mu even) or +-i (odd)
//   c0 = -S ; c1 = -S (mu 0,1) or +S (mu 2,3)
// and the lower half rebuilt from v = U h:
//   r2 = cA v_jA, r3 = cB v_jB ; jA = 1 for mu 1,2 else 0, jB = 1 - jA
//   cA = -S (mu 0) else +S ; cB = +S (mu 1) else -S ; times i for odd mu
// (qcd_wilson.h:17-387). The directions run 0, 3, 1, 2: the lower pair is
// accumulated as (spin 2, spin 3) for the first two and as (3, 2) for the
// others, so that no hop exchanges the halves of a pair.
//
// What bounds it: instruction issue and latency (about half of the issue slots
// are taken), the FP64 pipe next. So the two spins of a half spinor are the
// two halves of packed FP32 operations, which halves the issue slots of the
// products and sums; a link entry is broadcast to both. The FP64 pipe does
// only the spin projections (four adds per hop and warp: half the conversions
// of splitting all components first) and one add per joined result. The two
// hops of a direction are one loop body: four bodies of code stay in the
// instruction cache, eight did not. Each thread's four spinor components of
// the next hop are copied into shared memory with cp.async while the current
// hop computes, so the loads hold no registers.
// Measured on GB300 at 24^3 x 48, ms per apply: 0.366 with scalar operations
// (298 M warp instructions), nine warps a block and eight unrolled hops; packed 0.350
// (214 M); one body per direction 0.330; blocks of three warps 0.306; widening
// by integer operations in the join 0.302; one range test per four splits and
// per eight widenings, no negated packed operands and one barrier per hop
// instead of two 0.275 (209 M, 61 % of the issue slots, FP64 pipe 47 %). One
// thread per site (no exchange, 184 M warp instructions) holds 15 warps per SM
// at 128 registers and ran at 0.402.
constexpr int kFFSites = 32;
constexpr int kFFThreads = 3 * kFFSites;
constexpr int kFFMinBlocks = 7;  // resident blocks per SM the registers are sized for (8: 0.285, 9: 0.277, 10: 0.301 ms)

// site of output index e; EO: the site of parity eo_par among full indices
// 2e, 2e + 1 (even t extent)
template <bool EO>
__device__ __forceinline__ int ff_site(const DArgs &a, int e, int c[4])
{
  if (EO) {
    coords(a.geo, 2 * e, c);
    const int b = (a.eo_par ^ c[1] ^ c[2] ^ c[3]) & 1;
    c[0] += b;
    return 2 * e + b;
  }
  coords(a.geo, e, c);
  return e;
}

// neighbour of x across direction mu (backwards if back), periodic
__device__ __forceinline__ int ff_nb(const DArgs &a, int x, const int c[4], int mu, bool back)
{
  const int cm = mu == 0 ? c[0] : mu == 1 ? c[1] : mu == 2 ? c[2] : c[3];
  const int Lm = a.geo.L[mu], st = a.geo.st[mu];
  if (back) return cm == 0 ? x + (Lm - 1) * st : x - st;
  return cm == Lm - 1 ? x - (Lm - 1) * st : x + st;
}

// sign flip by integer operation (keeps the FP64 pipe for arithmetic)
__device__ __forceinline__ double dflip(double v, bool ng)
{
  return __longlong_as_double(__double_as_longlong(v) ^ ((long long)ng << 63));
}
// z -> (i z if ifl) then negated if ng
__device__ __forceinline__ double2 dcoef(double2 z, bool ifl, bool ng)
{
  return make_double2(dflip(ifl ? z.y : z.x, ng ^ ifl), dflip(ifl ? z.x : z.y, ng));
}
__device__ __forceinline__ double2 dadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }

// 16-byte asynchronous copy global -> shared (cached in L1: neighbour
// spinors are read by eight sites), and its group fences
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem)
{
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait()
{
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ F2x2 fin2(FAx2 a)
{
  const float2 s = __fadd2_rn(a.s, a.e);
  return F2x2{s, sub2(a.e, sub2(s, a.s))};
}
__device__ __forceinline__ FAx2 mul2(FAx2 a, float2 b) { return FAx2{__fmul2_rn(a.s, b), __fmul2_rn(a.e, b)}; }
__device__ __forceinline__ F2x2 neg2(F2x2 a) { return F2x2{neg2(a.h), neg2(a.l)}; }

// out = epilogue of the accumulated hopping term, for the spin pair (2 P, 2 P + 1)
template <int P, bool EO, bool AOS, bool SUMS>
__device__ __forceinline__ void ff_store(const DArgs &a, int x, int e, int i, CAx2 acc, bool act, double &n2)
{
  const F2x2 mp4{dup2(a.mp4_h), dup2(a.mp4_l)};
  const F2x2 tp{dup2(P ? -a.tm_h : a.tm_h), dup2(P ? -a.tm_l : a.tm_l)};
  const int k0 = 6 * P + i, k1 = k0 + 3;
  F2x2 hr = fin2(acc.re), hi = fin2(acc.im), dr, di;
  if (EO) {
    if (a.ainv) {  // (ai_r + i ai_i g5) H in
      const F2x2 air{dup2(a.ai_r_h), dup2(a.ai_r_l)};
      const F2x2 gi{dup2(P ? -a.ai_i_h : a.ai_i_h), dup2(P ? -a.ai_i_l : a.ai_i_l)};
      FAx2 re = mac02(air, neg2(air.h), hr), im = mac02(air, neg2(air.h), hi);
      mac2(re, neg2(gi), gi.h, hi);
      mac2(im, gi, neg2(gi.h), hr);
      hr = fin2(re);
      hi = fin2(im);
    }
    const F2x2 ch{dup2(a.ch_h), dup2(a.ch_l)};
    FAx2 re = mac02(ch, neg2(ch.h), hr), im = mac02(ch, neg2(ch.h), hi);
    if (a.zmode) {
      const double2 *z = (const double2 *)a.z;
      const double2 z0 = __ldg(z + (int64_t)k0 * a.stride + e), z1 = __ldg(z + (int64_t)k1 * a.stride + e);
      F2x2 zr, zi;
      split_pair(z0, z1, zr, zi);
      if (a.zmode >= 2) {  // + (m+4) z + i tm g5 z
        mac2(re, mp4, neg2(mp4.h), zr);
        mac2(re, neg2(tp), tp.h, zi);
        mac2(im, mp4, neg2(mp4.h), zi);
        mac2(im, tp, neg2(tp.h), zr);
      } else {
        acc_add2(re, FAx2{zr.h, zr.l});
        acc_add2(im, FAx2{zi.h, zi.l});
      }
      if (a.zmode == 3) {
        const double2 *w = (const double2 *)a.w;
        F2x2 wr, wi;
        split_pair(__ldg(w + (int64_t)k0 * a.stride + e), __ldg(w + (int64_t)k1 * a.stride + e), wr, wi);
        acc_add2(re, FAx2{wr.h, wr.l});
        acc_add2(im, FAx2{wi.h, wi.l});
      }
    }
    dr = fin2(re);
    di = fin2(im);
  } else {
    // (m+4) psi + i tm g5 psi - acc / 2
    const double2 *sp = (const double2 *)a.in;
    const double2 s0 = __ldg(AOS ? sp + (int64_t)x * 12 + k0 : sp + (int64_t)k0 * a.stride + x);
    const double2 s1 = __ldg(AOS ? sp + (int64_t)x * 12 + k1 : sp + (int64_t)k1 * a.stride + x);
    F2x2 sr, si;
    split_pair(s0, s1, sr, si);
    FAx2 re = mul2(FAx2{hr.h, hr.l}, dup2(-0.5f)), im = mul2(FAx2{hi.h, hi.l}, dup2(-0.5f));
    mac2(re, mp4, neg2(mp4.h), sr);
    mac2(re, neg2(tp), tp.h, si);
    mac2(im, mp4, neg2(mp4.h), si);
    mac2(im, tp, neg2(tp.h), sr);
    dr = fin2(re);
    di = fin2(im);
    if (a.op_q) {  // i g5: spins 0, 1 times i, spins 2, 3 times -i
      const F2x2 t = dr;
      dr = P ? di : neg2(di);
      di = P ? neg2(t) : t;
    }
  }
  double2 v0, v1;
  join_pair(dr, di, v0, v1);
  if (act) {
    double2 *out = (double2 *)a.out;
    const int o = EO ? e : x;
    out[AOS ? (int64_t)o * 12 + k0 : (int64_t)k0 * a.stride + o] = v0;
    out[AOS ? (int64_t)o * 12 + k1 : (int64_t)k1 * a.stride + o] = v1;
    if (SUMS) n2 += v0.x * v0.x + v0.y * v0.y + v1.x * v1.x + v1.y * v1.y;
  }
}

// the half spinors the three warps exchange, double-buffered by hop:
// [hop & 1][colour][re, im][site], a pair's high words, then its low words
typedef float4 FFShare[2][3][2][kFFSites];

// the two hops of direction MU for one site and colour row col. The staged
// components of hop (MU, back) are in stage `back`; the next hop's are
// requested first (NEXT: the direction after MU, 4 when MU is the last). BAR:
// the barrier of the three warps.
template <int MU, int NEXT, int BAR, bool DAG, bool EO, bool AOS>
__device__ __forceinline__ void ff_hops(const DArgs &a, int col, int lane, int x, const int c[4], FFShare &hs,
                                        double2 *stage, CAx2 &up, CAx2 &lo)
{
  const double2 *sp = (const double2 *)a.in;
  const float4 *gf = (const float4 *)a.gauge + (int64_t)MU * 9 * a.gstride;
  constexpr bool odd = MU & 1;
  constexpr int NB0 = (NEXT == 0 || NEXT == 3) ? 2 : 3, B0 = (MU == 0 || MU == 3) ? 2 : 3;
#pragma unroll 1
  for (int back = 0; back < 2; back++) {
    if (NEXT < 4 || back == 0) {
      const int yn = back ? ff_nb(a, x, c, NEXT & 3, false) : ff_nb(a, x, c, MU, true), ys = EO ? (yn >> 1) : yn;
      const int b0 = back ? NB0 : B0;
      double2 *to = stage + (back ^ 1) * 4 * kFFThreads;
      const int comp[4] = {col, 3 + col, 3 * b0 + col, 3 * (5 - b0) + col};
#pragma unroll
      for (int i = 0; i < 4; i++)
        cp_async16(to + i * kFFThreads, AOS ? sp + (int64_t)ys * 12 + comp[i] : sp + (int64_t)comp[i] * a.stride + ys);
      cp_async_commit();
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    // projector sign S > 0: forward for D^+, backward for D
    const bool pos = (back != 0) != DAG;
    const bool neg0 = pos, neg1 = MU < 2 ? pos : !pos;
    const double2 *b = stage + back * 4 * kFFThreads;  // this thread's own copies
    {
      const double2 d0 = dadd(b[0], dcoef(b[2 * kFFThreads], odd, neg0));
      const double2 d1 = dadd(b[kFFThreads], dcoef(b[3 * kFFThreads], odd, neg1));
      F2x2 r, i;
      split_pair(d0, d1, r, i);
      hs[back][col][0][lane] = make_float4(r.h.x, r.h.y, r.l.x, r.l.y);
      hs[back][col][1][lane] = make_float4(i.h.x, i.h.y, i.l.x, i.l.y);
    }
    // forward: U[col][k] at x; backward: conj(U[k][col]) at the neighbour
    const int lx = back ? ff_nb(a, x, c, MU, true) : x;
    const int64_t si = back ? a.gstride : 3 * a.gstride, sk = back ? 3 * a.gstride : a.gstride;
    const unsigned cj = back ? 0x80000000u : 0u;
    float4 wl[3];
#pragma unroll
    for (int k = 0; k < 3; k++) wl[k] = __ldg(gf + lx + col * si + k * sk);
    asm volatile("bar.sync %0, %1;" ::"n"(BAR), "n"(kFFThreads) : "memory");
    CAx2 u;  // U h for the two half-spinor components
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const float4 gr = hs[back][k][0][lane], gi = hs[back][k][1][lane];
      const F2x2 hr{make_float2(gr.x, gr.y), make_float2(gr.z, gr.w)}, hi{make_float2(gi.x, gi.y), make_float2(gi.z, gi.w)};
      float4 w = wl[k];
      w.z = __uint_as_float(__float_as_uint(w.z) ^ cj);
      w.w = __uint_as_float(__float_as_uint(w.w) ^ cj);
      const F2x2 wr{dup2(w.x), dup2(w.y)}, wp{dup2(w.z), dup2(w.w)}, wm{dup2(-w.z), dup2(-w.w)};
      const float2 nwr = dup2(-w.x);
      if (k == 0) {
        u.re = mac02(wr, nwr, hr);
        u.im = mac02(wr, nwr, hi);
      } else {
        mac2(u.re, wr, nwr, hr);
        mac2(u.im, wr, nwr, hi);
      }
      mac2(u.re, wm, wp.h, hi);
      mac2(u.im, wp, wm.h, hr);
    }
    // the products enter the spinor accumulators unnormalised. Lower spins:
    // sign pairs of (spin 2, spin 3) for MU 0, 3; (3, 2) for 1, 2
    const float S = pos ? 1.f : -1.f;
    const float2 sg = MU == 0 ? make_float2(-S, -S) : MU == 1 ? make_float2(S, S) : MU == 2 ? make_float2(-S, S)
                                                                                            : make_float2(S, -S);
    acc_add2(up.re, u.re);
    acc_add2(up.im, u.im);
    if (odd) {  // times i
      acc_add2(lo.re, mul2(u.im, neg2(sg)));
      acc_add2(lo.im, mul2(u.re, sg));
    } else {
      acc_add2(lo.re, mul2(u.re, sg));
      acc_add2(lo.im, mul2(u.im, sg));
    }
  }
}

// the components of the forward hop of direction mu into stage 0
template <bool EO, bool AOS>
__device__ __forceinline__ void ff_first(const DArgs &a, int mu, int col, int x, const int c[4], double2 *stage)
{
  const double2 *sp = (const double2 *)a.in;
  const int y = ff_nb(a, x, c, mu, false), ys = EO ? (y >> 1) : y;
  const int b0 = (mu == 0 || mu == 3) ? 2 : 3;
  const int comp[4] = {col, 3 + col, 3 * b0 + col, 3 * (5 - b0) + col};
#pragma unroll
  for (int i = 0; i < 4; i++)
    cp_async16(stage + i * kFFThreads, AOS ? sp + (int64_t)ys * 12 + comp[i] : sp + (int64_t)comp[i] * a.stride + ys);
  cp_async_commit();
}

// EO: even/odd kernel on half fields (sites of parity a.eo_par; neighbours
// read at (full index) >> 1) with the epilogue ch * [A^{-1}] H in + {z | A z};
// SUMS: with the block sums of |out|^2 (a.partials)
template <bool DAG, bool EO, bool AOS, bool SUMS>
__global__ void __launch_bounds__(kFFThreads, kFFMinBlocks) k_wilson_ff(const DArgs a)
{
  const int block = SUMS ? (int)blockIdx.x : work_block(a.red);
  if (block < 0) return;
  const int lane = threadIdx.x & 31, col = threadIdx.x >> 5;
  const int id = a.x0 + block * kFFSites + lane;  // output index
  const bool act = id < a.V;
  const int e = act ? id : a.V - 1;  // idle lanes repeat the last site
  __shared__ FFShare hs;
  __shared__ double2 staging[2 * 4 * kFFThreads];  // [hop & 1][component][thread]
  int c[4];
  const int x = ff_site<EO>(a, e, c);
  double2 *stage = staging + threadIdx.x;
  ff_first<EO, AOS>(a, 0, col, x, c, stage);
  const float2 z = make_float2(0.f, 0.f);
  CAx2 up{FAx2{z, z}, FAx2{z, z}}, lo = up;
  ff_hops<0, 3, 0, DAG, EO, AOS>(a, col, lane, x, c, hs, stage, up, lo);
  ff_hops<3, 1, 0, DAG, EO, AOS>(a, col, lane, x, c, hs, stage, up, lo);
  lo = CAx2{flip2(lo.re), flip2(lo.im)};
  ff_hops<1, 2, 0, DAG, EO, AOS>(a, col, lane, x, c, hs, stage, up, lo);
  ff_hops<2, 4, 0, DAG, EO, AOS>(a, col, lane, x, c, hs, stage, up, lo);
  lo = CAx2{flip2(lo.re), flip2(lo.im)};
  double n2 = 0.0;
  ff_store<0, EO, AOS, SUMS>(a, x, e, col, up, act, n2);
  ff_store<1, EO, AOS, SUMS>(a, x, e, col, lo, act, n2);
  if (SUMS) block_partial(n2, a.partials);
}

// The same for small lattices: four groups of three warps per 32 sites, one
// direction each, whose sums meet in shared memory (the upper spins' in group
// 0, the lower ones' in group 1, which store them). A lattice of a few hundred
// blocks leaves the SMs nearly empty and its time is the chain of the eight
// hops, here four chains of two (kernel times in a graph, one group against
// four): 2,048 sites 7.6 and 5.0 us, 8^3 x 16 9.1 and 7.4, 16,384 sites 12.0 and
// 13.3, 27,648 sites 16.5 and 19.6. The line lies where two blocks of four
// groups per SM hold the lattice at once.
constexpr int kFFGroups = 4;
constexpr int kFFSmall = 2 * 152 * kFFSites;
constexpr size_t kFF4Shared = kFFGroups * (sizeof(FFShare) + sizeof(double2) * 8 * kFFThreads);

template <bool DAG, bool EO, bool AOS, bool SUMS>
__global__ void __launch_bounds__(kFFGroups * kFFThreads, 2) k_wilson_ff4(const DArgs a)
{
  const int block = SUMS ? (int)blockIdx.x : work_block(a.red);
  if (block < 0) return;
  extern __shared__ __align__(16) char ff4_shared[];
  const int grp = threadIdx.x / kFFThreads, t = threadIdx.x - grp * kFFThreads;
  const int lane = t & 31, col = t >> 5;
  const int id = a.x0 + block * kFFSites + lane;  // output index
  const bool act = id < a.V;
  const int e = act ? id : a.V - 1;  // idle lanes repeat the last site
  FFShare &hs = ((FFShare *)ff4_shared)[grp];
  double2 *stage = (double2 *)(ff4_shared + kFFGroups * sizeof(FFShare)) + grp * 8 * kFFThreads + t;
  int c[4];
  const int x = ff_site<EO>(a, e, c);
  ff_first<EO, AOS>(a, grp, col, x, c, stage);
  const float2 z = make_float2(0.f, 0.f);
  CAx2 up{FAx2{z, z}, FAx2{z, z}}, lo = up;
  if (grp == 0) ff_hops<0, 4, 1, DAG, EO, AOS>(a, col, lane, x, c, hs, stage, up, lo);
  else if (grp == 1) ff_hops<1, 4, 2, DAG, EO, AOS>(a, col, lane, x, c, hs, stage, up, lo);
  else if (grp == 2) ff_hops<2, 4, 3, DAG, EO, AOS>(a, col, lane, x, c, hs, stage, up, lo);
  else ff_hops<3, 4, 4, DAG, EO, AOS>(a, col, lane, x, c, hs, stage, up, lo);
  if (grp == 1 || grp == 2) lo = CAx2{flip2(lo.re), flip2(lo.im)};
  __syncthreads();
  CAx2 *sums = (CAx2 *)ff4_shared + t;  // [group][upper, lower][thread]: the exchange is done
  sums[(2 * grp) * kFFThreads] = up;
  sums[(2 * grp + 1) * kFFThreads] = lo;
  __syncthreads();
  double n2 = 0.0;
  if (grp < 2) {
    CAx2 s = sums[grp * kFFThreads];
#pragma unroll
    for (int g = 1; g < kFFGroups; g++) {
      const CAx2 v = sums[(2 * g + grp) * kFFThreads];
      acc_add2(s.re, v.re);
      acc_add2(s.im, v.im);
    }
    if (grp == 0) ff_store<0, EO, AOS, SUMS>(a, x, e, col, s, act, n2);
    else ff_store<1, EO, AOS, SUMS>(a, x, e, col, s, act, n2);
  }
  if (SUMS) block_partial(n2, a.partials);
}
static_assert(kFF4Shared >= sizeof(CAx2) * 2 * kFFGroups * kFFThreads, "the sums replace the exchange");

// ------------------------------------------------------ float-pair links
__global__ void k_gauge_to_ff(float4 *dst, int64_t dstride, const double2 *src, int64_t sstride, int64_t V,
                              DArgs phases)
{
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= V * 4) return;
  int64_t x = i >> 2;
  int mu = (int)(i & 3);
  bool tw = (phases.twist_mask >> mu) & 1;
  double pr = phases.phr[mu], pi = phases.phi[mu];
#pragma unroll
  for (int k = 0; k < 9; k++) {
    double2 u = src[((int64_t)mu * 9 + k) * sstride + x];
    double re = u.x, im = u.y;
    if (tw) {
      re = u.x * pr - u.y * pi;
      im = u.x * pi + u.y * pr;
    }
    float rh = __double2float_rn(re), ih = __double2float_rn(im);
    dst[((int64_t)mu * 9 + k) * dstride + x] =
        make_float4(rh, __double2float_rn(re - (double)rh), ih, __double2float_rn(im - (double)ih));
  }
}

bool gauge_to_ff(qcdgpu_gauge d, qcdgpu_gauge s)
{
  if (s->prec != QCDGPU_F64) {
    set_error("float-pair links are made from an FP64 gauge field");
    return false;
  }
  DArgs ph;
  ph.twist_mask = 0;
  for (int mu = 0; mu < 4; mu++) {
    ph.phr[mu] = 1.0;
    ph.phi[mu] = 0.0;
    if (s->theta[mu] != 0.0) {
      ph.twist_mask |= 1 << mu;
      ph.phr[mu] = cos(s->theta[mu] / (double)s->L[mu]);
      ph.phi[mu] = sin(s->theta[mu] / (double)s->L[mu]);
    }
  }
  d->recon = 18;
  for (int i = 0; i < 4; i++) d->theta[i] = s->theta[i];
  unsigned gr = (unsigned)((s->V * 4 + 127) / 128);
  k_gauge_to_ff<<<gr, 128, 0, stream()>>>((float4 *)d->data, d->stride, (const double2 *)s->data, s->stride, s->V, ph);
  return QG_LAUNCHED("gauge_to_ff");
}

// the dynamic shared memory (73 KB) is opted in once per instantiation
template <bool D, bool E, bool A, bool P>
static void launch_ff(const DArgs &a)
{
  const int n = a.V - a.x0;
  const unsigned grid = (unsigned)((n + kFFSites - 1) / kFFSites) + (a.red.n ? 1 : 0);
  if (n > kFFSmall) {
    k_wilson_ff<D, E, A, P><<<grid, kFFThreads, 0, stream()>>>(a);
    return;
  }
  static const cudaError_t opted = cudaFuncSetAttribute(
      k_wilson_ff4<D, E, A, P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFF4Shared);
  (void)opted;  // a failure shows in the launch
  k_wilson_ff4<D, E, A, P><<<grid, kFFGroups * kFFThreads, kFF4Shared, stream()>>>(a);
}

int64_t dslash_df64_blocks(int64_t V) { return (V + kFFSites - 1) / kFFSites; }

bool dslash_df64(const DArgs &a, bool dag, bool eo)
{
  if (a.aos) {
    if (dag) launch_ff<true, false, true, false>(a);
    else launch_ff<false, false, true, false>(a);
  } else if (a.partials) {
    if (dag && eo) launch_ff<true, true, false, true>(a);
    else if (dag) launch_ff<true, false, false, true>(a);
    else if (eo) launch_ff<false, true, false, true>(a);
    else launch_ff<false, false, false, true>(a);
  } else {
    if (dag && eo) launch_ff<true, true, false, false>(a);
    else if (dag) launch_ff<true, false, false, false>(a);
    else if (eo) launch_ff<false, true, false, false>(a);
    else launch_ff<false, false, false, false>(a);
  }
  return QG_LAUNCHED("wilson_df64");
}

}  // namespace qg
