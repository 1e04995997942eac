// Device code of one tile of the fused FP64 NEMOLite2D step, shared by the
// single-domain kernel (nl2d_fused.cu) and the ensemble's persistent kernel
// (nl2d_ensemble.cu).  See nl2d_fused.cu for what a step computes and why it
// is bit-identical to the reference.
#pragma once
#include <cstring>
#include <type_traits>

#include "nl2d_exact.cuh"
#include "nl2d_internal.h"

namespace nl2d {
namespace {


// The copy region splits into interior cells, [xs+1, xe-1] x [ys+1, ye-1],
// and the ring around them (ring_pos).  A tile is TX x TY interior cells,
// worked on by NT threads laid out TX x (NT / TX); each thread updates TY / (NT
// / TX) cells of one column.  Tile<TX, TY, NT> holds a shape's constants;
// the ensemble instantiates several shapes (its autotuner picks one), the
// single-domain kernel picks by domain size.  Ring cells need the general
// per-cell code, a long FP64 chain, and are taken one per thread by blocks of
// their own that run beside the tiles.  The arithmetic does not depend on
// the split.

// A constant factor of the tiles: c and its integer form.
//
// Where every field a tile reads (ssh, u, v, the depths, stored face heights)
// is +-0 or of magnitude in [2^-200, 2^200) and the constants lie in [2^-40,
// 2^40], its update is straight-line code in the bounded forms
// (nl2d_exact.cuh): no product overflows (the largest, an advective flux, is
// below 2^730), every nonzero sum of fields is at least 2^-252, a face height
// 2^-333, a sum of depths 2^-385, and the smallest product (an advective
// flux: velocity, face speed, depth) 2^-880, normal, so a power of two may
// move between an operand and a constant without changing a bit.  Tendencies
// and momenta can cancel below that and are tested before they are scaled.
//
// Other tiles ("wide") run the same update with the plain operations and the
// exact helpers that branch to the IEEE ones.  From rest the tide sends ahead
// of it values that fall by five decades per cell down to the smallest
// subnormal, for thousands of steps: half of a 128^2 domain holds values
// below 2^-200 after 1000 steps, so this form matters too (per-cell fallback
// to the general code made steps from rest up to 4 times slower).
struct Factor {
  double c;
  IntFactor i;
};
__device__ __forceinline__ bool out_of_range(double field) { return beyond(field, 200, 200); }

// Step-invariant constants of the fast path, evaluated on the host with the
// operations the reference performs per point (e.g. dx_v[c] + dx_v[e] on a
// uniform grid is one add of two equal values), so they are bit-identical.
struct FastConst {
  double area_t, area_u, area_v, dx_u, dx_v, dx_t, dy_u, dy_v, dy_t;
  double dxv2, dyu2;                       // dx_v + dx_v, dy_u + dy_u
  double cor_u, cor_v, neg_cor_v;          // 2. * omega * sin(gphi * d2r)
  double neg_g, rdt, visc, g;
  // the constant divisors (fric: 1.0 + cbfr * rdt), and whether every one
  // lies in [2^-100, 2^100]
  IntDivisor q_area_t, q_area_u, q_area_v, q_dx_t, q_dy_t, q_dxv2, q_dyu2, q_fric;
  int fast_div;
  // The tiles' factors, with the powers of two of the face averages folded in
  // (the same bits: nothing they scale leaves the normal range, see Factor),
  // and the face heights' divisors 2 area_u, 2 area_v.
  Factor f_area_t, f_rdt, f_dy_u, f_dx_v, f_hdx_u, f_hdy_v;  // h: half
  Factor f_U, f_V, f_Uw, f_Vs;                   // dy_t/2, dx_t/2, dyu2/8, dxv2/8
  Factor f_cor_area_u, f_cor_area_v;             // area_u/4, area_v/4
  IntDivisor q_2area_u, q_2area_v;
  // whether the tiles' straight-line code applies: every constant divisor and
  // factor lies in [2^-40, 2^40] (visc, cor and g may be zero); and whether
  // all factors have the integer form
  int bounded, int_mul;
};

// One domain of an ensemble (device-resident descriptor).
struct EnsDomain {
  Fields f;
  FusedState fs[2];  // [parity]: state buffers read and written at that parity
  Dims d;
  Scalars p;
  UniformMetrics um;
  FastConst k;
};

// Multiplication by a constant: 20 instructions when every constant has the
// integer form (IC), 30 otherwise.
template <bool IC>
__device__ __forceinline__ double mlc(double x, const Factor& f) {
  return IC ? mul_bounded(x, f.i) : mul_bounded(x, f.c);
}

// Division by a step constant: in integers when the constants allow it,
// otherwise the IEEE divide.  Both give the same bits.
__device__ __forceinline__ double dvc(double x, const IntDivisor& v, int fast) {
  return fast ? div_const(x, v) : div_ieee(x, v.d);
}
// Division by a per-face depth with its 64-bit reciprocal; 0 marks a depth
// outside [2^-100, 2^100] (IEEE divide).
__device__ __forceinline__ double dvf(double x, double d, unsigned long long rc) {
  return rc != 0 ? div_depth(x, d, rc) : div_ieee(x, d);
}

// The general code's context without a tile: every input read from the domain's
// arrays in global memory (the members refer to the domain's descriptor, so no thread
// holds a copy of it).  Valid for the faces a copy-region cell's general
// update reads, all of which lie inside the array.
struct GlobalCtx {
  static constexpr bool kStaged = false;
  const double* const& sn;  // the state buffers read this step
  const double* const& un;
  const double* const& vn;
  double* const& hu;  // the domain's Fields
  double* const& hv;
  double* const& ht;
  double* const& ssha_u;
  double* const& ssha_v;
  unsigned long long* const& r_hu;
  unsigned long long* const& r_hv;
  int* const& m;
  double* const& sshn_u;
  double* const& sshn_v;
  const int& W;
  const Dims& d;
  const FastConst& k;

  __device__ __forceinline__ GlobalCtx(const Fields& f, const FusedState& fs, const Dims& dd,
                                       const FastConst& kk)
      : sn(fs.sshn_in), un(fs.un_in), vn(fs.vn_in), hu(f.hu), hv(f.hv), ht(f.ht),
        ssha_u(f.ssha_u), ssha_v(f.ssha_v), r_hu(f.r_hu), r_hv(f.r_hv), m(f.tmask), sshn_u(f.sshn_u), sshn_v(f.sshn_v), W(dd.width), d(dd), k(kk) {}

  // a cell's index in the fields and in the depths' reciprocals
  __device__ __forceinline__ int at(int i, int j) const { return j * W + i; }
  __device__ __forceinline__ int global(int i, int j) const { return j * W + i; }
  __device__ __forceinline__ bool in_copy(int i, int j) const {
    return i >= d.xs - 1 && i <= d.xe + 1 && j >= d.ys - 1 && j <= d.ye;
  }
  // next_sshu_code / next_sshv_code (time_update_kern.c:90-155) at face (i,j)
  // from the mask and sshn_t of its two cells and (pa, pb) area_t * sshn_t of
  // them, over the kernels' loop ranges; faces outside them keep the stored
  // value.  Everything a caller needs is loaded before any of it is used, and
  // nothing is loaded behind a mask test: the general code is a chain of
  // dependent loads and FP64 operations, and its length is what it costs.
  __device__ __forceinline__ double face_u(int i, int j, int mm, int mn, double a, double b,
                                           double pa, double pb, double stored) const {
    const double both = dvc(half(pa + pb), k.q_area_u, k.fast_div);
    const bool in = j >= d.ys && j <= d.ye && i >= d.xs && i <= d.xe - 1 && mm + mn > 0;
    return !in ? stored : (mm * mn > 0 ? both : (mm <= 0 ? b : a));
  }
  __device__ __forceinline__ double face_v(int i, int j, int mm, int mn, double a, double b,
                                           double pa, double pb, double stored) const {
    const double both = dvc(half(pa + pb), k.q_area_v, k.fast_div);
    const bool in = j >= d.ys && j <= d.ye - 1 && i >= d.xs && i <= d.xe && mm + mn > 0;
    return !in ? stored : (mm * mn > 0 ? both : (mm <= 0 ? b : a));
  }
  // the values of sshn_u / sshn_v from which face_u / face_v start
  __device__ __forceinline__ double su0(int c) const { return sshn_u[c]; }
  __device__ __forceinline__ double sv0(int c) const { return sshn_v[c]; }
  // sshn_u / sshn_v this step sees at one face
  __device__ __forceinline__ double su(int i, int j) const {
    const int c = j * W + i, n = min(c + 1, W * d.height - 1);
    const double a = sn[c], b = sn[n];
    return face_u(i, j, m[c], m[n], a, b, k.area_t * a, k.area_t * b, sshn_u[c]);
  }
  __device__ __forceinline__ double sv(int i, int j) const {
    const int c = j * W + i, n = j + 1 < d.height ? c + W : c;
    const double a = sn[c], b = sn[n];
    return face_v(i, j, m[c], m[n], a, b, k.area_t * a, k.area_t * b, sshn_v[c]);
  }
};

// (0.5 - copysign(0.5, w)) * p and (0.5 + copysign(0.5, w)) * p alone (the
// masked upwind forms): p, or +0 * p.
// (the IEEE form for a non-finite p is out of line, as for the helpers of
// nl2d_exact.cuh, so that it is not issued on every call)
static __device__ __noinline__ double zero_times_ieee(double p) { return 0.0 * p; }
__device__ __forceinline__ double zero_times(double p) {
  const long long b = bits(p);
  if (((b >> 52) & 0x7ff) == 0x7ff) return zero_times_ieee(p);
  return from_bits(b & (long long)0x8000000000000000ULL);
}
__device__ __forceinline__ double lo_only(double w, double p) {
  return bits(w) < 0 ? p : zero_times(p);
}
__device__ __forceinline__ double hi_only(double w, double p) {
  return bits(w) < 0 ? zero_times(p) : p;
}

// momentum_u_code (momentum_u_kern.c:150-262) at u face (i,j) in its loop
// range, with the masked (slip-wall) branches; returns false where the
// kernel returns early (ua keeps its value).  Same operations as the
// reference, with the exact helpers for halving, upwind picks and division.
template <class X>
__device__ __forceinline__ bool mom_u(const X& x, int i, int j, double& out) {
  const int W = x.W, c = x.at(i, j), e = c + 1, wst = c - 1, s = c - W, n = c + W,
            se = s + 1, ne = n + 1;
  const FastConst& k = x.k;
  // the masks, heights and stored face values of the six cells around
  const int m_c = x.m[c], m_e = x.m[e], m_s = x.m[s], m_se = x.m[se], m_n = x.m[n],
            m_ne = x.m[ne];
  const double sn_c = x.sn[c], sn_e = x.sn[e], sn_s = x.sn[s], sn_se = x.sn[se],
               sn_n = x.sn[n], sn_ne = x.sn[ne];
  double su_c = x.su0(c), su_s = x.su0(s), su_n = x.su0(n);
  double sv_c = x.sv0(c), sv_e = x.sv0(e), sv_s = x.sv0(s), sv_se = x.sv0(se);
  const double u_c = x.un[c], u_E = x.un[e], u_W = x.un[wst], u_S = x.un[s], u_N = x.un[n];
  const double v_C = x.vn[c], v_E = x.vn[e], v_S = x.vn[s], v_SE = x.vn[se];
  const double hu_c = x.hu[c], hu_s = x.hu[s], hu_n = x.hu[n];
  const double hv_c = x.hv[c], hv_e = x.hv[e], hv_s = x.hv[s], hv_se = x.hv[se];
  const double ht_c = x.ht[c], ht_e = x.ht[e], ssha = x.ssha_u[x.global(i, j)];
  const unsigned long long rhu = x.r_hu[x.global(i, j)];
  if (m_c + m_e <= 0) return false;
  if (m_c <= 0 || m_e <= 0) return false;
  if constexpr (!X::kStaged) {
    const double p_c = k.area_t * sn_c, p_e = k.area_t * sn_e, p_s = k.area_t * sn_s,
                 p_se = k.area_t * sn_se, p_n = k.area_t * sn_n, p_ne = k.area_t * sn_ne;
    su_c = x.face_u(i, j, m_c, m_e, sn_c, sn_e, p_c, p_e, su_c);
    su_s = x.face_u(i, j - 1, m_s, m_se, sn_s, sn_se, p_s, p_se, su_s);
    su_n = x.face_u(i, j + 1, m_n, m_ne, sn_n, sn_ne, p_n, p_ne, su_n);
    sv_s = x.face_v(i, j - 1, m_s, m_c, sn_s, sn_c, p_s, p_c, sv_s);
    sv_se = x.face_v(i + 1, j - 1, m_se, m_e, sn_se, sn_e, p_se, p_e, sv_se);
    sv_c = x.face_v(i, j, m_c, m_n, sn_c, sn_n, p_c, p_n, sv_c);
    sv_e = x.face_v(i + 1, j, m_e, m_ne, sn_e, sn_ne, p_e, p_ne, sv_e);
  }

  double u_e = half(u_c + u_E) * k.dy_t;
  double depe = ht_e + sn_e;
  double u_w = half(u_c + u_W) * k.dy_t;
  double depw = ht_c + sn_c;
  double v_sc = half(v_S + v_SE);
  double v_s = half(v_sc) * k.dxv2;
  double deps = half(hv_s + sv_s + hv_se + sv_se);
  double v_nc = half(v_C + v_E);
  double v_n = half(v_nc) * k.dxv2;
  double depn = half(hv_c + sv_c + hv_e + sv_e);

  double uu_w = upwind(u_w, u_c, u_W);
  double uu_e = upwind(u_e, u_E, u_c);
  const bool south_dry = m_s <= 0 || m_se <= 0;
  const bool north_dry = m_n <= 0 || m_ne <= 0;
  double uu_s = south_dry ? lo_only(v_s, u_c) : upwind(v_s, u_c, u_S);
  double uu_n = north_dry ? hi_only(v_n, u_c) : upwind(v_n, u_N, u_c);
  double adv = uu_w * u_w * depw - uu_e * u_e * depe + uu_s * v_s * deps -
               uu_n * v_n * depn;

  double dudx_e = dvc(u_E - u_c, k.q_dx_t, k.fast_div) * depe;
  double dudx_w = dvc(u_c - u_W, k.q_dx_t, k.fast_div) * depw;
  double dudy_s = south_dry ? 0.0
                            : dvc(u_c - u_S, k.q_dyu2, k.fast_div) *
                                  (hu_c + su_c + hu_s + su_s);
  double dudy_n = north_dry ? 0.0
                            : dvc(u_N - u_c, k.q_dyu2, k.fast_div) *
                                  (hu_c + su_c + hu_n + su_n);
  double vis = (dudx_e - dudx_w) * k.dy_u + half((dudy_n - dudy_s) * k.dx_u);
  vis = k.visc * vis;
  double cor = half(k.cor_u * (v_sc + v_nc)) * k.area_u * (hu_c + su_c);
  double hpg = k.neg_g * (hu_c + su_c) * k.dy_u * (sn_e - sn_c);
  const double num =
      u_c * (hu_c + su_c) + dvc(k.rdt * (adv + vis + cor + hpg), k.q_area_u, k.fast_div);
  out = dvc(dvf(num, hu_c + ssha, rhu), k.q_fric, k.fast_div);
  return true;
}

// momentum_v_code (momentum_v_kern.c:125-241) at v face (i,j).
template <class X>
__device__ __forceinline__ bool mom_v(const X& x, int i, int j, double& out) {
  const int W = x.W, c = x.at(i, j), e = c + 1, wst = c - 1, s = c - W, n = c + W,
            nw = n - 1, ne = n + 1;
  const FastConst& k = x.k;
  const int m_c = x.m[c], m_e = x.m[e], m_w = x.m[wst], m_n = x.m[n], m_nw = x.m[nw],
            m_ne = x.m[ne];
  const double sn_c = x.sn[c], sn_e = x.sn[e], sn_w = x.sn[wst], sn_n = x.sn[n],
               sn_nw = x.sn[nw], sn_ne = x.sn[ne];
  double su_c = x.su0(c), su_w = x.su0(wst), su_n = x.su0(n), su_nw = x.su0(nw);
  double sv_c = x.sv0(c), sv_w = x.sv0(wst), sv_e = x.sv0(e);
  const double v_c = x.vn[c], v_E = x.vn[e], v_W = x.vn[wst], v_S = x.vn[s], v_N = x.vn[n];
  const double u_C = x.un[c], u_N = x.un[n], u_W = x.un[wst], u_NW = x.un[nw];
  const double hv_c = x.hv[c], hv_w = x.hv[wst], hv_e = x.hv[e];
  const double hu_c = x.hu[c], hu_n = x.hu[n], hu_w = x.hu[wst], hu_nw = x.hu[nw];
  const double ht_c = x.ht[c], ht_n = x.ht[n], ssha = x.ssha_v[x.global(i, j)];
  const unsigned long long rhv = x.r_hv[x.global(i, j)];
  if (m_c + m_e <= 0) return false;
  if (m_c <= 0 || m_n <= 0) return false;
  if constexpr (!X::kStaged) {
    const double p_c = k.area_t * sn_c, p_e = k.area_t * sn_e, p_w = k.area_t * sn_w,
                 p_n = k.area_t * sn_n, p_nw = k.area_t * sn_nw, p_ne = k.area_t * sn_ne;
    su_w = x.face_u(i - 1, j, m_w, m_c, sn_w, sn_c, p_w, p_c, su_w);
    su_nw = x.face_u(i - 1, j + 1, m_nw, m_n, sn_nw, sn_n, p_nw, p_n, su_nw);
    su_c = x.face_u(i, j, m_c, m_e, sn_c, sn_e, p_c, p_e, su_c);
    su_n = x.face_u(i, j + 1, m_n, m_ne, sn_n, sn_ne, p_n, p_ne, su_n);
    sv_c = x.face_v(i, j, m_c, m_n, sn_c, sn_n, p_c, p_n, sv_c);
    sv_w = x.face_v(i - 1, j, m_w, m_nw, sn_w, sn_nw, p_w, p_nw, sv_w);
    sv_e = x.face_v(i + 1, j, m_e, m_ne, sn_e, sn_ne, p_e, p_ne, sv_e);
  }

  double v_n = half(v_c + v_N) * k.dx_t;
  double depn = ht_n + sn_n;
  double v_s = half(v_c + v_S) * k.dx_t;
  double deps = ht_c + sn_c;
  double u_wc = half(u_W + u_NW);
  double u_w = half(u_wc) * k.dyu2;
  double depw = half(hu_w + su_w + hu_nw + su_nw);
  double u_ec = half(u_C + u_N);
  double u_e = half(u_ec) * k.dyu2;
  double depe = half(hu_c + su_c + hu_n + su_n);

  double vv_s = upwind(v_s, v_c, v_S);
  double vv_n = upwind(v_n, v_N, v_c);
  const bool west_dry = m_w <= 0 || m_nw <= 0;
  const bool east_dry = m_e <= 0 || m_ne <= 0;
  double vv_w = west_dry ? lo_only(u_w, v_c) : upwind(u_w, v_c, v_W);
  double vv_e = east_dry ? hi_only(u_e, v_c) : upwind(u_e, v_E, v_c);
  double adv = vv_w * u_w * depw - vv_e * u_e * depe + vv_s * v_s * deps -
               vv_n * v_n * depn;

  double dvdy_n = dvc(v_N - v_c, k.q_dy_t, k.fast_div) * depn;
  double dvdy_s = dvc(v_c - v_S, k.q_dy_t, k.fast_div) * deps;
  double dvdx_w = west_dry ? 0.0
                           : dvc(v_c - v_W, k.q_dxv2, k.fast_div) *
                                 (hv_c + sv_c + hv_w + sv_w);
  double dvdx_e = east_dry ? 0.0
                           : dvc(v_E - v_c, k.q_dxv2, k.fast_div) *
                                 (hv_c + sv_c + hv_e + sv_e);
  double vis = (dvdy_n - dvdy_s) * k.dx_v + half((dvdx_e - dvdx_w) * k.dy_v);
  vis = k.visc * vis;
  double cor = -half(k.cor_v * (u_ec + u_wc)) * k.area_v * (hv_c + sv_c);
  double hpg = k.neg_g * (hv_c + sv_c) * k.dx_v * (sn_n - sn_c);
  const double num =
      v_c * (hv_c + sv_c) + dvc(k.rdt * (adv + vis + cor + hpg), k.q_area_v, k.fast_div);
  out = dvc(dvf(num, hv_c + ssha, rhv), k.q_fric, k.fast_div);
  return true;
}

// ua at u face (i,j) after momentum_u and bc_solid_u, before Flather: the
// value bc_flather_u reads.  On the copy region the previous step's ua is
// the current un; elsewhere it is the ua array, which no fused step changes.
template <class X>
__device__ __forceinline__ double ua_pre_flather(const X& x, const double* ua_arr, int i,
                                                 int j) {
  const int c = x.at(i, j);
  double ua = x.in_copy(i, j) ? x.un[c] : ua_arr[x.global(i, j)];
  if (i >= x.d.xs && i <= x.d.xe - 1 && j >= x.d.ys && j <= x.d.ye) {
    double v;
    if (mom_u(x, i, j, v)) ua = v;
  }
  if (i >= x.d.xs - 1 && i <= x.d.xe && j >= x.d.ys - 1 && j <= x.d.ye + 1 &&
      x.m[c] * x.m[c + 1] == 0)
    ua = 0.0;  // bc_solid_u
  return ua;
}

template <class X>
__device__ __forceinline__ double va_pre_flather(const X& x, const double* va_arr, int i,
                                                 int j) {
  const int c = x.at(i, j);
  double va = x.in_copy(i, j) ? x.vn[c] : va_arr[x.global(i, j)];
  if (i >= x.d.xs && i <= x.d.xe && j >= x.d.ys && j <= x.d.ye - 1) {
    double v;
    if (mom_v(x, i, j, v)) va = v;
  }
  if (i >= x.d.xs - 1 && i <= x.d.xe + 1 && j >= x.d.ys - 1 && j <= x.d.ye &&
      x.m[c] * x.m[c + x.W] == 0)
    va = 0.0;  // bc_solid_v
  return va;
}

// A copy-region cell's update by the reference's per-point code, in three
// independent parts (each reads the old state only), so that three threads
// share what would be one long chain: v at the north face (momentum_v,
// bc_solid_v, bc_flather_v), u at the east face (momentum_u, bc_solid_u,
// bc_flather_u), sea-surface height (continuity_kern.c:90-117, then bc_ssh).
// A Flather face takes the momentum of the face next to it instead of its
// own (bc_flather replaces it), so each part evaluates one momentum update.
// (The IEEE operations and branching helpers here, not the tiles' bounded
// forms: with those a small domain's step was no shorter, and the
// FP64-equivalent form's, whose march fills the integer pipes, 4 % longer.)
enum { kPartV, kPartU, kPartSsh, kParts };
template <class X>
__device__ __forceinline__ double general_ssh(const X& x, const FastConst& k, double tide, int i,
                                              int j) {
  const Dims& d = x.d;
  const int W = x.W, c = x.at(i, j);
  const auto& m = x.m;
  if (!(i >= d.xs && i <= d.xe && j >= d.ys && j <= d.ye)) return x.sn[c];
  const int w = c - 1, s = c - W;
  double r1 = (x.su(i, j) + x.hu[c]) * x.un[c];
  double r2 = (x.su(i - 1, j) + x.hu[w]) * x.un[w];
  double r3 = (x.sv(i, j) + x.hv[c]) * x.vn[c];
  double r4 = (x.sv(i, j - 1) + x.hv[s]) * x.vn[s];
  const double ssh = x.sn[c] + dvc((r2 - r1 + r4 - r3) * k.rdt, k.q_area_t, k.fast_div);
  return m[c] > 0 && (m[c - W] < 0 || m[c + W] < 0 || m[c + 1] < 0 || m[c - 1] < 0) ? tide : ssh;
}
// The face whose momentum a copy-region cell's u (north-south: v) face takes:
// its own, or the next one for a Flather face.  mc, mn: the masks of the
// face's two cells.
__device__ __forceinline__ int flather_face(int mc, int mn, int i) {
  if (mc + mn > -1) {
    if (mc < 0) return i + 1;
    if (mn < 0 && i >= 1) return i - 1;  // i == 0 would read outside the array
  }
  return i;
}
__device__ __forceinline__ void general_part(const Fields& f, const FusedState& fs,
                                             const Dims& d, const Scalars& p, const FastConst& k,
                                             double tide, int part, int i, int j) {
  const GlobalCtx x(f, fs, d, k);
  const int* __restrict__ m = x.m;
  const int c = x.at(i, j);

  if (part == kPartSsh) {
    fs.sshn_out[c] = general_ssh(x, k, tide, i, j);
  } else if (part == kPartU) {
    double ua;
    if (i <= d.xe) {  // u whole range [xs-1, xe] x [ys-1, ye+1] (the copy region gives the rest)
      const int fi = flather_face(m[c], m[c + 1], i);
      ua = ua_pre_flather(x, f.ua, fi, j);
      if (fi != i) ua = ua + sqrt(p.g / f.hu[c]) * (x.su(i, j) - x.su(fi, j));
    } else {
      ua = x.un[c];
    }
    fs.un_out[c] = ua;
  } else {
    // the copy region is exactly the v whole range [xs-1, xe+1] x [ys-1, ye]
    const int fj = flather_face(m[c], m[c + d.width], j);
    double va = va_pre_flather(x, f.va, i, fj);
    if (fj != j) va = va + sqrt(p.g / f.hv[c]) * (x.sv(i, j) - x.sv(i, fj));
    fs.vn_out[c] = va;
  }
}

// general_part out of line, for the ring's cells and the tiles' Flather faces:
// the tiles' registers are sized by the regular update.
static __device__ __noinline__ void general_at(const Fields& f, const FusedState& fs,
                                               const Dims& d, const Scalars& p,
                                               const FastConst& k, double tide, int part, int i,
                                               int j) {
  general_part(f, fs, d, p, k, tide, part, i, j);
}

// The ring: the copy region's cells outside the interior, rows ys-1, ys, ye
// and columns xs-1, xs, xe, xe+1 (the whole copy region when it has no
// interior).  ring_count: its cells in copy-region rows [ja, jb); ring_pos:
// the g-th of them, the full rows first.
struct RingRows {
  int nfull, npart, part0;  // full rows; the others, from row part0
};
__host__ __device__ __forceinline__ RingRows ring_rows(const Dims& d, int ja, int jb) {
  if (d.xe - d.xs < 2 || d.ye - d.ys < 2) return RingRows{jb - ja, 0, 0};
  const int p0 = ja > d.ys + 1 ? ja : d.ys + 1, p1 = jb < d.ye ? jb : d.ye;
  const int np = p1 > p0 ? p1 - p0 : 0;
  return RingRows{jb - ja - np, np, p0};
}
__host__ __device__ __forceinline__ int ring_count(const Dims& d, int ja, int jb) {
  const RingRows r = ring_rows(d, ja, jb);
  return r.nfull * (d.xe - d.xs + 3) + r.npart * 4;
}
__host__ __device__ __forceinline__ void ring_pos(const Dims& d, int ja, int jb, int g, int& i,
                                                  int& j) {
  const RingRows r = ring_rows(d, ja, jb);
  const int nx = d.xe - d.xs + 3;
  if (g < r.nfull * nx) {
    const int q = g / nx;
    i = d.xs - 1 + (g - q * nx);
    j = ja + q;  // rows below the partial ones, then those above
    if (r.npart > 0 && j >= r.part0) j += r.npart;
  } else {
    const int h = g - r.nfull * nx, c = h & 3;
    j = r.part0 + (h >> 2);
    i = c < 2 ? d.xs - 1 + c : d.xe + c - 2;
  }
}

// Shared-memory layout of one tile, all on the tile plus one cell on each
// side: the loaded fields and the sshn_u / sshn_v this step sees, then the
// terms that two neighbouring updates share.
enum { A_SN, A_UN, A_VN, A_HU, A_HV, A_HT, A_SU, A_SV, A_HUS, A_HVS, N_A0 };
enum { B_FLXU, B_FLXV, B_GX, B_GY, B_FXU, B_FYV, B_VS2, B_FYU, B_QY, B_UW2, B_FXV, B_QX, N_B1 };
// area_t * sshn_t, needed until the face values are formed, shares the slot
// of a term that is formed after them
constexpr int B_AREA_SSH = B_QX;

// NT threads per CTA.  MB: CTAs per SM to hold the registers to, 0 for what
// the shared memory allows, up to two.
template <int TX_, int TY_, int NT = 256, int MB = 0>
struct Tile {
  static constexpr int TX = TX_, TY = TY_, NTHREADS = NT;
  static constexpr int RPP = NTHREADS / TX;  // rows per pass of the thread block
  static constexpr int RPT = TY / RPP;       // cells per thread in the update phase
  static_assert(NTHREADS % TX == 0 && TY % RPP == 0 && (RPT == 1 || RPT == 2 || RPT == 4),
                "tile shape");
  static constexpr int SX = TX + 2, SY = TY + 2;
  static constexpr int S0 = SX * SY;  // staged positions (34 x 18 for 32 x 16)
  // + the mask, the list of the tile's general (non-regular) cells
  static constexpr size_t kSmemBytes =
      sizeof(double) * (N_A0 + N_B1) * S0 + sizeof(int) * (S0 + TX * TY + 1);
  // shared memory per CTA (with the 1 KB the driver reserves) against the
  // SM's 228 KB
  static constexpr int kMinBlocks = MB > 0 ? MB : 2 * (kSmemBytes + 1024) <= 228 * 1024 ? 2 : 1;
  static_assert(kMinBlocks * (kSmemBytes + 1024) <= 228 * 1024 || kMinBlocks == 1, "tile shape");
  // Items along the tile's edges are handled by whole warps: an edge's items
  // start at a multiple of 32 of the thread index.
  static constexpr int RX = (TX + 31) / 32 * 32, RY = (TY + 31) / 32 * 32,
                       RY1 = (TY + 32) / 32 * 32;
};

template <class T>
struct TileSmem {
  double *a0, *b1;       // [N_A0][S0], [N_B1][S0]
  int* mk;               // [S0] the mask
  int *glist, *gcount;   // [TX * TY] the tile's general cells, their number
  __device__ __forceinline__ explicit TileSmem(double* smem)
      : a0(smem), b1(smem + N_A0 * T::S0), mk((int*)(b1 + N_B1 * T::S0)), glist(mk + T::S0),
        gcount(glist + T::TX * T::TY) {}
};

// The general code's context for the interior cells of a tile: the fields and
// the sshn_u / sshn_v of the cells around are the staged ones.
template <class T>
struct TileCtx {
  static constexpr bool kStaged = true;
  static constexpr int W = T::SX;
  const double *sn, *un, *vn, *hu, *hv, *ht, *su_at, *sv_at;
  const double *ssha_u, *ssha_v;
  const unsigned long long *r_hu, *r_hv;
  const int* m;
  const Dims& d;
  const FastConst& k;
  int i0, j0;

  __device__ __forceinline__ TileCtx(double* smem, const Fields& f, const Dims& dd,
                                     const FastConst& kk, int i0_, int j0_)
      : ssha_u(f.ssha_u), ssha_v(f.ssha_v), r_hu(f.r_hu), r_hv(f.r_hv), d(dd), k(kk), i0(i0_),
        j0(j0_) {
    const TileSmem<T> t(smem);
    const double* a0 = t.a0;
    constexpr int S0 = T::S0;
    sn = a0 + A_SN * S0, un = a0 + A_UN * S0, vn = a0 + A_VN * S0;
    hu = a0 + A_HU * S0, hv = a0 + A_HV * S0, ht = a0 + A_HT * S0;
    su_at = a0 + A_SU * S0, sv_at = a0 + A_SV * S0;
    m = t.mk;
  }
  __device__ __forceinline__ int at(int i, int j) const {
    return (j - j0 + 1) * W + (i - i0 + 1);
  }
  __device__ __forceinline__ int global(int i, int j) const { return j * d.width + i; }
  __device__ __forceinline__ bool in_copy(int, int) const { return true; }
  __device__ __forceinline__ double su0(int c) const { return su_at[c]; }
  __device__ __forceinline__ double sv0(int c) const { return sv_at[c]; }
  __device__ __forceinline__ double su(int i, int j) const { return su_at[at(i, j)]; }
  __device__ __forceinline__ double sv(int i, int j) const { return sv_at[at(i, j)]; }
};

// A cell of the tile staged in shared memory, by the general code: the same
// operations as general_part's on the staged values, whose faces are formed once
// per tile.  By general_at, which reads global memory and forms each part's seven
// faces anew (FP64 products, the pipe that bounds the step), us per step: 2048^2
// with 3 % of the cells dry 2820, with the staged values 1320; 601 x 413 with a
// coast and an island 61.2 and 49.6.  A Flather face reads two cells on and goes
// there.  One thread takes a cell's three parts, as independent chains: a thread
// for each part kept three times as many warps on the FP64 and integer pipes for
// it (10 % of the cells dry: 601 x 413 110.1 us, so 102.2; 1024^2 412 and 371; 16
// domains of 256^2 537 and 466; 200 of 60^2 on static schedules in 32 x 8 tiles
// 589 and 459; where such cells are few the chain is longer: 601 x 413 with the
// coast 50.8 and 51.9).
template <class T>
__device__ __forceinline__ void general_in_tile(const Fields& f, const FusedState& fs,
                                                const Dims& d, const Scalars& p,
                                                const FastConst& k, double tide, int i, int j,
                                                int i0, int j0) {
  extern __shared__ double smem[];
  const TileCtx<T> x(smem, f, d, k, i0, j0);
  const int c = x.at(i, j), g = x.global(i, j);
  if (flather_face(x.m[c], x.m[c + x.W], j) == j)
    fs.vn_out[g] = va_pre_flather(x, f.va, i, j);
  else
    general_at(f, fs, d, p, k, tide, kPartV, i, j);
  if (flather_face(x.m[c], x.m[c + 1], i) == i)
    fs.un_out[g] = ua_pre_flather(x, f.ua, i, j);
  else
    general_at(f, fs, d, p, k, tide, kPartU, i, j);
  fs.sshn_out[g] = general_ssh(x, k, tide, i, j);
}
// The same out of line, for kernels whose regular update it would slow down.
template <class T>
__device__ __noinline__ void general_in_tile_apart(const Fields& f, const FusedState& fs,
                                                   const Dims& d, const Scalars& p,
                                                   const FastConst& k, double tide, int i, int j,
                                                   int i0, int j0) {
  general_in_tile<T>(f, fs, d, p, k, tide, i, j, i0, j0);
}

// A regular cell's new (sshn_t, un, vn) from the tile's staged fields (a0)
// and shared terms (b1) at its slot q: continuity (continuity_kern.c:90-117)
// and unmasked momentum (momentum_u_kern.c:184-261,
// momentum_v_kern.c:159-239) in the reference's operation order, without a
// branch.  dhu, rhu, dhv, rhv: hu + ssha_u and hv + ssha_v at the cell and
// their reciprocals.  bad: a tendency or momentum is outside the bounded
// forms' range (or a depth has no reciprocal), the results are not valid.
struct RegOut {
  double ssh, u, v;
  bool bad;
};
template <class T, bool IC>
__device__ __forceinline__ RegOut regular_cell(const double* a0, const double* b1, int q,
                                               double dhu, unsigned long long rhu, double dhv,
                                               unsigned long long rhv, const FastConst& k) {
  constexpr int S0 = T::S0, SX = T::SX;
#define A(qq, t) a0[(qq) * S0 + (t)]
#define B(qq, t) b1[(qq) * S0 + (t)]
  RegOut o;
  o.bad = rhu == 0 || rhv == 0;
  const double snc = A(A_SN, q), Hu = A(A_HUS, q), Hv = A(A_HVS, q);
  const double ssh =
      mlc<IC>(((B(B_FLXU, q - 1) - B(B_FLXU, q)) + B(B_FLXV, q - SX)) - B(B_FLXV, q), k.f_rdt);
  o.ssh = snc + div_bounded(ssh, k.q_area_t);
  {
    const double adv = ((B(B_FXU, q) - B(B_FXU, q + 1)) + B(B_FYU, q)) - B(B_FYU, q + SX);
    const double dudy_s = mul_bounded(B(B_QY, q), (Hu + A(A_HU, q - SX)) + A(A_SU, q - SX));
    const double dudy_n =
        mul_bounded(B(B_QY, q + SX), (Hu + A(A_HU, q + SX)) + A(A_SU, q + SX));
    double vis = mlc<IC>(B(B_GX, q + 1) - B(B_GX, q), k.f_dy_u) +
                 mlc<IC>(dudy_n - dudy_s, k.f_hdx_u);
    vis = mul_bounded(vis, k.visc);
    const double cor = mul_bounded(
        mlc<IC>(mul_bounded(B(B_VS2, q) + B(B_VS2, q + SX), k.cor_u), k.f_cor_area_u), Hu);
    const double hpg =
        mul_bounded(mlc<IC>(mul_bounded(Hu, k.neg_g), k.f_dy_u), A(A_SN, q + 1) - snc);
    const double tend = ((adv + vis) + cor) + hpg;
    const double num =
        mul_bounded(A(A_UN, q), Hu) + div_bounded(mlc<IC>(tend, k.f_rdt), k.q_area_u);
    o.bad |= beyond(tend, 699, 699) || beyond(num, 699, 699);
    o.u = div_bounded(div_bounded(num, dhu, rhu), k.q_fric);
  }
  {
    const double adv = ((B(B_FXV, q) - B(B_FXV, q + 1)) + B(B_FYV, q)) - B(B_FYV, q + SX);
    const double dvdx_w = mul_bounded(B(B_QX, q), (Hv + A(A_HV, q - 1)) + A(A_SV, q - 1));
    const double dvdx_e =
        mul_bounded(B(B_QX, q + 1), (Hv + A(A_HV, q + 1)) + A(A_SV, q + 1));
    double vis = mlc<IC>(B(B_GY, q + SX) - B(B_GY, q), k.f_dx_v) +
                 mlc<IC>(dvdx_e - dvdx_w, k.f_hdy_v);
    vis = mul_bounded(vis, k.visc);
    const double cor = mul_bounded(
        mlc<IC>(mul_bounded(B(B_UW2, q + 1) + B(B_UW2, q), k.neg_cor_v), k.f_cor_area_v), Hv);
    const double hpg =
        mul_bounded(mlc<IC>(mul_bounded(Hv, k.neg_g), k.f_dx_v), A(A_SN, q + SX) - snc);
    const double tend = ((adv + vis) + cor) + hpg;
    const double num =
        mul_bounded(A(A_VN, q), Hv) + div_bounded(mlc<IC>(tend, k.f_rdt), k.q_area_v);
    o.bad |= beyond(tend, 699, 699) || beyond(num, 699, 699);
    o.v = div_bounded(div_bounded(num, dhv, rhv), k.q_fric);
  }
  return o;
}

// The same in the plain operations and the helpers that take any value.
template <class T>
__device__ __forceinline__ RegOut regular_cell_any(const double* a0, const double* b1, int q,
                                                   double dhu, unsigned long long rhu, double dhv,
                                                   unsigned long long rhv, const FastConst& k) {
  constexpr int S0 = T::S0, SX = T::SX;
  RegOut o;
  o.bad = false;
  const double snc = A(A_SN, q), Hu = A(A_HUS, q), Hv = A(A_HVS, q);
  const double ssh = (((B(B_FLXU, q - 1) - B(B_FLXU, q)) + B(B_FLXV, q - SX)) - B(B_FLXV, q)) *
                     k.rdt;
  o.ssh = snc + dvc(ssh, k.q_area_t, k.fast_div);
  {
    const double adv = ((B(B_FXU, q) - B(B_FXU, q + 1)) + B(B_FYU, q)) - B(B_FYU, q + SX);
    const double dudy_s = B(B_QY, q) * ((Hu + A(A_HU, q - SX)) + A(A_SU, q - SX));
    const double dudy_n = B(B_QY, q + SX) * ((Hu + A(A_HU, q + SX)) + A(A_SU, q + SX));
    double vis = (B(B_GX, q + 1) - B(B_GX, q)) * k.dy_u + half((dudy_n - dudy_s) * k.dx_u);
    vis = k.visc * vis;
    const double cor = (half(k.cor_u * (B(B_VS2, q) + B(B_VS2, q + SX))) * k.area_u) * Hu;
    const double hpg = ((k.neg_g * Hu) * k.dy_u) * (A(A_SN, q + 1) - snc);
    const double num =
        A(A_UN, q) * Hu + dvc(k.rdt * (((adv + vis) + cor) + hpg), k.q_area_u, k.fast_div);
    const double t1 = dvf(num, dhu, rhu);
    o.u = dvc(t1, k.q_fric, k.fast_div);
  }
  {
    const double adv = ((B(B_FXV, q) - B(B_FXV, q + 1)) + B(B_FYV, q)) - B(B_FYV, q + SX);
    const double dvdx_w = B(B_QX, q) * ((Hv + A(A_HV, q - 1)) + A(A_SV, q - 1));
    const double dvdx_e = B(B_QX, q + 1) * ((Hv + A(A_HV, q + 1)) + A(A_SV, q + 1));
    double vis = (B(B_GY, q + SX) - B(B_GY, q)) * k.dx_v + half((dvdx_e - dvdx_w) * k.dy_v);
    vis = k.visc * vis;
    const double cor = (-half(k.cor_v * (B(B_UW2, q + 1) + B(B_UW2, q))) * k.area_v) * Hv;
    const double hpg = ((k.neg_g * Hv) * k.dx_v) * (A(A_SN, q + SX) - snc);
    const double num =
        A(A_VN, q) * Hv + dvc(k.rdt * (((adv + vis) + cor) + hpg), k.q_area_v, k.fast_div);
    const double t1 = dvf(num, dhv, rhv);
    o.v = dvc(t1, k.q_fric, k.fast_div);
  }
  return o;
}

// The terms at slot q (cell (i, j)) that neighbouring updates share.  X: the
// terms of the cell's west side, Y: of its south side (a tile's east and
// north neighbours need one of the two only).  Every term is the exact
// operation sequence of momentum_{u,v}_kern.c / continuity_kern.c for one of
// the two updates that use it, up to powers of two moved into the constants
// (the face speeds of B_FXV and B_FYU carry the half of their depth's
// average, B_VS2 and B_UW2 are twice the averaged velocities); for the other
// update the reference evaluates the same operations on the same operands
// (addition commuted), so the bits agree.
template <class T, bool IC, bool X, bool Y>
__device__ __forceinline__ void shared_terms(const double* a0, double* b1, int q,
                                             const FastConst& k) {
  constexpr int S0 = T::S0, SX = T::SX;
  const int qw = q - 1, qs = q - SX, qse = qs + 1, qwn = qw + SX;
  const double D = A(A_HT, q) + A(A_SN, q);  // ht + sshn at T(i,j)
  const double u_c = A(A_UN, q), v_c = A(A_VN, q);
  if (X && Y) {  // continuity fluxes (sshn_u + hu) * un and (sshn_v + hv) * vn
    B(B_FLXU, q) = mul_bounded(A(A_HUS, q), u_c);
    B(B_FLXV, q) = mul_bounded(A(A_HVS, q), v_c);
  }
  if (X) {
    const double u_w = A(A_UN, qw), v_w = A(A_VN, qw);
    // dudx at T(i,j): dudx_w of u face i, dudx_e of face i-1
    B(B_GX, q) = mul_bounded(div_bounded(u_c - u_w, k.q_dx_t), D);
    // x-advective flux of u through T(i,j): uu_w * u_w * depw of face i
    const double U = mlc<IC>(u_c + u_w, k.f_U);
    B(B_FXU, q) = mul_bounded(mul_bounded(upwind_bounded(U, u_c, u_w), U), D);
    // west edge of v face (i,j): u_wc, u_w, depw, vv_w (unmasked form)
    const double uw2 = u_w + A(A_UN, qwn);
    B(B_UW2, q) = uw2;
    const double Uw = mlc<IC>(uw2, k.f_Uw);
    const double depw = (A(A_HUS, qw) + A(A_HU, qwn)) + A(A_SU, qwn);
    B(B_FXV, q) = mul_bounded(mul_bounded(upwind_bounded(Uw, v_c, v_w), Uw), depw);
    B(B_QX, q) = div_bounded(v_c - v_w, k.q_dxv2);
  }
  if (Y) {
    const double u_s = A(A_UN, qs), v_s = A(A_VN, qs);
    // dvdy at T(i,j): dvdy_s of v face j, dvdy_n of face j-1
    B(B_GY, q) = mul_bounded(div_bounded(v_c - v_s, k.q_dy_t), D);
    // y-advective flux of v through T(i,j): vv_s * v_s * deps of face j
    const double V = mlc<IC>(v_c + v_s, k.f_V);
    B(B_FYV, q) = mul_bounded(mul_bounded(upwind_bounded(V, v_c, v_s), V), D);
    // south edge of u face (i,j): v_sc, v_s, deps, uu_s (unmasked form)
    const double vs2 = v_s + A(A_VN, qse);
    B(B_VS2, q) = vs2;
    const double Vs = mlc<IC>(vs2, k.f_Vs);
    const double deps = (A(A_HVS, qs) + A(A_HV, qse)) + A(A_SV, qse);
    B(B_FYU, q) = mul_bounded(mul_bounded(upwind_bounded(Vs, u_c, u_s), Vs), deps);
    B(B_QY, q) = div_bounded(u_c - u_s, k.q_dyu2);
  }
}

// The same in the plain operations and the helpers that take any value
// (B_VS2 and B_UW2 hold the averaged velocities themselves).
template <class T, bool X, bool Y>
__device__ __forceinline__ void shared_terms_any(const double* a0, double* b1, int q,
                                                 const FastConst& k) {
  constexpr int S0 = T::S0, SX = T::SX;
  const int qw = q - 1, qs = q - SX, qse = qs + 1, qwn = qw + SX;
  const double D = A(A_HT, q) + A(A_SN, q);  // ht + sshn at T(i,j)
  const double u_c = A(A_UN, q), v_c = A(A_VN, q);
  if (X && Y) {  // continuity fluxes (sshn_u + hu) * un and (sshn_v + hv) * vn
    B(B_FLXU, q) = A(A_HUS, q) * u_c;
    B(B_FLXV, q) = A(A_HVS, q) * v_c;
  }
  if (X) {
    const double u_w = A(A_UN, qw), v_w = A(A_VN, qw);
    // dudx at T(i,j): dudx_w of u face i, dudx_e of face i-1
    B(B_GX, q) = dvc(u_c - u_w, k.q_dx_t, k.fast_div) * D;
    // x-advective flux of u through T(i,j): uu_w * u_w * depw of face i
    const double U = half(u_c + u_w) * k.dy_t;
    B(B_FXU, q) = (upwind(U, u_c, u_w) * U) * D;
    // west edge of v face (i,j): u_wc, u_w, depw, vv_w (unmasked form)
    const double uwc = half(u_w + A(A_UN, qwn));
    B(B_UW2, q) = uwc;
    const double Uw = half(uwc) * k.dyu2;
    const double depw = half((A(A_HUS, qw) + A(A_HU, qwn)) + A(A_SU, qwn));
    B(B_FXV, q) = (upwind(Uw, v_c, v_w) * Uw) * depw;
    B(B_QX, q) = dvc(v_c - v_w, k.q_dxv2, k.fast_div);
  }
  if (Y) {
    const double u_s = A(A_UN, qs), v_s = A(A_VN, qs);
    // dvdy at T(i,j): dvdy_s of v face j, dvdy_n of face j-1
    B(B_GY, q) = dvc(v_c - v_s, k.q_dy_t, k.fast_div) * D;
    // y-advective flux of v through T(i,j): vv_s * v_s * deps of face j
    const double V = half(v_c + v_s) * k.dx_t;
    B(B_FYV, q) = (upwind(V, v_c, v_s) * V) * D;
    // south edge of u face (i,j): v_sc, v_s, deps, uu_s (unmasked form)
    const double vsc = half(v_s + A(A_VN, qse));
    B(B_VS2, q) = vsc;
    const double Vs = half(vsc) * k.dxv2;
    const double deps = half((A(A_HVS, qs) + A(A_HV, qse)) + A(A_SV, qse));
    B(B_FYU, q) = (upwind(Vs, u_c, u_s) * Vs) * deps;
    B(B_QY, q) = dvc(u_c - u_s, k.q_dyu2, k.fast_div);
  }
}

// The sshn_u / sshn_v this step reads: next_sshu_code / next_sshv_code
// (time_update_kern.c:90-155) over their loop ranges; other faces keep the
// stored value, which is read only for them.  Returns whether this thread met
// a stored value out of range (the wide form takes any).
template <class T, bool WIDE>
__device__ __forceinline__ bool tile_faces(const Fields& f, const Dims& d, const FastConst& k,
                                           int i0, int j0, double* smem) {
  constexpr int TX = T::TX, TY = T::TY, SX = T::SX, S0 = T::S0, NTHREADS = T::NTHREADS;
  constexpr int RX = T::RX, RY = T::RY, RY1 = T::RY1;
  const TileSmem<T> sm(smem);
  double *a0 = sm.a0, *b1 = sm.b1;
  const int* mk = sm.mk;
  const int W = d.width, imax = d.xe + 1, jmax = d.ye + 1;
  const int tid = threadIdx.y * TX + threadIdx.x;
  bool out = false;
  auto face_u = [&](int tx, int ty, bool sum) {
    const int q = (ty + 1) * SX + tx + 1, fi = i0 + tx, fj = j0 + ty;
    double su;
    const int mm = mk[q], mn = mk[q + 1];
    if (fj <= d.ye && fi <= d.xe - 1 && mm + mn > 0) {
      const double two = B(B_AREA_SSH, q) + B(B_AREA_SSH, q + 1);
      const double both = WIDE ? dvc(half(two), k.q_area_u, k.fast_div)
                               : div_bounded(two, k.q_2area_u);
      su = mm * mn > 0 ? both : (mm <= 0 ? A(A_SN, q + 1) : A(A_SN, q));
    } else {
      su = f.sshn_u[min(fj, jmax) * W + min(fi, imax)];
      out |= out_of_range(su);
    }
    A(A_SU, q) = su;
    if (sum) A(A_HUS, q) = A(A_HU, q) + su;
  };
  auto face_v = [&](int tx, int ty, bool sum) {
    const int q = (ty + 1) * SX + tx + 1, fi = i0 + tx, fj = j0 + ty;
    double sv;
    const int mm = mk[q], mn = mk[q + SX];
    if (fj <= d.ye - 1 && fi <= d.xe && mm + mn > 0) {
      const double two = B(B_AREA_SSH, q) + B(B_AREA_SSH, q + SX);
      const double both = WIDE ? dvc(half(two), k.q_area_v, k.fast_div)
                               : div_bounded(two, k.q_2area_v);
      sv = mm * mn > 0 ? both : (mm <= 0 ? A(A_SN, q + SX) : A(A_SN, q));
    } else {
      sv = f.sshn_v[min(fj, jmax) * W + min(fi, imax)];
      out |= out_of_range(sv);
    }
    A(A_SV, q) = sv;
    if (sum) A(A_HVS, q) = A(A_HV, q) + sv;
  };
#pragma unroll
  for (int e = 0; e < T::RPT; e++) {
    face_u(threadIdx.x, threadIdx.y + e * T::RPP, true);
    face_v(threadIdx.x, threadIdx.y + e * T::RPP, true);
  }
  // u faces: rows -1 and TY, column -1 (rows 0 .. TY); v faces: row -1,
  // columns -1 and TX (rows -1 .. TY-1)
  for (int t = tid; t < 3 * RX + RY + 2 * RY1; t += NTHREADS) {
    int e = t;
    if (e < RX) {
      if (e < TX) face_u(e, -1, false);
    } else if ((e -= RX) < RX) {
      if (e < TX) face_u(e, TY, false);
    } else if ((e -= RX) < RX) {
      if (e < TX) face_v(e, -1, true);
    } else if ((e -= RX) < RY1) {
      if (e <= TY) face_u(-1, e, true);
    } else if ((e -= RY1) < RY1) {
      if (e <= TY) face_v(TX, e - 1, false);
    } else {
      e -= RY1;
      if (e < TY) face_v(-1, e, false);
    }
  }
  return out;
}

// The shared terms and the regular cells' update; the other cells go to
// the tile's list.  SUMS: Fields::depth_sums.
template <class T, bool IC, bool WIDE, bool SUMS>
__device__ __forceinline__ void tile_update(const Fields& f, const FusedState& fs, const Dims& d,
                                            const FastConst& k, int i0, int j0, double* smem) {
  constexpr int TX = T::TX, TY = T::TY, SX = T::SX, S0 = T::S0, NTHREADS = T::NTHREADS;
  constexpr int RX = T::RX, RY = T::RY;
  const TileSmem<T> sm(smem);
  double *a0 = sm.a0, *b1 = sm.b1;
  int *mk = sm.mk, *glist = sm.glist, *gcount = sm.gcount;
  const int W = d.width;
  const int tid = threadIdx.y * TX + threadIdx.x;
  const int i = i0 + threadIdx.x;

  // ---- the terms shared by neighbouring updates ----
  auto terms = [&](auto x, auto y, int q) {
    if constexpr (WIDE)
      shared_terms_any<T, decltype(x)::value, decltype(y)::value>(a0, b1, q, k);
    else
      shared_terms<T, IC, decltype(x)::value, decltype(y)::value>(a0, b1, q, k);
  };
  auto flux = [&](double h, double v) { return WIDE ? h * v : mul_bounded(h, v); };
#pragma unroll
  for (int e = 0; e < T::RPT; e++) {
    const int q = (threadIdx.y + e * T::RPP + 1) * SX + threadIdx.x + 1;
    terms(std::true_type{}, std::true_type{}, q);
  }
  // the south terms of row TY, the west terms of column TX, and the fluxes
  // through the tile's west and south edges
  for (int t = tid; t < 2 * RX + 2 * RY; t += NTHREADS) {
    int e = t;
    if (e < RX) {
      if (e < TX) {
        const int q = (TY + 1) * SX + e + 1;
        terms(std::false_type{}, std::true_type{}, q);
      }
    } else if ((e -= RX) < RY) {
      if (e < TY) {
        const int q = (e + 1) * SX + TX + 1;
        terms(std::true_type{}, std::false_type{}, q);
      }
    } else if ((e -= RY) < RY) {
      const int q = (e + 1) * SX;
      if (e < TY) B(B_FLXU, q) = flux(A(A_HUS, q), A(A_UN, q));
    } else {
      e -= RY;
      const int q = e + 1;
      if (e < TX) B(B_FLXV, q) = flux(A(A_HVS, q), A(A_VN, q));
    }
  }
  __syncthreads();

  // ---- the update ----
  // Each thread owns the cells (i, j0 + row) of its rows.  Regular cells
  // (wet 3x3 neighbourhood: continuity without bc_ssh, unmasked momentum, no
  // solid-wall or Flather change; values in the bounded forms' range) are
  // computed here, two of a thread's cells in one straight-line block, so
  // that the compiler interleaves independent FP64 chains; the others are
  // queued for the packed general pass below, so that a warp holding a few
  // land-side cells does not run both paths.  The per-face global inputs are
  // loaded first and the results stored last, so no store can alias a later
  // load.
#pragma unroll
  for (int pb = 0; pb < T::RPT; pb += 2) {
    constexpr int NP = T::RPT >= 2 ? 2 : 1;  // rows taken together
    int c[NP], q[NP];
    bool live[NP], reg[NP];
    bool any = false;
#pragma unroll
    for (int e = 0; e < NP; e++) {
      const int row = threadIdx.y + (pb + e) * T::RPP, j = j0 + row;
      c[e] = j * W + i;
      q[e] = (row + 1) * SX + (threadIdx.x + 1);
      live[e] = i <= d.xe - 1 && j <= d.ye - 1;
      bool regular = live[e];
#pragma unroll
      for (int dj = -1; dj <= 1; dj++)
#pragma unroll
        for (int di = -1; di <= 1; di++) regular &= mk[q[e] + dj * SX + di] > 0;
      reg[e] = regular;
      any |= regular;
    }
    if (any) {
      double dhu[NP], dhv[NP];
      unsigned long long rhu[NP], rhv[NP];
#pragma unroll
      for (int e = 0; e < NP; e++) {  // (a cell that is not regular: the other's values)
        const int cc = reg[e] ? c[e] : c[NP - 1 - e];
        dhu[e] = f.d_hu[cc];
        rhu[e] = f.r_hu[cc];
        dhv[e] = f.d_hv[cc];
        rhv[e] = f.r_hv[cc];
        if (!SUMS) {
          dhu[e] += f.hu[cc];
          dhv[e] += f.hv[cc];
        }
      }
      RegOut o[NP];
#pragma unroll
      for (int e = 0; e < NP; e++)
        o[e] = WIDE ? regular_cell_any<T>(a0, b1, q[e], dhu[e], rhu[e], dhv[e], rhv[e], k)
                    : regular_cell<T, IC>(a0, b1, q[e], dhu[e], rhu[e], dhv[e], rhv[e], k);
#pragma unroll
      for (int e = 0; e < NP; e++) {
        reg[e] = reg[e] && !o[e].bad;
        if (reg[e]) {
          fs.sshn_out[c[e]] = o[e].ssh;
          fs.un_out[c[e]] = o[e].u;
          fs.vn_out[c[e]] = o[e].v;
        }
      }
    }
#pragma unroll
    for (int e = 0; e < NP; e++)
      if (live[e] && !reg[e])
        glist[atomicAdd(gcount, 1)] = (threadIdx.y + (pb + e) * T::RPP) * TX + threadIdx.x;
  }
  __syncthreads();
}

// One tile of the fused step: interior cells [i0, i0+TX) x [j0, j0+TY) of one
// domain.  `tide` is this step's bc_ssh value (general cells).  APART: the general
// cells' code out of line.
//
// The FP64 pipe bounds the step (about 1.7 instructions per clock per SM;
// each holds a scheduler's share of it for 64 issue slots), so every phase
// forms a value on exactly the positions that are read (a full warp per row
// of the tile, and the edges' extra values, next column and next row, packed
// into warps of their own), and products and quotients are formed in
// integers: the pipe has the step's adds only, 57 of the 140 instructions per
// cell of the form that used it for everything on 2- and 1-cell halos.  The
// integer forms pay only as straight-line code: with a range branch each,
// the same products made the step slower.
template <class T, bool IC, bool SUMS = true, bool APART = false>
__device__ __forceinline__ void fused_tile(const Fields& f, const FusedState& fs, const Dims& d,
                                           const Scalars& p, const FastConst& k, double tide,
                                           int i0, int j0, double* smem) {
  constexpr int TX = T::TX, TY = T::TY, SX = T::SX, S0 = T::S0;
  constexpr int NTHREADS = T::NTHREADS;
  const TileSmem<T> sm(smem);
  double *a0 = sm.a0, *b1 = sm.b1;
  int *mk = sm.mk, *glist = sm.glist, *gcount = sm.gcount;

  const int W = d.width;
  const int tid = threadIdx.y * TX + threadIdx.x;

  if (tid == 0) {
    *gcount = 0;
  }
  // ---- the fields (positions past the copy region hold what its last column
  // or row does; no cell that is written reads them) ----
  const int imax = d.xe + 1, jmax = d.ye + 1;
  bool wide = !k.bounded;
  for (int t = tid; t < S0; t += NTHREADS) {
    const int c = min(j0 - 1 + t / SX, jmax) * W + min(i0 - 1 + t % SX, imax);
    const double sn = fs.sshn_in[c], un = fs.un_in[c], vn = fs.vn_in[c], hu = f.hu[c],
                 hv = f.hv[c], ht = f.ht[c];
    wide |= out_of_range(sn) | out_of_range(un) | out_of_range(vn) | out_of_range(hu) |
            out_of_range(hv) | out_of_range(ht);
    A(A_SN, t) = sn;
    A(A_UN, t) = un;
    A(A_VN, t) = vn;
    A(A_HU, t) = hu;
    A(A_HV, t) = hv;
    A(A_HT, t) = ht;
    mk[t] = f.tmask[c];
    B(B_AREA_SSH, t) = mlc<IC>(sn, k.f_area_t);
  }
  // what the update will read from global memory, into L2 meanwhile: one line
  // (16 doubles) per thread (2048^2: 615 -> 597 us)
  for (int t = tid; t < 4 * TY * (TX / 16); t += NTHREADS) {
    const int l = t % (TX / 16), r = t / (TX / 16) % TY, a = t / (TX / 16 * TY);
    const double* base = a == 0   ? f.d_hu
                         : a == 1 ? f.d_hv
                                  : reinterpret_cast<const double*>(a == 2 ? f.r_hu : f.r_hv);
    asm volatile("prefetch.global.L2 [%0];" ::"l"(
        base + min(j0 + r, jmax) * W + min(i0 + 16 * l, imax)));
  }
  bool any_wide = __syncthreads_or(wide);
  if (!any_wide) any_wide = __syncthreads_or(tile_faces<T, false>(f, d, k, i0, j0, smem));
  if (!any_wide) {
    tile_update<T, IC, false, SUMS>(f, fs, d, k, i0, j0, smem);
  } else {
    for (int t = tid; t < S0; t += NTHREADS) B(B_AREA_SSH, t) = k.area_t * A(A_SN, t);
    __syncthreads();
    tile_faces<T, true>(f, d, k, i0, j0, smem);
    __syncthreads();
    tile_update<T, IC, true, SUMS>(f, fs, d, k, i0, j0, smem);
  }

  // ---- general cells: the reference's per-point code, in its order ----
  const int ngen = *gcount;
  for (int g = tid; g < ngen; g += NTHREADS) {
    const int row = glist[g] / TX, col = glist[g] - row * TX;
    if (APART)
      general_in_tile_apart<T>(f, fs, d, p, k, tide, i0 + col, j0 + row, i0, j0);
    else
      general_in_tile<T>(f, fs, d, p, k, tide, i0 + col, j0 + row, i0, j0);
  }
#undef A
#undef B
}

bool in_fast_range(double d) {
  return d > 0.0 && d >= 0x1p-100 && d <= 0x1p100;
}

// c as mul_bounded's factor (host side).
inline IntFactor int_factor(double c) {
  if (!in_fast_range(c)) return IntFactor{0, 0};
  unsigned long long b;
  memcpy(&b, &c, sizeof b);
  const unsigned long long m = (b & 0xfffffffffffffULL) | (1ULL << 52);
  if (m & ((1ULL << 21) - 1)) return IntFactor{0, 0};  // more than 32 significant bits
  // the product's exponent field: x's plus c's unbiased exponent (plus the
  // leading bit, added there); minus one for q's own leading bit
  return IntFactor{(unsigned)(m >> 21), ((unsigned)((int)(b >> 52) - 1023) - 1u) << 20};
}

inline Factor factor(double c) { return Factor{c, int_factor(c)}; }

// d as div_const's divisor (host side).
inline IntDivisor int_divisor(double d) {
  unsigned long long b;
  memcpy(&b, &d, sizeof b);
  const unsigned long long md = (b & 0xfffffffffffffULL) | (1ULL << 52);
  return IntDivisor{d, md, recip64(md), (unsigned)(1021 - (int)(b >> 52 & 0x7ff)) << 20};
}

// The fast path's constants for one domain (host side).
inline FastConst make_fast_const(const Scalars& s, const UniformMetrics& um) {
  FastConst k;
  k.area_t = um.area_t, k.area_u = um.area_u, k.area_v = um.area_v;
  k.dx_u = um.dx_u, k.dx_v = um.dx_v, k.dx_t = um.dx_t;
  k.dy_u = um.dy_u, k.dy_v = um.dy_v, k.dy_t = um.dy_t;
  k.dxv2 = um.dx_v + um.dx_v;
  k.dyu2 = um.dy_u + um.dy_u;
  k.cor_u = 2. * s.omega * um.sin_u;
  k.cor_v = 2. * s.omega * um.sin_v;
  k.neg_g = -s.g;
  k.g = s.g;
  k.rdt = s.rdt;
  k.visc = s.visc;
  const double fric = 1.0 + s.cbfr * s.rdt;
  const double divisors[8] = {k.area_t, k.area_u, k.area_v, k.dx_t, k.dy_t,
                              k.dxv2,   k.dyu2,   fric};
  bool fast = true;
  for (double v : divisors) fast = fast && in_fast_range(v);
  k.fast_div = fast ? 1 : 0;
  k.q_area_t = int_divisor(k.area_t), k.q_area_u = int_divisor(k.area_u);
  k.q_area_v = int_divisor(k.area_v), k.q_dx_t = int_divisor(k.dx_t);
  k.q_dy_t = int_divisor(k.dy_t), k.q_dxv2 = int_divisor(k.dxv2);
  k.q_dyu2 = int_divisor(k.dyu2), k.q_fric = int_divisor(fric);
  k.neg_cor_v = -k.cor_v;
  k.f_area_t = factor(k.area_t), k.f_rdt = factor(k.rdt);
  k.f_dy_u = factor(k.dy_u), k.f_dx_v = factor(k.dx_v);
  k.f_hdx_u = factor(0.5 * k.dx_u), k.f_hdy_v = factor(0.5 * k.dy_v);
  k.f_U = factor(0.5 * k.dy_t), k.f_V = factor(0.5 * k.dx_t);
  k.f_Uw = factor(0.125 * k.dyu2), k.f_Vs = factor(0.125 * k.dxv2);
  k.f_cor_area_u = factor(0.25 * k.area_u), k.f_cor_area_v = factor(0.25 * k.area_v);
  k.q_2area_u = int_divisor(2.0 * k.area_u), k.q_2area_v = int_divisor(2.0 * k.area_v);
  const Factor* all[12] = {&k.f_area_t, &k.f_rdt, &k.f_dy_u, &k.f_dx_v, &k.f_hdx_u, &k.f_hdy_v,
                           &k.f_U, &k.f_V, &k.f_Uw, &k.f_Vs, &k.f_cor_area_u, &k.f_cor_area_v};
  k.int_mul = 1;
  for (const Factor* q : all) k.int_mul &= q->i.co != 0;
  bool bounded = fast;
  for (double v : {k.area_t, k.area_u, k.area_v, k.dx_u, k.dx_v, k.dx_t, k.dy_u, k.dy_v, k.dy_t,
                   k.dxv2, k.dyu2, k.rdt, fric})
    bounded = bounded && v >= 0x1p-40 && v <= 0x1p40;
  for (double v : {k.visc, k.cor_u, k.cor_v, k.neg_g}) {
    const double a = v < 0 ? -v : v;
    bounded = bounded && (a == 0.0 || (a >= 0x1p-40 && a <= 0x1p40));
  }
  k.bounded = bounded ? 1 : 0;
  return k;
}

}  // namespace
}  // namespace nl2d
