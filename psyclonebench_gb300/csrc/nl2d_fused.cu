// Fused NEMOLite2D FP64 time step: one sm_103a kernel per step.
//
// What one launch does, per cell of the copy region [xs-1,xe+1] x [ys-1,ye]
// (psykal_cpp/time_step.cpp:114-122), in the reference's operation order:
//   continuity + bc_ssh          -> sshn_out   (interior cells)
//   momentum_u + bc_solid_u + bc_flather_u -> un_out
//   momentum_v + bc_solid_v + bc_flather_v -> vn_out
// The state that crosses HBM is (sshn_t, un, vn) in ping-pong buffers,
// which replaces the three field copies.  sshn_u / sshn_v are recomputed
// from sshn_t with next_sshu / next_sshv's own operations
// (time_update_kern.c:90-155): those kernels are their only writers, so the
// recomputed values are bit-identical to the stored ones; faces outside
// their range keep their stored (never-updated) value and are read from the
// sshn_u / sshn_v arrays.  The recomputed face values of a tile and of the
// faces around it are staged in shared memory once and shared by the
// continuity and both momentum updates.
//
// Preconditions, checked on the host before this path is used:
//  * the state is "step-consistent": at least one reference-structured step
//    has run since the last host upload, so un == ua, vn == va and
//    sshn_t == ssha_t on the copy region and the faces that no kernel writes
//    hold the same value in both ping-pong buffers;
//  * every grid metric array is uniform (values taken as scalars);
//  * no Flather face reads another Flather face (the reference's serial
//    Flather loops then equal a parallel update).
//
// Built with -fmad=false, as the reference oracle is with
// -ffp-contract=off: results are bit-identical to the reference serial build.
#include <type_traits>

#include "nl2d_fused_tile.cuh"
#include "nl2d_intfp.cuh"

namespace nl2d {
namespace {

// 32 x 8 cells, one per thread, three CTAs per SM (80 registers): the integer
// forms' long dependency chains need warps more than they need a second cell
// per thread (2048^2: 32 x 16 and two CTAs 597 us, 16 x 16 and three 540,
// 32 x 12 and two CTAs of 384 threads 565, 32 x 8 and two 620, three 537).
using T = Tile<32, 8, 256, 3>;
// Domains too small to give every SM two of those take 16 x 8 cells and 128
// threads: twice the tiles, the same bits (the arithmetic does not depend on
// the shape).  32 x 8 and 16 x 8, us per step: 256^2 (256 tiles of 32 x 8) 17.7 /
// 15.0, 384 x 256 (384) 19.1 / 21.5, 512 x 256 (512) 24.9 / 25.1, 1024 x 512
// (2048) 75.4 / 87.3.
using SmallTile = Tile<16, 8, 128, 4>;

// One step of copy-region rows [ja, jb).  The first nring blocks take the
// ring's cells in those rows, rc parts of them each (one per thread: their
// long FP64 chains start first and run beside the tiles); the others one tile
// each of the ntx per row of tiles, from tile row row0.
template <class TT, bool IC, bool SUMS>
__global__ void __launch_bounds__(TT::NTHREADS, TT::kMinBlocks)
    k_fused_step(const __grid_constant__ Fields f, const __grid_constant__ FusedState fs,
                 const __grid_constant__ Dims d, const __grid_constant__ Scalars p,
                 const __grid_constant__ FastConst k, const double* __restrict__ tide_table,
                 int tide_index, double tide, int row0, int ntx, int ja, int jb, int nring,
                 int rc) {
  extern __shared__ double smem[];
  const double td = tide_table ? tide_table[tide_index] : tide;
  if ((int)blockIdx.x < nring) {
    const int tid = threadIdx.y * TT::TX + threadIdx.x, g = blockIdx.x * rc + tid;
    const int n = ring_count(d, ja, jb);
    if (tid < rc && g < kParts * n) {
      const int part = g / n;
      int i, j;
      ring_pos(d, ja, jb, g - part * n, i, j);
      general_at(f, fs, d, p, k, td, part, i, j);
    }
    return;
  }
  const int t = blockIdx.x - nring, by = t / ntx, bx = t - by * ntx;
  // (in line, the general cells' code made large domains without land slower:
  // 1024^2 146.7 -> 151.9 us, 2048^2 560 -> 572; with 10 % of the cells dry faster,
  // 371 -> 361; small domains 13.4 -> 13.1, with land 22.8 -> 22.1)
  fused_tile<TT, IC, SUMS, std::is_same<TT, T>::value>(f, fs, d, p, k, td, d.xs + 1 + bx * TT::TX,
                                                       d.ys + 1 + (row0 + by) * TT::TY, smem);
}

int tiles_over(int n, int t) { return n > 0 ? (n + t - 1) / t : 0; }
int interior_x(const Dims& d) { return d.xe - d.xs - 1; }
int interior_y(const Dims& d) { return d.ye - d.ys - 1; }

bool small_tiles(const Dims& d) {
  return (long long)tiles_over(interior_x(d), T::TX) * tiles_over(interior_y(d), T::TY) <
         2LL * 152;
}
int tile_height(const Dims& d) { return small_tiles(d) ? SmallTile::TY : T::TY; }

template <class TT>
void launch_rows(const Fields& f, const FusedState& fs, const Dims& d, const Scalars& s,
                 const UniformMetrics& um, double tide, const double* tide_table, int tide_index,
                 int row0, int row1, cudaStream_t st) {
  if (row1 <= row0) return;
  const int ja = fused_step_first_row(d, row0), jb = fused_step_first_row(d, row1);
  const int ntx = tiles_over(interior_x(d), TT::TX);
  const int nty = interior_y(d) > 0 ? row1 - row0 : 0;
  // One warp of the ring's parts per block until that would be more than a
  // block per SM: each is ~100 dependent FP64 operations.
  const int nr = kParts * ring_count(d, ja, jb);
  int rc = 32;
  while (rc < TT::NTHREADS && nr > rc * 152) rc *= 2;
  const int nring = (nr + rc - 1) / rc;
  const FastConst k = make_fast_const(s, um);
  auto step = k.int_mul ? k_fused_step<TT, true, true> : k_fused_step<TT, false, true>;
  // (one form without the depth sums must do: it is for the few registrations
  // that fill the memory; a branch in the others would cost all 1 %)
  if (!f.depth_sums()) step = k_fused_step<TT, false, false>;
  step<<<nring + ntx * nty, dim3(TT::TX, TT::RPP), TT::kSmemBytes, st>>>(
      f, fs, d, s, k, tide_table, tide_index, tide, row0, ntx, ja, jb, nring, rc);
}

void set_step_attrs() {
  static bool attr_set = false;
  if (!attr_set) {
    for (auto* fn : {k_fused_step<T, false, true>, k_fused_step<T, true, true>,
                     k_fused_step<T, false, false>})
      cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::kSmemBytes);
    for (auto* fn : {k_fused_step<SmallTile, false, true>, k_fused_step<SmallTile, true, true>,
                     k_fused_step<SmallTile, false, false>})
      cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)SmallTile::kSmemBytes);
    attr_set = true;
  }
}

}  // namespace

int fused_step_tile_rows(const Dims& d) {
  const int n = interior_x(d) > 0 ? tiles_over(interior_y(d), tile_height(d)) : 0;
  return n > 0 ? n : 1;  // without an interior: the ring alone
}

int fused_step_first_row(const Dims& d, int row) {
  if (row <= 0) return d.ys - 1;
  if (row >= fused_step_tile_rows(d)) return d.ye + 1;
  return d.ys + 1 + row * tile_height(d);
}

void launch_fused_step_rows(const Fields& f, const FusedState& fs, const Dims& d,
                            const Scalars& s, const UniformMetrics& um, double tide, int row0,
                            int row1, cudaStream_t st) {
  set_step_attrs();
  if (small_tiles(d))
    launch_rows<SmallTile>(f, fs, d, s, um, tide, nullptr, 0, row0, row1, st);
  else
    launch_rows<T>(f, fs, d, s, um, tide, nullptr, 0, row0, row1, st);
}

void launch_fused_step(const Fields& f, const FusedState& fs, const Dims& d,
                       const Scalars& s, const UniformMetrics& um, double tide,
                       const double* tide_table, int tide_index, cudaStream_t st) {
  set_step_attrs();
  const int rows = fused_step_tile_rows(d);
  if (small_tiles(d))
    launch_rows<SmallTile>(f, fs, d, s, um, tide, tide_table, tide_index, 0, rows, st);
  else
    launch_rows<T>(f, fs, d, s, um, tide, tide_table, tide_index, 0, rows, st);
}

namespace {

// The momentum denominators h + ssha (not stored where dh is null) and their
// 64-bit reciprocals, 0 where the depth lies outside [2^-100, 2^100] (the
// kernel then divides).
__global__ void k_depth_reciprocal(const double* __restrict__ h,
                                   const double* __restrict__ ssha, double* __restrict__ dh,
                                   unsigned long long* __restrict__ r, long long n) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    const double dd = h[t] + ssha[t];
    if (dh) dh[t] = dd;
    r[t] = recip64_of(dd);
  }
}

}  // namespace

void launch_depth_reciprocals(const Fields& f, const Dims& d, cudaStream_t st, int row0,
                              int row1) {
  if (row1 < 0) row1 = d.height;
  const size_t o = (size_t)row0 * d.width;
  const long long n = (long long)(row1 - row0) * d.width;
  if (n <= 0) return;
  double* du = f.depth_sums() ? f.d_hu + o : nullptr;
  double* dv = f.depth_sums() ? f.d_hv + o : nullptr;
  k_depth_reciprocal<<<152 * 8, 256, 0, st>>>(f.hu + o, f.ssha_u + o, du, f.r_hu + o, n);
  k_depth_reciprocal<<<152 * 8, 256, 0, st>>>(f.hv + o, f.ssha_v + o, dv, f.r_hv + o, n);
}

}  // namespace nl2d

// ---- self-test of the exact helpers against the plain IEEE operations ----
namespace nl2d {
namespace {

__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
  z += 0x9e3779b97f4a7c15ULL;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
  return z ^ (z >> 31);
}

// A double from 64 random bits: mostly finite values with exponents across
// the whole normal range, plus zeros, subnormals and non-finite values.
__device__ __forceinline__ double sample(unsigned long long z) {
  const unsigned sel = (unsigned)(z >> 59);  // 0..31
  long long b = (long long)(z & 0x800fffffffffffffULL);
  if (sel == 0) return from_bits(b & 0x8000000000000000LL);        // +-0
  if (sel == 1) return from_bits(b);                                // subnormal
  if (sel == 2) return from_bits(b | 0x7ff0000000000000LL);         // inf / nan
  const long long ex = 1 + (long long)((z >> 40) % 2046ULL);
  return from_bits(b | (ex << 52));
}

__global__ void k_selftest_exact(long long n, unsigned long long seed, IntDivisor v,
                                 IntFactor fac, unsigned long long* bad) {
  const double d = v.d;
  unsigned long long nd = 0, nh = 0, nu = 0;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    const unsigned long long z = mix64(seed ^ (unsigned long long)t);
    const double x = sample(z);
    // division: finite quotients must agree bit for bit
    const double q_ref = x / d;
    for (const double q : {div_const(x, v), div_depth(x, d, v.rc)})
      if (bits(q_ref) != bits(q) && !(q_ref != q_ref && q != q)) nd++;
    // the bounded forms on zeros and normal operands with normal results
    if (!beyond(x, 900, 900)) {
      if (bits(div_bounded(x, v)) != bits(q_ref) || bits(div_bounded(x, d, v.rc)) != bits(q_ref))
        nd++;
      // the product with d (counted with the quotients), where d has that form
      if (fac.co != 0 && bits(mul_bounded(x, fac)) != bits(x * d)) nd++;
    }
    // Quotients within ~2^-53 ulp of a midpoint: RN((Q + ulp(Q)/2) * d) and
    // its neighbours; quotients at and next to a power of two.
    {
      const unsigned long long y = mix64(z + 3);
      const long long eq = (long long)((y >> 40) % 1201ULL) - 600;  // Q in [2^-600, 2^601)
      long long qb = (long long)(y & 0x800fffffffffffffULL) | ((eq + 1023) << 52);
      if ((y >> 38) & 1) qb &= (long long)0x8000000000000000ULL | (0x7ffLL << 52);  // +-2^eq
      const double Q = from_bits(qb);
      const double h = d * from_bits((eq - 53 + 1023) << 52);      // d * ulp(Q) / 2, exact
      const double xm = fma(Q, d, qb < 0 ? -h : h);
      const long long nudge = (long long)((y >> 32) & 7) - 3;
      const double cand[3] = {xm, from_bits(bits(xm) + nudge), from_bits(bits(Q * d) + nudge)};
      for (int c = 0; c < 3; c++) {
        const double xr = cand[c] / d;
        if (bits(xr) != bits(div_const(cand[c], v))) nd++;
        if (bits(xr) != bits(div_depth(cand[c], d, v.rc))) nd++;
      }
    }
    // Quotients at and beside the midpoints of the subnormals: (2c + 1)
    // 2^-1075 d for c of every length, and its neighbours.
    {
      const unsigned long long y = mix64(z + 4);
      const unsigned long long c = (y >> 12) >> (y & 63);
      const long long nudge = (long long)((y >> 6) & 7) - 3;
      const double xm = ((double)(2 * c + 1) * 0x1p-600) * d * 0x1p-475;
      const double cand[3] = {xm, -xm, from_bits(bits(xm) + nudge)};
      for (int i = 0; i < 3; i++) {
        const double xr = cand[i] / d;
        const bool nan = xr != xr;
        if (!nan && bits(xr) != bits(div_const(cand[i], v))) nd++;
        if (!nan && bits(xr) != bits(div_depth(cand[i], d, v.rc))) nd++;
      }
    }
    const double h_ref = 0.5 * x, h = half(x);
    if (bits(h_ref) != bits(h) && !(h_ref != h_ref && h != h)) nh++;
    const double p = sample(mix64(z + 1)), w = sample(mix64(z + 2));
    const double u_ref = (0.5 - copysign(0.5, w)) * x + (0.5 + copysign(0.5, w)) * p;
    // products (counted with the picks): of x and p, and of moderate operands
    // with full, short and trailing significands
    {
      auto wrong = [](double a, double c) {
        return !beyond(a, 1022, 1024) && !beyond(c, 1022, 1024) && !beyond(a * c, 1022, 1024) &&
               ((a * c != 0.0) || a == 0.0 || c == 0.0) && bits(mul_bounded(a, c)) != bits(a * c);
      };
      const unsigned long long y = mix64(z + 5);
      const double f = from_bits((long long)((y & 0x800fffffffffffffULL) |
                                             (1000ULL + (y >> 53) % 40) << 52));
      const double s1 = from_bits((bits(f) >> (y % 53)) << (y % 53));  // a short significand
      const double g = from_bits((bits(x) & 0x800fffffffffffffLL) | (1020LL << 52));
      if (wrong(x, p) || wrong(f, g) || wrong(g, s1) || wrong(s1, s1)) nu++;
    }
    const double u = upwind(w, x, p);
    if (bits(u_ref) != bits(u) && !(u_ref != u_ref && u != u)) nu++;
    if (!beyond(x, 1022, 1024) && !beyond(p, 1022, 1024) && bits(upwind_bounded(w, x, p)) != bits(u_ref)) nu++;
  }
  if (nd) atomicAdd(&bad[0], nd);
  if (nh) atomicAdd(&bad[1], nh);
  if (nu) atomicAdd(&bad[2], nu);
}

// Pairs for the integer add / multiply: generic samples (zeros, subnormals,
// infinities and NaNs included), operands a few binades apart with either
// sign (alignment shifts of 0..70 bits), near-cancelling pairs (the partner
// is -a with its low significand bits changed), and products near the
// bottom and top of the normal range.
__device__ void intfp_pair(unsigned long long z, double& a, double& b) {
  a = sample(z);
  const unsigned long long w = mix64(z + 7);
  const unsigned mode = (unsigned)(w >> 61);  // 0..7
  if (mode <= 2) {
    b = sample(mix64(z + 3));
    return;
  }
  const long long ab = bits(a);
  const int ea = (int)((ab >> 52) & 0x7ff);
  long long bb = (long long)(mix64(z + 5) & 0x800fffffffffffffULL);
  if (mode <= 4) {  // exponent within +-70 of a's
    int eb = ea + (int)((w >> 20) % 141) - 70;
    eb = eb < 1 ? 1 : (eb > 2046 ? 2046 : eb);
    b = from_bits(bb | ((long long)eb << 52));
  } else if (mode == 5) {  // -a with the low 1..52 significand bits replaced
    const int k = 1 + (int)((w >> 20) % 52);
    const long long m = (1LL << k) - 1;
    b = from_bits(((ab ^ (long long)0x8000000000000000ULL) & ~m) | (bb & m));
  } else {  // a product near an edge of the normal range
    const int target = (mode == 6) ? (int)((w >> 20) % 60) - 5 : 2046 - (int)((w >> 20) % 60);
    int eb = target - ea + 1023;
    eb = eb < 1 ? 1 : (eb > 2046 ? 2046 : eb);
    b = from_bits(bb | ((long long)eb << 52));
  }
}

__global__ void k_selftest_intfp(long long n, unsigned long long seed,
                                 unsigned long long* bad) {
  unsigned long long na = 0, nm = 0;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    double a, b;
    intfp_pair(mix64(seed ^ (unsigned long long)t), a, b);
    const double s_ref = a + b, s = dadd_i(a, b);
    if (bits(s_ref) != bits(s) && !(s_ref != s_ref && s != s)) na++;
    const double p_ref = a * b, p = dmul_i(a, b);
    if (bits(p_ref) != bits(p) && !(p_ref != p_ref && p != p)) nm++;
  }
  if (na) atomicAdd(&bad[0], na);
  if (nm) atomicAdd(&bad[1], nm);
}

}  // namespace
}  // namespace nl2d

// Test hook (no reference counterpart): counts, over n sampled operand
// pairs, where the integer-pipe add and multiply (dadd_i, dmul_i) differ
// from the FP64 instructions; out[2] receives the two counts.
extern "C" int nl2d_selftest_intfp(long long n, unsigned long long seed, long long* out) {
  unsigned long long* bad = nullptr;
  if (!out || n < 0) return 2;
  if (cudaMalloc(&bad, 2 * sizeof(unsigned long long)) != cudaSuccess) return 1;
  cudaMemset(bad, 0, 2 * sizeof(unsigned long long));
  nl2d::k_selftest_intfp<<<152 * 16, 256>>>(n, seed, bad);
  unsigned long long h[2] = {0, 0};
  const cudaError_t e = cudaMemcpy(h, bad, sizeof h, cudaMemcpyDeviceToHost);
  cudaFree(bad);
  if (e != cudaSuccess) return 1;
  out[0] = (long long)h[0];
  out[1] = (long long)h[1];
  return 0;
}

// Test hook (no reference counterpart): counts, over n sampled doubles x,
// the inputs where the exact helpers of the fused step differ from the IEEE
// expressions they replace: x / d (and x * d, for a d of at most 32
// significant bits), 0.5 * x and the upwind pick.  d must be
// in [2^-100, 2^100].  out[3] receives the three mismatch counts.
extern "C" int nl2d_selftest_exact(long long n, unsigned long long seed, double d,
                                   long long* out) {
  unsigned long long* bad = nullptr;
  if (!(d >= 0x1p-100 && d <= 0x1p100)) return 2;
  if (cudaMalloc(&bad, 3 * sizeof(unsigned long long)) != cudaSuccess) return 1;
  cudaMemset(bad, 0, 3 * sizeof(unsigned long long));
  nl2d::k_selftest_exact<<<152 * 16, 256>>>(n, seed, nl2d::int_divisor(d), nl2d::int_factor(d),
                                             bad);
  unsigned long long h[3] = {0, 0, 0};
  const cudaError_t e = cudaMemcpy(h, bad, sizeof h, cudaMemcpyDeviceToHost);
  cudaFree(bad);
  if (e != cudaSuccess) return 1;
  for (int k = 0; k < 3; k++) out[k] = (long long)h[k];
  return 0;
}
