// Learned emulator kernels: a 3x3 convolution as an implicit GEMM on the
// 5th-generation tensor cores (tcgen05, BF16 operands, FP32 accumulation in
// tensor memory), plus the small elementwise kernels training needs.
//
// Layouts.  Activations are NHWC BF16 with the channel count padded to a
// multiple of 16; weights are [tap][Cout][Cin] BF16 (tap = 3*dy + dx,
// dy, dx in 0..2 for offsets -1..1), Cin contiguous.  The GEMM of one CTA:
//   D[m][n] = sum over tap, k of A[m][(tap, k)] * B[n][(tap, k)]
// with m = 128 consecutive output pixels of one image row, n = output
// channel, k = input channel, A = the input shifted by the tap (zero
// outside the image).  D lives in tensor memory (128 lanes x Cout FP32
// columns); operands are staged in shared memory in the no-swizzle K-major
// core-matrix layout (8 rows x 16 bytes per core matrix, core matrices
// adjacent along K 128 bytes apart, along M/N 16*Cin bytes apart).
//
// The backward pass reuses the same kernel: the input gradient is the
// convolution of the output gradient with the tap-flipped, channel-
// transposed weights.  The weight gradient is a GEMM over pixels, on the
// tensor cores too (k_conv_wgrad_pipe).
//
// Every wait on an mbarrier is bounded; on timeout the kernel records an
// error flag, ends its roles' loops, waits for the MMAs in flight, frees its
// tensor memory and returns.
#include <cuda_bf16.h>
#include <algorithm>
#include <cstdint>
#include <mutex>
#include <type_traits>

#include "../../include/nl2d_gpu.h"

namespace nl2d {
namespace emu {
namespace {

constexpr int kTileM = 128;       // pixels per CTA (one row segment)
constexpr long long kMaxWaitCycles = 1LL << 31;  // ~1 s at 2 GHz

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// Shared-memory matrix descriptor (tcgen05): start address, leading (K)
// byte offset, stride (M/N) byte offset, descriptor version 1, no swizzle.
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
  d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;
  return d;
}

// Instruction descriptor of tcgen05.mma kind::f16: FP32 accumulator, BF16
// A and B, both K-major, N = n, M = 128.
__host__ __device__ constexpr uint32_t idesc_bf16(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(kTileM >> 4) << 24);
}

// Byte offset of element (row, k) of a K-major operand with `cin` columns.
__device__ __forceinline__ uint32_t core_off(int row, int k, int cin) {
  return (uint32_t)((row >> 3) * (cin * 16) + (k >> 3) * 128 + (row & 7) * 16 + (k & 7) * 2);
}

// Pixels staged per image row: the 128 of the tile plus one on each side,
// rounded up to a multiple of 8 (one core-matrix column of pixels).
constexpr int kRowPix = 136;

// ---- 3x3 convolution ------------------------------------------------------
//
// Implicit GEMM on the tensor cores: M = 128 pixels of one image row, N =
// output channels, K = input channels.  With one MMA per tap the tensor core's
// operand reads from shared memory were the largest item (62 % of its data
// path's time), so an input row is read once for all three output rows it
// enters: with the weights of dy = 2, 1, 0 side by side
// (N = 3 cout), input row y adds to output rows y-1, y and y+1 in one MMA per
// dx and 16 channels, their accumulators lying in adjacent column blocks of a
// ring in tensor memory: 9 MMAs of N = 144 per row at 48 -> 48 channels
// instead of 27 of N = 48.  (The ring's end splits an MMA in two, and the new
// row's block takes its first MMA apart, to start from zero.)  16 x 256^2: 88.1
// -> 67.3 us.  Of an SM's active clocks the operand reads now take 37 %, the
// tensor core's data path 58 %, its arithmetic 32 %, DRAM 37 %: nothing is full;
// which hand-off between the roles the rest waits on has not been told apart.
//
// The weights stay in shared memory for the CTA's lifetime.  A staged input
// row keeps each 8-channel group of its pixels 16 bytes apart, so the operand
// of tap dx is the row started dx pixels (16 * dx bytes) later: a descriptor
// offset, no per-tap copies.  Warp-specialised and persistent: a CTA takes an
// equal, contiguous share of the rows of all 128-pixel columns.  Roles:
//   warps 0-3  epilogue: TMEM -> bias, ReLU -> BF16 / FP32 stores
//   warp 4     one thread issues the MMAs of an input row once it is staged
//              and the new output row's accumulator block is free
//   warps 5-7  stage input rows into a ring of slots by cp.async
// Hand-offs are mbarriers: full[slot] (stagers -> MMA), empty[slot] (MMA
// completion -> stagers), done[block] (MMA completion -> epilogue),
// drained[block] (epilogue -> MMA).  Every wait is bounded (kMaxWaitCycles);
// one that runs out sets the error flag and a shared abort flag that ends
// every role's loop, a whole warp at a time (warp_wait), and the MMA thread
// waits for its last commit before the tensor memory is freed.
constexpr int kConvSlots = 5;  // the input ring
constexpr int kConvDepth = 2;  // rows in flight (four: 68.2 us, two: 66.3)
constexpr int kConvMaxBlocks = 8;
constexpr int kPipeThreads = 256;
constexpr int kEpiWarps = 4;
constexpr int kStageThreads = 96;  // warps 5-7
constexpr uint32_t kLboX = kRowPix * 16 + 16;  // next 8 input channels (padded: banks)

// Accumulator blocks of cout columns (at least four: three being summed, one
// being drained) and the tensor memory they take: two CTAs share an SM's 512
// columns.
__host__ __device__ constexpr int conv_blocks(int cout) {
  return 256 / cout < kConvMaxBlocks ? 256 / cout : kConvMaxBlocks;
}
__host__ __device__ constexpr int conv_tmem(int cout) {
  return conv_blocks(cout) * cout <= 128 ? 128 : 256;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("{\n.reg .b64 st;\nmbarrier.arrive.shared::cta.b64 st, [%0];\n}" ::"r"(
                   smem_u32(bar))
               : "memory");
}
// The MMAs and commits below are executed by a whole, converged warp of which
// one elected lane (always the same) issues them: the operands then stay in
// uniform registers (the convolution 72.1 -> 68.2 us against issuing them from
// a branch of one lane).
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile(
      "{\n.reg .pred q;\nelect.sync _|q, 0xffffffff;\n"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}" ::"r"(
          smem_u32(bar))
      : "memory");
}
// [dcol] (+)= A B with M = 128, BF16 operands from shared memory.
__device__ __forceinline__ void tc_mma(uint32_t dcol, uint64_t ad, uint64_t bd, uint32_t idesc,
                                       uint32_t acc) {
  asm volatile(
      "{\n.reg .pred p, q;\nsetp.ne.b32 p, %4, 0;\nelect.sync _|q, 0xffffffff;\n"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(dcol),
      "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
      : "memory");
}
// 16 FP32 columns of 32 tensor-memory lanes; the values are there after
// tcgen05.wait::ld (which the caller puts before their first use).
__device__ __forceinline__ void tmem_ld16(uint32_t (&r)[16], uint32_t ta) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,"
      "%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(ta));
}
// 32 bytes to p: one store where p is 32-byte aligned (`whole`: a whole
// sector per lane), else two.
__device__ __forceinline__ void store_32b(void* p, const uint32_t (&v)[8], int whole) {
  if (whole)
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(v[0]),
                 "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
  else {
    reinterpret_cast<uint4*>(p)[0] = make_uint4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<uint4*>(p)[1] = make_uint4(v[4], v[5], v[6], v[7]);
  }
}
// Waits for the phase with the given parity to complete; false if the wait
// ran out after max_cycles (flag and error set) or another role aborted.  The
// lanes of a warp may be answered differently: see warp_wait.  POLL: without
// the hardware's own wait in each try, so that short limits hold (tests).
template <bool POLL>
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity,
                                          volatile int* abort_flag, int* err,
                                          long long max_cycles) {
  const long long t0 = clock64();
  for (;;) {
    uint32_t ok;
    if constexpr (POLL)
      asm volatile(
          "{\n.reg .pred p;\nmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
          "selp.u32 %0, 1, 0, p;\n}"
          : "=r"(ok)
          : "r"(smem_u32(bar)), "r"(parity)
          : "memory");
    else
      asm volatile(
          "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
          "selp.u32 %0, 1, 0, p;\n}"
          : "=r"(ok)
          : "r"(smem_u32(bar)), "r"(parity)
          : "memory");
    if (ok) return true;
    if (*abort_flag) return false;
    if (clock64() - t0 > max_cycles) {
      *abort_flag = 1;
      atomicExch(err, 1);
      return false;
    }
  }
}

// The waits and tests of the abort flag by which the roles' loops go on, for
// a whole converged warp: one answer for all its lanes.  (The loops' bodies
// hold warp-wide operations, __syncwarp and tcgen05.ld among them; a lane
// that left a loop by itself would leave the others waiting there for ever.)
template <bool POLL>
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                          int* err, long long max_cycles) {
  return __all_sync(0xffffffffu, mbar_wait<POLL>(bar, parity, abort_flag, err, max_cycles));
}
__device__ __forceinline__ bool warp_goes_on(volatile int* abort_flag) {
  return __all_sync(0xffffffffu, !*abort_flag);
}

// The failure path of the bounded waits, exercised on purpose: one thread
// waits on a barrier that nothing arrives on, gives up after max_cycles,
// sets the error flag and returns (err = 2 would mean the phase completed).
__global__ void k_selftest_wait(long long max_cycles, int* err) {
  __shared__ __align__(8) uint64_t bar;
  __shared__ int abort_flag;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  __syncthreads();
  if (threadIdx.x == 0 && mbar_wait<false>(&bar, 0, &abort_flag, err, max_cycles)) atomicExch(err, 2);
}

// A CTA's share of the rows: rows [g, end) of the list of all columns' rows,
// cut into segments of one column each.
struct RowSegments {
  long long g, end;
  int H, segs;
  __device__ RowSegments(int batch, int H_, int segs_) : H(H_), segs(segs_) {
    const long long total = (long long)batch * segs * H;
    g = total * blockIdx.x / gridDim.x;
    end = total * (blockIdx.x + 1) / gridDim.x;
  }
  __device__ bool next(int& img, int& x0, int& y0, int& rows) {
    if (g >= end) return false;
    const long long col = g / H;
    img = (int)(col / segs);
    x0 = (int)(col - (long long)img * segs) * kTileM;
    y0 = (int)(g - col * H);
    rows = (int)(end - g < H - y0 ? end - g : H - y0);
    g += rows;
    return true;
  }
};

// (max_cycles: the limit of the roles' waits for each other in the POLL form.)
template <bool POLL>
__global__ void __launch_bounds__(kPipeThreads)
    k_conv3x3_pipe(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                   const float* __restrict__ bias, __nv_bfloat16* __restrict__ y,
                   float* __restrict__ y32, int batch, int H, int W, int cin, int cout,
                   int relu, int wide_store, long long max_cycles, int* __restrict__ err) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t full_bar[kConvSlots], empty_bar[kConvSlots];
  __shared__ __align__(8) uint64_t done_bar[kConvMaxBlocks], drained_bar[kConvMaxBlocks], last_bar;
  __shared__ __align__(16) float bias_s[64];
  __shared__ uint32_t taddr_slot;
  __shared__ int abort_flag;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int kc = cin >> 3;
  const int blocks = conv_blocks(cout);
  const uint32_t row_bytes = (uint32_t)kc * kLboX;
  const uint32_t b_bytes = 3u * (uint32_t)cout * cin * 2;  // one dx: [dy = 2, 1, 0][cout][cin]
  unsigned char* b_s = smem;
  unsigned char* ring = smem + ((3 * b_bytes + 1023) & ~1023u);
  volatile int* abort_v = &abort_flag;
  const long long max_wait = POLL ? max_cycles : kMaxWaitCycles;

  if (warp == 0) {
    if (conv_tmem(cout) == 128)
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 128;" ::"r"(
          smem_u32(&taddr_slot)));
    else
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;" ::"r"(
          smem_u32(&taddr_slot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int q = 0; q < kConvSlots; q++) {
      mbar_init(&full_bar[q], kStageThreads / 32);
      mbar_init(&empty_bar[q], 1);
    }
    for (int q = 0; q < blocks; q++) {
      mbar_init(&done_bar[q], 1);
      mbar_init(&drained_bar[q], kEpiWarps);
    }
    mbar_init(&last_bar, 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  for (int t = tid; t < 9 * cout * kc; t += kPipeThreads) {
    const int tap = t / (cout * kc), rem = t - tap * cout * kc;
    const int n = rem / kc, ch = rem - n * kc;
    const int dy = tap / 3, dx = tap - 3 * dy;
    const uint4 v =
        *reinterpret_cast<const uint4*>(w + ((size_t)tap * cout + n) * cin + ch * 8);
    *reinterpret_cast<uint4*>(b_s + dx * b_bytes + core_off((2 - dy) * cout + n, ch * 8, cin)) = v;
  }
  if (tid < cout) bias_s[tid] = bias ? bias[tid] : 0.f;
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t taddr = taddr_slot;
  const int segs = W / kTileM;
  RowSegments rs(batch, H, segs);
  int img, x0, y0, rows;
  // Positions in the rings of slots and blocks: the index, and the parity of
  // the phase to wait for.
  struct Pos {
    int at;
    uint32_t par;
  };
  auto next = [](Pos p, int n) {
    const bool wrap = p.at + 1 == n;
    return Pos{wrap ? 0 : p.at + 1, p.par ^ (wrap ? 1u : 0u)};
  };

  if (warp >= 5) {
    // ---- stagers: input rows y0-1 .. y0+rows of every segment, in order.
    // cp.async copies each 16-byte group of 8 channels straight into its
    // ring slot (zero-filled outside the image); consecutive threads take
    // consecutive groups of a pixel, so a warp's copies cover whole lines,
    // and a thread's chunks have the same offsets in every row.  A row is
    // marked full once kConvDepth - 1 younger rows are in flight.
    const int st = tid - 5 * 32;
    constexpr int kX = (8 * kRowPix + kStageThreads - 1) / kStageThreads;  // cin <= 64
    uint32_t dst[kX];
    int off[kX];
    unsigned mine = 0, left = 0, right = 0;  // chunks there are; in the edge columns
#pragma unroll
    for (int k = 0; k < kX; k++) {
      const int t = st + k * kStageThreads, p = t / kc, ch = t - p * kc;
      dst[k] = (uint32_t)(ch * kLboX + p * 16);
      off[k] = (p - 1) * cin + ch * 8;
      if (p < kRowPix) mine |= 1u << k;
      if (p == 0) left |= 1u << k;
      if (p > kTileM) right |= 1u << k;  // pixel x0 + 128 and beyond (only the first is read)
    }
    Pos put{0, 1}, mark{0, 0};
    int ahead = 0;  // rows started and not yet marked full
    bool fresh = true, ok = true;  // the ring's first turn waits for nothing
    auto finish = [&]() {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&full_bar[mark.at]);
      mark = next(mark, kConvSlots);
      ahead--;
    };
    while (ok && rs.next(img, x0, y0, rows) && warp_goes_on(abort_v)) {
      const unsigned in = mine & ~(x0 == 0 ? left : 0u) & ~(x0 + kTileM >= W ? right : 0u);
      const __nv_bfloat16* seg = x + (((size_t)img * H + y0) * W + x0) * cin;
      for (int a = 0; a < rows + 2; a++) {
        const int yy = y0 - 1 + a;
        if (!fresh) ok = warp_wait<POLL>(&empty_bar[put.at], put.par, abort_v, err, max_wait);
        if (!ok) break;
        const unsigned take = yy >= 0 && yy < H ? in : 0u;
        const __nv_bfloat16* src = seg + (long long)(a - 1) * W * cin;
        const uint32_t d0 = smem_u32(ring + put.at * row_bytes);
#pragma unroll
        for (int k = 0; k < kX; k++)
          if (mine >> k & 1u) {
            const bool t = take >> k & 1u;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d0 + dst[k]),
                         "l"(t ? src + off[k] : x), "r"(t ? 16 : 0)
                         : "memory");
          }
        asm volatile("cp.async.commit_group;" ::: "memory");
        put = next(put, kConvSlots);
        if (put.at == 0) fresh = false;
        if (++ahead == kConvDepth) {
          asm volatile("cp.async.wait_group %0;" ::"n"(kConvDepth - 1) : "memory");
          finish();
        }
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    while (ahead > 0 && warp_goes_on(abort_v)) finish();
  } else if (warp == 4) {
    // ---- MMA issuer: the whole warp walks, one lane issues ----
    {
      const uint64_t b_desc0 = smem_desc(smem_u32(b_s), 128, (uint32_t)cin * 16);
      const uint64_t a_desc0 = smem_desc(smem_u32(ring), kLboX, 128);
      const uint32_t a_kstep = (2 * kLboX) >> 4;
      const uint32_t b_block = ((uint32_t)cout * cin * 2) >> 4;  // one dy's weights
      const int kcq = cin / 16;
      const uint32_t idesc[3] = {idesc_bf16(cout), idesc_bf16(2 * cout), idesc_bf16(3 * cout)};
      // n blocks from column block `at`, weights from dy block `from`
      auto mma = [&](int at, int from, int n, uint64_t ad, uint64_t bd, uint32_t acc) {
        tc_mma(taddr + (uint32_t)(at * cout), ad, bd + (uint64_t)((uint32_t)from * b_block),
               n == 1 ? idesc[0] : (n == 2 ? idesc[1] : idesc[2]), acc);
      };
      Pos in{0, 0};            // the input row's slot
      Pos fresh{0, 1};         // the new output row's block
      Pos oldest{0, 0};        // the block of the oldest output row being summed
      bool first_turn = true, issued = false, ok = true;
      while (ok && rs.next(img, x0, y0, rows) && warp_goes_on(abort_v)) {
        for (int a = 0; a < rows + 2 && ok; a++) {
          // output rows (of the segment) max(0, a-2) .. min(rows-1, a)
          const int lo = a > 2 ? a - 2 : 0, hi = a < rows ? a : rows - 1;
          const int n = hi - lo + 1, from = lo - (a - 2);
          const bool opens = a < rows;
          ok = mbar_wait<POLL>(&full_bar[in.at], in.par, abort_v, err, max_wait);
          if (ok && opens && !first_turn)
            ok = mbar_wait<POLL>(&drained_bar[fresh.at], fresh.par, abort_v, err, max_wait);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const int to_end = blocks - oldest.at;  // blocks before the ring's end
          uint64_t arow = a_desc0 + (uint64_t)((uint32_t)in.at * (row_bytes >> 4));
          uint64_t bdx = b_desc0;
#pragma unroll
          for (int dx = 0; dx < 3; dx++, arow += 1, bdx += b_bytes >> 4) {
            uint64_t ad = arow, bd = bdx;
            for (int kq = 0; kq < kcq; kq++, ad += a_kstep, bd += 256 >> 4) {
              // the new row's block starts from zero: its first MMA apart
              const bool apart = opens && dx == 0 && kq == 0;
              const int m = apart ? n - 1 : n, m1 = m < to_end ? m : to_end;
              if (m1 > 0) mma(oldest.at, from, m1, ad, bd, 1u);
              if (m > m1) mma(0, from + m1, m - m1, ad, bd, 1u);
              if (apart) mma(fresh.at, from + m, 1, ad, bd, 0u);
            }
          }
          issued = true;
          tc_commit(&empty_bar[in.at]);
          in = next(in, kConvSlots);
          if (opens) {
            fresh = next(fresh, blocks);
            if (fresh.at == 0) first_turn = false;
          }
          if (a >= 2) {  // output row a - 2 is complete
            tc_commit(&done_bar[oldest.at]);
            oldest = next(oldest, blocks);
          }
        }
      }
      if (issued) {  // nothing may be in flight when the tensor memory is freed
        tc_commit(&last_bar);
        volatile int never = 0;
        if (!mbar_wait<false>(&last_bar, 0, &never, err, kMaxWaitCycles)) atomicExch(err, 1);
      }
    }
  } else {
    // ---- epilogue: warp w owns accumulator lanes (pixels) 32w .. 32w+31 ----
    Pos blk{0, 0};
    bool ok = true;
    while (ok && rs.next(img, x0, y0, rows) && warp_goes_on(abort_v)) {
      size_t pix = ((size_t)img * H + y0) * W + x0 + warp * 32 + lane;
      for (int o = 0; o < rows; o++, pix += W) {
        ok = warp_wait<POLL>(&done_bar[blk.at], blk.par, abort_v, err, max_wait);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t ta =
            taddr + ((uint32_t)(warp * 32) << 16) + (uint32_t)(blk.at * cout);
        uint32_t r[4][16];
        const int nq = cout >> 4;
#pragma unroll
        for (int q = 0; q < 4; q++)
          if (q < nq) tmem_ld16(r[q], ta + 16 * q);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&drained_bar[blk.at]);  // the values are in registers
#pragma unroll
        for (int q = 0; q < 4; q++) {
          if (q >= nq) break;
          float v[16];
#pragma unroll
          for (int k = 0; k < 16; k += 4) {
            const float4 b4 = *reinterpret_cast<const float4*>(bias_s + 16 * q + k);
            v[k] = __uint_as_float(r[q][k]) + b4.x;
            v[k + 1] = __uint_as_float(r[q][k + 1]) + b4.y;
            v[k + 2] = __uint_as_float(r[q][k + 2]) + b4.z;
            v[k + 3] = __uint_as_float(r[q][k + 3]) + b4.w;
          }
          if (relu)
#pragma unroll
            for (int k = 0; k < 16; k++) v[k] = fmaxf(v[k], 0.f);
          if (y) {
            uint32_t o2[8];
#pragma unroll
            for (int k = 0; k < 8; k++) {
              const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
              o2[k] = *reinterpret_cast<const uint32_t*>(&h);
            }
            store_32b(y + pix * cout + 16 * q, o2, wide_store & 1);
          }
          if (y32) {
#pragma unroll
            for (int h = 0; h < 2; h++) {
              uint32_t o4[8];
#pragma unroll
              for (int k = 0; k < 8; k++) o4[k] = __float_as_uint(v[8 * h + k]);
              store_32b(y32 + pix * cout + 16 * q + 8 * h, o4, wide_store & 2);
            }
          }
        }
        blk = next(blk, blocks);
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == 0) {
    if (conv_tmem(cout) == 128)
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 128;" ::"r"(taddr));
    else
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" ::"r"(taddr));
  }
}

// Tap-flipped, channel-transposed weights for the input gradient:
// wt[8 - tap][ci][co] = w[tap][co][ci].
__global__ void k_flip_transpose(const __nv_bfloat16* __restrict__ w,
                                 __nv_bfloat16* __restrict__ wt, int cout, int cin) {
  const int n = 9 * cout * cin;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    const int tap = t / (cout * cin), rem = t - tap * cout * cin;
    const int co = rem / cin, ci = rem - co * cin;
    wt[((size_t)(8 - tap) * cin + ci) * cout + co] = w[t];
  }
}

// Weight gradient on the tensor cores.  For each tap it is a GEMM over
// pixels, D[co][ci] = sum_p dY[p][co] X[p + off][ci], with both operands
// "MN-major" (channels contiguous per pixel, as the data already is): M =
// output channels, N = input channels, K = pixels.  X is staged as in the
// convolution, so the tap (dy, dx) operand is again a row block started 16 *
// dx bytes later.
//
// One MMA per tap is mostly operand reads from shared memory: an M = 128, N =
// 48 MMA reads 5.6 KB for 48 of its 128 rows' worth of products.  So two
// adjacent rows are stacked on each side (cout <= 64): A = dY rows (r,
// r+1), B = X rows (r, r+1), and the four quadrants of one accumulator are
// dY(r) X(r): dy = 1, dY(r) X(r+1): dy = 2, dY(r+1) X(r): dy = 0, and dY(r+1)
// X(r+1), which is not used (every row meets itself in the first).  As r runs
// over the rows, with zero rows of dY before and after, each quadrant sums
// its tap over all of them: 24 MMAs of N = 96 per row of 48 channels instead
// of 72 of N = 48.  Rows lie in a ring of slots, adjacent rows in adjacent
// slots (slot 0 is staged a second time behind the last).  cout > 64: one row
// of dY, and the nine taps as separate MMAs.
//
// The accumulators stay in tensor memory for the CTA's lifetime; at the end
// each CTA writes its partial sums to its own slot of `part`, and k_sum_parts
// adds the slots in a fixed order, so that the gradient has the same bits on
// every run (atomic additions would sum in whatever order the CTAs finished).
// A CTA (alone on its SM: it holds all 512 TMEM columns) takes an equal,
// contiguous share of the rows of all 128-pixel columns.  Roles:
//   warps 0-6  stage rows of X and dY by cp.async, kWgDepth rows in flight,
//              and add up their dY values for the bias gradient; at the end
//              warps 0-3 move the accumulators out of TMEM
//   warp 7     one thread issues the MMAs
// 48 -> 48 channels at 16 x 256^2: 193 us (9 x N = 48 per row, one row in
// flight in registers) plus 100 us for a separate bias pass and the sums before,
// 100 us with everything now.  Of an SM's active clocks the operand reads take 49
// %, the tensor core's data path 52 %, its arithmetic (an unused quadrant in
// four) 42 %, DRAM 32 %; about 15 us are the launch's start and the accumulators'
// way out, which nothing runs beside.
constexpr int kWgTmemCols = 512;
constexpr int kWgThreads = 256, kWgStagers = kWgThreads - 32;  // the last warp issues
constexpr int kWgDepth = 2;  // rows in flight per CTA (1: 118 us, 2: 99, 3: 101, 4: 104)
constexpr int kWgMaxSlots = 8;
constexpr uint32_t kWgLboY = kTileM * 16 + 16;   // next 8 output channels (padded: banks)
constexpr uint32_t kWgLboX = kLboX;
constexpr size_t kWgMaxSmem = 216 * 1024;

__host__ __device__ constexpr uint32_t idesc_bf16_mn(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) |
         ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kTileM >> 4) << 24);
}
// One slot: a row of dY and a row of X.
__host__ __device__ constexpr uint32_t wg_ybytes(int cout) { return (cout >> 3) * kWgLboY; }
__host__ __device__ constexpr uint32_t wg_xbytes(int cin) { return (cin >> 3) * kWgLboX; }
// dY slots, then X slots, each with the copy of slot 0 where rows are paired;
// an operand of M = 128 reads 16 channel groups from its first row on.
__host__ __device__ constexpr size_t wg_smem(int cin, int cout, int slots) {
  const int n = slots + (cout <= 64 ? 1 : 0);
  const size_t all = (size_t)n * (wg_ybytes(cout) + wg_xbytes(cin));
  const size_t last = (size_t)(slots - 1) * wg_ybytes(cout) + 16 * kWgLboY;
  return all > last ? all : last;
}
// Rows in flight: an MMA step frees a row once the next one (paired) or the
// next two are marked full, which the stagers do depth - 1 rows later.
__host__ __device__ constexpr int wg_depth(int cout, int slots) {
  const int d = slots - (cout <= 64 ? 1 : 2);
  return d < kWgDepth ? d : kWgDepth;
}

template <bool POLL>
__global__ void __launch_bounds__(kWgThreads)
    k_conv_wgrad_pipe(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ dy,
                      float* __restrict__ part, int batch, int H, int W, int cin, int cout,
                      int slots, long long max_cycles, int* __restrict__ err) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t full_bar[kWgMaxSlots], empty_bar[kWgMaxSlots], last_bar;
  __shared__ uint32_t taddr_slot;
  __shared__ int abort_flag, s_issued;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int kc = cin >> 3, kco = cout >> 3;
  const bool pair = cout <= 64;
  const uint32_t ybytes = wg_ybytes(cout), xbytes = wg_xbytes(cin);
  unsigned char* yring = smem;
  unsigned char* xring = smem + (size_t)(slots + (pair ? 1 : 0)) * ybytes;
  const int depth = wg_depth(cout, slots);
  volatile int* abort_v = &abort_flag;
  const long long max_wait = POLL ? max_cycles : kMaxWaitCycles;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&taddr_slot)),
                 "r"(kWgTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int q = 0; q < slots; q++) {
      mbar_init(&full_bar[q], kWgStagers / 32);
      mbar_init(&empty_bar[q], 1);
    }
    mbar_init(&last_bar, 1);
    abort_flag = 0;
    s_issued = 0;
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t taddr = taddr_slot;
  const int segs = W / kTileM;
  const long long nel = 9LL * cout * cin;
  float* mine = part + (size_t)blockIdx.x * (nel + cout);

  if (tid >= kWgStagers) {
    // ---- MMA issuer: the whole warp walks, one lane issues ----
    {
      const uint32_t idesc = idesc_bf16_mn(pair ? 2 * cin : cin);
      RowSegments rs(batch, H, segs);
      bool issued = false, ok = true;
      int img, x0, y0, rows;
      // Ring positions are counted in 32 bits, slot and parity apart, and the
      // slots' descriptors formed by one multiply-add: this thread's work per
      // row is what the tensor core waits for between rows.
      struct Pos {
        int slot;
        uint32_t par;
      };
      auto next = [&](Pos p) {
        const bool wrap = p.slot + 1 == slots;
        return Pos{wrap ? 0 : p.slot + 1, p.par ^ (wrap ? 1u : 0u)};
      };
      auto full = [&](Pos p) {
        return warp_wait<POLL>(&full_bar[p.slot], p.par, abort_v, err, max_wait);
      };
      const uint64_t yd0 = smem_desc(smem_u32(yring), 128, kWgLboY);
      const uint64_t xd0 = smem_desc(smem_u32(xring), 128, kWgLboX);
      // One K-step (16 pixels) of a row after the other, its accumulators in
      // turn.  MN-major, no swizzle: LBO steps along K (8 pixels = 128
      // B), SBO along M / N (the next 8 channels); + 256 / 16 per K-step (the
      // address field never carries: shared addresses stay below 256 KB).
      auto mmas = [&](auto count, uint64_t yd, auto xdesc, uint32_t cols) {
#pragma unroll
        for (int kq = 0; kq < kTileM / 16; kq++)
#pragma unroll
          for (int b = 0; b < decltype(count)::value; b++)
            tc_mma(taddr + (uint32_t)b * cols, yd + (uint64_t)(kq * (256 >> 4)),
                   xdesc(b) + (uint64_t)(kq * (256 >> 4)), idesc, issued || kq > 0 ? 1u : 0u);
      };
      Pos cur{0, 0};  // the ring row of the segment's row y0 - 1, then of each row
      while (ok && rs.next(img, x0, y0, rows) && warp_goes_on(abort_v)) {
        ok = full(cur);
        if (pair) {
          for (int o = 0; o <= rows && ok; o++) {  // rows (cur, nxt)
            const Pos nxt = next(cur);
            ok = full(nxt);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t yd = yd0 + (uint64_t)((uint32_t)cur.slot * (ybytes >> 4));
            const uint64_t xd = xd0 + (uint64_t)((uint32_t)cur.slot * (xbytes >> 4));
            mmas(std::integral_constant<int, 3>{}, yd,
                 [&](int dx) { return xd + (uint64_t)dx; }, (uint32_t)(2 * cin));
            issued = true;
            tc_commit(&empty_bar[cur.slot]);  // no later step of this segment reads cur
            cur = nxt;
          }
        } else {
          Pos mid = next(cur);
          ok = ok && full(mid);
          for (int o = 1; o <= rows && ok; o++) {  // dY row mid, X rows cur, mid, nxt
            const Pos nxt = next(mid);
            ok = full(nxt);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t yd = yd0 + (uint64_t)((uint32_t)mid.slot * (ybytes >> 4));
            const uint64_t xs[3] = {xd0 + (uint64_t)((uint32_t)cur.slot * (xbytes >> 4)),
                                    xd0 + (uint64_t)((uint32_t)mid.slot * (xbytes >> 4)),
                                    xd0 + (uint64_t)((uint32_t)nxt.slot * (xbytes >> 4))};
            mmas(std::integral_constant<int, 9>{}, yd,
                 [&](int tap) { return xs[tap / 3] + (uint64_t)(tap % 3); }, (uint32_t)cin);
            issued = true;
            tc_commit(&empty_bar[cur.slot]);
            cur = mid;
            mid = nxt;
          }
          if (ok) tc_commit(&empty_bar[cur.slot]);
          cur = mid;
        }
        if (ok) tc_commit(&empty_bar[cur.slot]);
        cur = next(cur);
      }
      if (lane == 0) s_issued = (issued && ok) ? 1 : 0;
      __threadfence_block();
      __syncwarp();
      if (issued)
        tc_commit(&last_bar);  // arrives once every MMA above has completed
      else if (lane == 0)
        mbar_arrive(&last_bar);
    }
  } else {
    // ---- stagers.  Consecutive threads take consecutive 16-byte channel
    // groups of a pixel, so a warp's copies cover whole lines; every thread
    // keeps one channel group of dY and so its eight bias sums.  A thread's
    // chunks of a row have the same offsets in every row (formed once: index
    // arithmetic per chunk had the stagers at 700 instructions per warp and
    // row, longer than the row's MMAs).
    const int yg = tid % kco, yl = tid / kco, yL = kWgStagers / kco;  // group, first pixel, step
    const int yn = yl < yL ? (kTileM - yl + yL - 1) / yL : 0;         // its pixels
    const uint32_t ydst = (uint32_t)(yg * kWgLboY + yl * 16);
    const int ysrc = yl * cout + yg * 8;
    constexpr int kX = (6 * kRowPix + kWgStagers - 1) / kWgStagers;  // cin <= 48
    uint32_t xdst[kX];
    int xpix[kX], xsrc[kX];
#pragma unroll
    for (int k = 0; k < kX; k++) {
      const int t = tid + k * kWgStagers, p = t / kc, ch = t - p * kc;
      xpix[k] = p < kRowPix ? p - 1 : -2;  // -2: no chunk
      xdst[k] = (uint32_t)(ch * kWgLboX + p * 16);
      xsrc[k] = (p - 1) * cin + ch * 8;
    }
    float bs[8] = {};
    long long q = 0, done = 0;      // rows started, rows marked full
    int qslot = 0, dslot = 0;       // their slots
    uint32_t qphase = 1;            // parity of empty_bar the next row waits for
    unsigned real = 0;              // bit k: ring row q-1-k carries dY values
    auto finish = [&]() {           // row `done` has landed
      if (real >> (int)(q - 1 - done) & 1u) {
        const unsigned char* src = yring + dslot * ybytes + ydst;
        for (int k = 0; k < yn; k++, src += yL * 16) {
          const uint4 v = *reinterpret_cast<const uint4*>(src);
          const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int e = 0; e < 4; e++) {
            bs[2 * e] += __uint_as_float(w[e] << 16);
            bs[2 * e + 1] += __uint_as_float(w[e] & 0xffff0000u);
          }
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();  // one arrival per warp: 224 serialised ones took longer than the copies
      if (lane == 0) mbar_arrive(&full_bar[dslot]);
      done++;
      if (++dslot == slots) dslot = 0;
    };
    RowSegments rs(batch, H, segs);
    int img, x0, y0, rows;
    bool ok = true;  // this lane's waits; see below
    while (rs.next(img, x0, y0, rows)) {
      unsigned xin = 0;  // bit k: chunk k lies inside the image's columns
#pragma unroll
      for (int k = 0; k < kX; k++)
        if (xpix[k] >= -1 && x0 + xpix[k] >= 0 && x0 + xpix[k] < W) xin |= 1u << k;
      const size_t row0 = ((size_t)img * H + y0) * W + x0;  // the segment's first pixel
      const __nv_bfloat16* yrow_p = dy + row0 * cout + ysrc;
      const __nv_bfloat16* xrow_p = x + row0 * cin;
      for (int a = 0; a < rows + 2; a++) {
        const long long dr = a - 1;
        // A lane whose wait ran out goes through its remaining rows without
        // waits or copies, so that its warp stays whole for finish() without a
        // vote per row (which cost 4 us of 100); the results are not valid then.
        if (q >= slots && ok)
          ok = mbar_wait<POLL>(&empty_bar[qslot], qphase, abort_v, err, max_wait);
        const bool yrow = a >= 1 && a <= rows, xrow = y0 + dr >= 0 && y0 + dr < H;
        const __nv_bfloat16* ys = yrow ? yrow_p + dr * W * cout : dy;
        const __nv_bfloat16* xs = xrow_p + dr * W * cin;
        const int ystep = yrow ? yL * cout : 0;
        for (int copy = qslot; ok && copy <= slots; copy += slots) {  // slot 0: twice, paired
          uint32_t yd = smem_u32(yring + copy * ybytes) + ydst;
          const __nv_bfloat16* yp = ys;
          for (int k = 0; k < yn; k++, yd += yL * 16, yp += ystep)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(yd), "l"(yp),
                         "r"(yrow ? 16 : 0)
                         : "memory");
          const uint32_t xd = smem_u32(xring + copy * xbytes);
#pragma unroll
          for (int k = 0; k < kX; k++)
            if (xpix[k] >= -1) {
              const bool in = xrow && (xin >> k & 1u);
              asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(xd + xdst[k]),
                           "l"(in ? xs + xsrc[k] : x), "r"(in ? 16 : 0)
                           : "memory");
            }
          if (qslot != 0 || !pair) break;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        real = real << 1 | (yrow ? 1u : 0u);
        q++;
        if (++qslot == slots) {
          qslot = 0;
          qphase ^= 1u;
        }
        if (q - done >= depth) {  // all but the newest depth - 1 rows must have landed
          if (depth == 1)
            asm volatile("cp.async.wait_group 0;" ::: "memory");
          else
            asm volatile("cp.async.wait_group 1;" ::: "memory");
          finish();
        }
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    while (done < q) finish();
    // the accumulators: rows 32w .. 32w+31 of M
    volatile int never = 0;
    const bool mmas = warp_wait<false>(&last_bar, 0, &never, err, kMaxWaitCycles);
    if (warp < 4 && mmas && s_issued && warp_goes_on(abort_v)) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int m = warp * 32 + lane;
      const bool second = pair && m >= cout;  // dY row r+1: the tap dy = 0
      const int co = second ? m - cout : m;
      const int ncols = pair ? 6 * cin : 9 * cin;
      // (ncols is a multiple of 48: three loads in flight)
      for (int c0 = 0; c0 < ncols; c0 += 48) {
        uint32_t r[3][16];
#pragma unroll
        for (int l = 0; l < 3; l++)
          tmem_ld16(r[l], taddr + ((uint32_t)(warp * 32) << 16) + (uint32_t)(c0 + 16 * l));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int l = 0; l < 3; l++) {
          const int c = c0 + 16 * l;
          const int blk = c / cin, ci0 = c - blk * cin;  // (dx, X row) or the tap
          int tap = blk;
          if (pair) {
            const int dx = blk >> 1, xr = blk & 1;
            tap = second ? (xr ? -1 : dx) : (xr ? 6 + dx : 3 + dx);
          }
          if (co < cout && tap >= 0)
#pragma unroll
            for (int k = 0; k < 4; k++)
              *reinterpret_cast<float4*>(mine + ((size_t)tap * cout + co) * cin + ci0 + 4 * k) =
                  make_float4(__uint_as_float(r[l][4 * k]), __uint_as_float(r[l][4 * k + 1]),
                              __uint_as_float(r[l][4 * k + 2]), __uint_as_float(r[l][4 * k + 3]));
        }
      }
    }
    // the bias sums, added over the threads of a channel group in thread order
    float* sb = reinterpret_cast<float*>(smem);  // [yL][cout]: the rings are done with
    asm volatile("bar.sync 1, %0;" ::"n"(kWgStagers) : "memory");
    if (yl < yL)
#pragma unroll
      for (int k = 0; k < 8; k++) sb[yl * cout + yg * 8 + k] = bs[k];
    asm volatile("bar.sync 1, %0;" ::"n"(kWgStagers) : "memory");
    for (int c = tid; c < cout; c += kWgStagers) {
      float acc = 0.f;
      for (int r = 0; r < yL; r++) acc += sb[r * cout + c];
      mine[nel + c] = acc;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr),
                 "r"(kWgTmemCols));
}

// out[e] += the sum over the parts' slots of nel + cout values (dw, then db):
// kSumWays threads add a contiguous share of the slots each, in order, and
// their sums are added in order.  (One thread per element made the 1216 bias
// parts of a separate pass 100 us of dependent loads, the 152 weight parts 17.)
constexpr int kSumWays = 8, kSumElems = 32;

// The call's inputs, for k_sum_parts.
struct WgradInputs {
  const __nv_bfloat16 *x, *dy;
  int batch, H, W, cin, cout;
};
// Element e of dw over image rows [r0, r1), by itself: per 128 pixels in FP32,
// these in FP64.  Ends at a NaN.
__device__ __noinline__ double wgrad_element(const WgradInputs& in, long long e, long long r0,
                                             long long r1) {
  const int ci = (int)(e % in.cin), co = (int)(e / in.cin % in.cout),
            tap = (int)(e / ((long long)in.cin * in.cout));
  const int oy = tap / 3 - 1, ox = tap % 3 - 1;
  double sum = 0.0;
  for (long long r = r0; r < r1 && sum == sum; r++) {
    const int y = (int)(r % in.H);
    const bool yin = y + oy >= 0 && y + oy < in.H;
    const __nv_bfloat16* d = in.dy + (size_t)r * in.W * in.cout + co;
    for (int x0 = 0; x0 < in.W; x0 += kTileM) {
      float acc = 0.f;
#pragma unroll 4
      for (int px = x0; px < x0 + kTileM; px++) {
        const bool xin = yin && px + ox >= 0 && px + ox < in.W;
        const float xv =
            xin ? __bfloat162float(in.x[((r + oy) * in.W + px + ox) * in.cin + ci]) : 0.f;
        acc = fmaf(__bfloat162float(d[(size_t)px * in.cout]), xv, acc);
      }
      sum += acc;
    }
  }
  return sum;
}

// direct: the rows were stacked in pairs.  At the ends of a CTA's rows the pair
// holds a zero row of dY, whose products with an infinity or a NaN of X are NaN
// where the gradient has none, so sums that are NaN are formed again without it.
// (Finite inputs: never; the vote takes 1 us of a call's 99.5 at 16 x 256^2.  Six
// blocks per SM, so that 648 run at once: at the 64 registers that
// wgrad_element asks for the call took 1 us more.)
__global__ void __launch_bounds__(kSumWays * kSumElems, 6)
    k_sum_parts(const float* __restrict__ part, int nparts, long long nel, int cout,
                float* __restrict__ dw, float* __restrict__ db,
                const __grid_constant__ WgradInputs in, int direct) {
  __shared__ float sums[kSumWays][kSumElems];
  const int lane = threadIdx.x % kSumElems, way = threadIdx.x / kSumElems;
  const long long n = nel + cout, e = (long long)blockIdx.x * kSumElems + lane;
  const int b0 = (int)((long long)nparts * way / kSumWays),
            b1 = (int)((long long)nparts * (way + 1) / kSumWays);
  float acc = 0.f;
  if (e < n) {
#pragma unroll 8
    for (int b = b0; b < b1; b++) acc += part[(size_t)b * n + e];
  }
  sums[way][lane] = acc;
  __syncthreads();
  float total = sums[0][lane];
#pragma unroll
  for (int w = 1; w < kSumWays; w++) total += sums[w][lane];
  const bool again = direct && e < nel && total != total;
  if (__syncthreads_or(again)) {
    __shared__ double exact[kSumWays][kSumElems];
    const long long rows = (long long)in.batch * in.H;
    exact[way][lane] = again ? wgrad_element(in, e, rows * way / kSumWays,
                                             rows * (way + 1) / kSumWays)
                             : 0.0;
    __syncthreads();
    if (again) {
      double t = exact[0][lane];
      for (int w = 1; w < kSumWays; w++) t += exact[w][lane];
      total = (float)t;
    }
  }
  if (way == 0 && e < n) {
    if (e < nel)
      dw[e] += total;
    else
      db[e - nel] += total;
  }
}

// Scratch for one call's per-CTA partial gradients, which no other call may
// touch until the reduction has read them.  A stream (by its id: handles are
// used again) keeps a buffer of its own, in which its calls follow each other;
// `lock` is held until the call's launches are made, so that two threads'
// launches on one stream do not mix.  The first kPartsStreams streams of a
// device get one (at most 34 MB each); others, and calls under capture, whose
// graphs may run beside their stream, allocate and free in stream order (3 us
// per call) from a pool that keeps kPartsKept bytes.  nl2d_finalize gives all
// of it back.  Memory and pool are made in the relaxed capture mode: in the
// others making them would invalidate a capture, this thread's (a program that
// has called on its own streams so far has no pool yet) or another's.
constexpr int kPartsStreams = 4, kMaxDevices = 64;
constexpr uint64_t kPartsKept = 64ull << 20;
struct PartsKept {
  std::mutex lock;
  cudaMemPool_t pool;
  struct {
    unsigned long long id;
    float* p;
    size_t cap;
  } of[kPartsStreams];
} g_parts[kMaxDevices];

class Parts {
 public:
  Parts(int dev, size_t n, cudaStream_t st) : st_(st) {
    if (dev < 0 || dev >= kMaxDevices) return;
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    if (cudaThreadExchangeStreamCaptureMode(&mode) != cudaSuccess) return;
    take(g_parts[dev], dev, n);
    cudaThreadExchangeStreamCaptureMode(&mode);
  }
  // After the last launch that reads p; false on a CUDA error.
  bool done() { return !ordered_ || cudaFreeAsync(p, st_) == cudaSuccess; }
  float* p = nullptr;  // null: none to be had

 private:
  void take(PartsKept& d, int dev, size_t n) {
    hold_ = std::unique_lock<std::mutex>(d.lock);
    unsigned long long id = 0;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st_, &capture) != cudaSuccess ||
        (capture == cudaStreamCaptureStatusNone && cudaStreamGetId(st_, &id) != cudaSuccess))
      return;
    if (capture == cudaStreamCaptureStatusNone)
      for (auto& e : d.of) {
        if (e.p && e.id != id) continue;
        e.id = id;
        if (e.cap < n) {
          cudaFree(e.p);  // (waits for the stream's calls)
          e.p = nullptr;
          e.cap = 0;
          if (cudaMalloc(&e.p, n * sizeof(float)) != cudaSuccess) return;
          e.cap = n;
        }
        p = e.p;
        return;
      }
    if (!d.pool) {
      cudaMemPoolProps props = {};
      props.allocType = cudaMemAllocationTypePinned;
      props.location.type = cudaMemLocationTypeDevice;
      props.location.id = dev;
      uint64_t kept = kPartsKept;
      if (cudaMemPoolCreate(&d.pool, &props) != cudaSuccess) {
        d.pool = nullptr;
        return;
      }
      cudaMemPoolSetAttribute(d.pool, cudaMemPoolAttrReleaseThreshold, &kept);
    }
    if (cudaMallocFromPoolAsync(&p, n * sizeof(float), d.pool, st_) == cudaSuccess)
      ordered_ = true;
    else
      p = nullptr;
  }
  std::unique_lock<std::mutex> hold_;
  cudaStream_t st_;
  bool ordered_ = false;
};

// dx = (y > 0) ? g : 0 for a ReLU output y (BF16), g FP32 -> BF16.
__global__ void k_relu_bwd(const float* __restrict__ g, const __nv_bfloat16* __restrict__ y,
                           __nv_bfloat16* __restrict__ out, long long n) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x)
    out[t] = __float2bfloat16(__bfloat162float(y[t]) > 0.f ? g[t] : 0.f);
}

// Mean-squared error of the first `nc` of `cpad` predicted channels against
// an FP32 target [p][nc]; grad (BF16, [p][cpad], zero in padded channels)
// = 2 (pred - target) / (P * nc); loss accumulated into *loss.
__global__ void k_mse(const float* __restrict__ pred, const float* __restrict__ target,
                      const float* __restrict__ weight, __nv_bfloat16* __restrict__ grad,
                      float* __restrict__ loss, long long P, int nc, int cpad) {
  __shared__ float red[8];
  float acc = 0.f;
  const float scale = 2.f / (float)(P * nc);
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < P * cpad;
       t += (long long)gridDim.x * blockDim.x) {
    const long long p = t / cpad;
    const int c = (int)(t - p * cpad);
    float gv = 0.f;
    if (c < nc) {
      const float d = pred[t] - target[p * nc + c];
      const float w = weight ? weight[p] : 1.f;
      acc += w * d * d;
      gv = scale * w * d;
    }
    grad[t] = __float2bfloat16(gv);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float s = 0.f;
    for (int k = 0; k < (int)(blockDim.x >> 5); k++) s += red[k];
    atomicAdd(loss, s / (float)(P * nc));
  }
}

// Adam on FP32 master weights; also writes the BF16 copy the convolution
// reads (bias: w16 == nullptr).
__global__ void k_adam(float* __restrict__ w, float* __restrict__ m, float* __restrict__ v,
                       const float* __restrict__ g, __nv_bfloat16* __restrict__ w16, int n,
                       float lr, float b1, float b2, float eps, float c1, float c2) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    const float gt = g[t];
    const float mt = b1 * m[t] + (1.f - b1) * gt;
    const float vt = b2 * v[t] + (1.f - b2) * gt * gt;
    m[t] = mt;
    v[t] = vt;
    const float wt = w[t] - lr * (mt / c1) / (sqrtf(vt / c2) + eps);
    w[t] = wt;
    if (w16) w16[t] = __float2bfloat16(wt);
  }
}

// Zero-mean, unit-variance noise that depends only on (seed, key): the sum
// of four uniforms from a 64-bit mix (splitmix64 finaliser), rescaled.
__device__ __forceinline__ float hash_noise(unsigned long long seed, unsigned long long key) {
  unsigned long long z = seed ^ (key * 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  float sum = 0.f;
#pragma unroll
  for (int q = 0; q < 4; q++) sum += (float)((z >> (16 * q)) & 0xFFFF) * (1.f / 65536.f);
  return (sum - 2.f) * 1.7320508f;  // variance of the sum is 4/12
}

// Per-pixel statics of a domain: depth (ht / 500 m), open-boundary
// indicator (1 on wet cells next to the open side), and 1 where the pixel's
// east (u) or north (v) face is a wall.
constexpr int kStatics = 4;

// Network inputs of `batch` domain states (each an H x W image of
// (ssh, u, v), u / v on the east / north face of the pixel's cell):
//   0-2  ssh - tidal ssh at the target time, u, v / state scales (ssh as a
//        departure from the tide keeps BF16's resolution where the level
//        follows the tide, next to the open side)
//   3    depth (ht / 500 m)
//   4    tidal ssh at the target time on cells next to the open side
//   5    ssh(i+1, j) - ssh(i, j)      (east-face pressure gradient)
//   6    ssh(i, j+1) - ssh(i, j)      (north-face pressure gradient)
//   7    sum of face depth x velocity out of the cell (flux divergence)
//   8    open-boundary indicator
//   9    ssh - tidal ssh on cells next to the open side (what the Flather
//        condition radiates out)
//   10, 11  east / north face is a wall
//   12-14   low BF16 parts of channels 0-2 (value - BF16(value)): next to
//        the open side the state is 20-50x its k-step change, so one BF16
//        (8-bit mantissa) would leave a few per cent of noise in what the
//        network predicts; high + low carry 16 bits
// Channels 5-7 and 9 are differences of nearly equal numbers, so they are
// formed in FP32 before the BF16 rounding; the scales of 5-7 come from the
// data.  A face outside the image (the closed or open boundary) contributes
// zero.
// With noise (training only) the input state is the snapshot plus white
// noise of the given standard deviations, the same value wherever a cell is
// read, and the target is the increment from that perturbed state.
struct Noisy {
  const float* img;
  float3 sd;
  unsigned long long seed, base;
  __device__ float get(int q, int ch) const {
    float v = img[(size_t)q * 3 + ch];
    const float s = ch == 0 ? sd.x : (ch == 1 ? sd.y : sd.z);
    if (s != 0.f) v += s * hash_noise(seed, (base + (unsigned long long)q) * 3ull + ch);
    return v;
  }
};

__global__ void k_assemble(const float* __restrict__ snaps, const float* __restrict__ statics,
                           const int* __restrict__ src, const int* __restrict__ dom,
                           const float* __restrict__ forcing, float3 scale, float3 inc_scale,
                           float3 dscale, float3 noise, unsigned long long seed,
                           __nv_bfloat16* __restrict__ x, float* __restrict__ target, int H,
                           int W, int cpad, int batch) {
  const long long HW = (long long)H * W;
  const long long n = (long long)batch * HW;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    const int b = (int)(t / HW), p = (int)(t - (long long)b * HW);
    const int r = p / W, c = p - r * W;
    const Noisy img{snaps + (size_t)src[b] * HW * 3, noise, seed,
                    (unsigned long long)b * (unsigned long long)HW};
    const float* sti = statics + (size_t)dom[b] * HW * kStatics;
    const float* st = sti + (size_t)p * kStatics;
    const int pe = c + 1 < W ? p + 1 : p, pw = c > 0 ? p - 1 : -1;
    const int pn = r + 1 < H ? p + W : p, ps = r > 0 ? p - W : -1;
    const float d = st[0];
    const float e0 = img.get(p, 0), u0 = img.get(p, 1), v0 = img.get(p, 2);
    const float gx = (pe != p ? img.get(pe, 0) : e0) - e0;
    const float gy = (pn != p ? img.get(pn, 0) : e0) - e0;
    float div = 0.5f * (d + sti[(size_t)pe * kStatics]) * u0 +
                0.5f * (d + sti[(size_t)pn * kStatics]) * v0;
    if (pw >= 0) div -= 0.5f * (d + sti[(size_t)pw * kStatics]) * img.get(pw, 1);
    if (ps >= 0) div -= 0.5f * (d + sti[(size_t)ps * kStatics]) * img.get(ps, 2);
    __nv_bfloat16* xo = x + (size_t)t * cpad;
    const float st0[3] = {(e0 - forcing[b]) / scale.x, u0 / scale.y, v0 / scale.z};
#pragma unroll
    for (int ch = 0; ch < 3; ch++) {  // high and low BF16 parts
      const __nv_bfloat16 hi = __float2bfloat16(st0[ch]);
      xo[ch] = hi;
      xo[12 + ch] = __float2bfloat16(st0[ch] - __bfloat162float(hi));
    }
    xo[3] = __float2bfloat16(d);
    xo[4] = __float2bfloat16(forcing[b] * st[1] / scale.x);
    xo[5] = __float2bfloat16(gx / dscale.x);
    xo[6] = __float2bfloat16(gy / dscale.y);
    xo[7] = __float2bfloat16(div / dscale.z);
    xo[8] = __float2bfloat16(st[1]);
    xo[9] = __float2bfloat16((e0 - forcing[b]) * st[1] / scale.x);
    xo[10] = __float2bfloat16(st[2]);
    xo[11] = __float2bfloat16(st[3]);
    for (int ch = 15; ch < cpad; ch++) xo[ch] = __float2bfloat16(0.f);
    if (target) {
      // the next snapshot of the same domain
      const float* s1 = img.img + ((size_t)HW + p) * 3;
      float* to = target + (size_t)t * 3;
      to[0] = (s1[0] - e0) / inc_scale.x;
      to[1] = (s1[1] - u0) / inc_scale.y;
      to[2] = (s1[2] - v0) / inc_scale.z;
    }
  }
}

// state += increment (first 3 of cpad FP32 output channels) * inc_scale.
// With statics, the solver's boundary conditions are applied as the solver
// applies them: velocities on wall faces are held at zero, and the ssh of
// wet cells next to the open side is the tide at the target time.
__global__ void k_advance(float* __restrict__ state, const float* __restrict__ inc,
                          float3 inc_scale, const float* __restrict__ statics,
                          const int* __restrict__ dom, const float* __restrict__ forcing,
                          long long HW, long long P, int cpad) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < P;
       t += (long long)gridDim.x * blockDim.x) {
    float e = state[t * 3 + 0] + inc[t * cpad + 0] * inc_scale.x;
    float u = state[t * 3 + 1] + inc[t * cpad + 1] * inc_scale.y;
    float v = state[t * 3 + 2] + inc[t * cpad + 2] * inc_scale.z;
    if (statics) {
      const long long b = t / HW;
      const float* st = statics + ((size_t)dom[b] * HW + (t - b * HW)) * kStatics;
      if (st[1] > 0.f) e = forcing[b];
      if (st[2] > 0.f) u = 0.f;
      if (st[3] > 0.f) v = 0.f;
    }
    state[t * 3 + 0] = e;
    state[t * 3 + 1] = u;
    state[t * 3 + 2] = v;
  }
}

// The launches of the two kernels (POLL with its limit: the test hook's form).
template <bool POLL>
int conv3x3(const void* x, const void* w, const float* bias, void* y, float* y32, int batch, int H,
            int W, int cin, int cout, int relu, long long max_cycles, int* err, void* stream) {
  if (cin % 16 || cout % 16 || cout > 64 || cin < 16 || cin > 64 || W % kTileM || H < 1 ||
      batch < 1 || !x || !w || !err || (!y && !y32))
    return NL2D_ERR_ARGS;
  const size_t wbytes = ((9 * (size_t)cout * cin * 2) + 1023) & ~(size_t)1023;
  const size_t smem = wbytes + kConvSlots * (size_t)(cin / 8) * kLboX;
  constexpr int kMaxSmem = 200 * 1024;
  static bool attr = false;
  if (!attr) {
    if (cudaFuncSetAttribute(k_conv3x3_pipe<POLL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kMaxSmem) != cudaSuccess)
      return NL2D_ERR_CUDA;
    attr = true;
  }
  if (smem > kMaxSmem) return NL2D_ERR_ARGS;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const long long rows = (long long)batch * H * (W / kTileM);
  // Persistent CTAs: as many as are resident at once, with two rows or more
  // each.  Counted from the kernel's registers (allocated per warp in units of
  // 256) and shared memory (dynamic + static + the driver's reserve per
  // block), as the hardware limits them; each CTA also holds conv_tmem() of
  // the SM's 512 TMEM columns.  (cudaOccupancyMaxActiveBlocksPerMultiprocessor
  // answered 1 where 2 are resident.)
  static cudaFuncAttributes fa;
  static bool fa_ok = false;
  if (!fa_ok) {
    if (cudaFuncGetAttributes(&fa, k_conv3x3_pipe<POLL>) != cudaSuccess) return NL2D_ERR_CUDA;
    fa_ok = true;
  }
  int regs_sm = 0, smem_sm = 0, smem_rsv = 0;
  cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, dev);
  cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
  cudaDeviceGetAttribute(&smem_rsv, cudaDevAttrReservedSharedMemoryPerBlock, dev);
  const int warp_regs = (fa.numRegs * 32 + 255) / 256 * 256;
  const int by_regs = regs_sm / (warp_regs * (kPipeThreads / 32));
  const int by_smem = smem_sm / (int)(smem + fa.sharedSizeBytes + smem_rsv);
  int per_sm = by_regs < by_smem ? by_regs : by_smem;
  per_sm = per_sm < 512 / conv_tmem(cout) ? per_sm : 512 / conv_tmem(cout);
  per_sm = per_sm < 1 ? 1 : per_sm;
  const int grid =
      (int)std::max<long long>(1, std::min<long long>(rows / 2, (long long)per_sm * sms));
  // 32-byte stores where an output starts on a 32-byte boundary (every pixel
  // then does: cout is a multiple of 16)
  const int wide = ((uintptr_t)y % 32 == 0 ? 1 : 0) | ((uintptr_t)y32 % 32 == 0 ? 2 : 0);
  k_conv3x3_pipe<POLL><<<grid, kPipeThreads, smem, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)x, (const __nv_bfloat16*)w, bias, (__nv_bfloat16*)y, y32, batch, H,
      W, cin, cout, relu, wide, max_cycles, err);
  return cudaGetLastError() == cudaSuccess ? NL2D_OK : NL2D_ERR_CUDA;
}

template <bool POLL>
int conv_wgrad(const void* x, const void* dy, float* dw, float* db, int batch, int H, int W,
               int cin, int cout, long long max_cycles, int* err, void* stream) {
  if (!x || !dy || !dw || !db || !err || cin % 16 || cin < 16 || 9 * cin > kWgTmemCols ||
      cout % 8 || cout < 8 || cout > 128 || W % kTileM || H < 1 || batch < 1)
    return NL2D_ERR_ARGS;
  // As many ring slots as fit (at least one row in flight: wg_depth).
  // The kernel holds all 512 TMEM columns, so it must be alone on its SM:
  // asking for more than half an SM's shared memory guarantees that.
  int slots = kWgMaxSlots;
  while (slots > 3 && wg_smem(cin, cout, slots) > kWgMaxSmem) slots--;
  const size_t need = wg_smem(cin, cout, slots);
  const size_t smem = need > 120 * 1024 ? need : 120 * 1024;
  static bool attr = false;
  if (!attr) {
    if (cudaFuncSetAttribute(k_conv_wgrad_pipe<POLL>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kWgMaxSmem) != cudaSuccess)
      return NL2D_ERR_CUDA;
    attr = true;
  }
  if (smem > kWgMaxSmem) return NL2D_ERR_ARGS;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // one CTA per SM (512 TMEM columns), with four rows or more each
  const long long rows = (long long)batch * H * (W / kTileM);
  const int grid = (int)std::max<long long>(1, std::min<long long>(rows / 4, sms));
  const long long nel = 9LL * cout * cin;
  const cudaStream_t st = (cudaStream_t)stream;
  Parts parts(dev, (size_t)(grid * (nel + cout)), st);
  if (!parts.p) return NL2D_ERR_CUDA;
  k_conv_wgrad_pipe<POLL><<<grid, kWgThreads, smem, st>>>(
      (const __nv_bfloat16*)x, (const __nv_bfloat16*)dy, parts.p, batch, H, W, cin, cout, slots,
      max_cycles, err);
  k_sum_parts<<<(int)((nel + cout + kSumElems - 1) / kSumElems), kSumWays * kSumElems, 0, st>>>(
      parts.p, grid, nel, cout, dw, db,
      WgradInputs{(const __nv_bfloat16*)x, (const __nv_bfloat16*)dy, batch, H, W, cin, cout},
      cout <= 64);
  const cudaError_t launched = cudaGetLastError();
  return parts.done() && launched == cudaSuccess ? NL2D_OK : NL2D_ERR_CUDA;
}

}  // namespace
}  // namespace emu

void emu_release() {
  for (emu::PartsKept& d : emu::g_parts) {
    std::lock_guard<std::mutex> hold(d.lock);
    for (auto& e : d.of) {
      cudaFree(e.p);  // (waits for the calls in flight)
      e = {};
    }
    if (d.pool) cudaMemPoolDestroy(d.pool);
    d.pool = nullptr;
  }
}
}  // namespace nl2d

using namespace nl2d::emu;

extern "C" {

// Test hook (no reference counterpart): runs k_selftest_wait and returns
// its status in *status: 1 when the wait ran out and reported it, as the
// convolution kernels' waits do.
int nl2d_selftest_wait(long long max_cycles, int* status) {
  if (!status || max_cycles < 1 || max_cycles > (1LL << 32)) return NL2D_ERR_ARGS;
  int* d = nullptr;
  if (cudaMalloc(&d, sizeof(int)) != cudaSuccess) return NL2D_ERR_CUDA;
  cudaMemset(d, 0, sizeof(int));
  k_selftest_wait<<<1, 32>>>(max_cycles, d);
  const cudaError_t e = cudaMemcpy(status, d, sizeof(int), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e == cudaSuccess ? NL2D_OK : NL2D_ERR_CUDA;
}

// 3x3 convolution (stride 1, zero padding 1) of a batch of NHWC BF16
// images on the tensor cores.  cin, cout: multiples of 16, cout <= 64;
// W a multiple of 128.  y (BF16) and/or y32 (FP32) receive bias + conv,
// ReLU'd if relu.  err: device int set to 1 if a wait timed out.
int nl2d_emu_conv3x3(const void* x, const void* w, const float* bias, void* y, float* y32,
                     int batch, int H, int W, int cin, int cout, int relu, int* err,
                     void* stream) {
  return conv3x3<false>(x, w, bias, y, y32, batch, H, W, cin, cout, relu, 0, err, stream);
}

int nl2d_emu_flip_transpose(const void* w, void* wt, int cout, int cin, void* stream) {
  if (!w || !wt || cout < 1 || cin < 1) return NL2D_ERR_ARGS;
  k_flip_transpose<<<64, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)w,
                                                          (__nv_bfloat16*)wt, cout, cin);
  return cudaGetLastError() == cudaSuccess ? NL2D_OK : NL2D_ERR_CUDA;
}

int nl2d_emu_conv_wgrad(const void* x, const void* dy, float* dw, float* db, int batch, int H,
                        int W, int cin, int cout, int* err, void* stream) {
  return conv_wgrad<false>(x, dy, dw, db, batch, H, W, cin, cout, 0, err, stream);
}

// Test hook (no reference counterpart): the convolution (wgrad = 0; b the
// weights, out FP32 values, db unused) or the weight gradient (b the output's
// gradient, out dw) with another limit on the roles' waits for each other.
int nl2d_selftest_emu_wait(int wgrad, const void* x, const void* b, float* out, float* db,
                           int batch, int H, int W, int cin, int cout, long long max_cycles,
                           int* err) {
  if (max_cycles < 0 || max_cycles > kMaxWaitCycles) return NL2D_ERR_ARGS;
  return wgrad ? conv_wgrad<true>(x, b, out, db, batch, H, W, cin, cout, max_cycles, err, nullptr)
               : conv3x3<true>(x, b, nullptr, nullptr, out, batch, H, W, cin, cout, 0, max_cycles,
                               err, nullptr);
}

int nl2d_emu_relu_bwd(const float* g, const void* y, void* out, long long n, void* stream) {
  k_relu_bwd<<<152 * 8, 256, 0, (cudaStream_t)stream>>>(g, (const __nv_bfloat16*)y,
                                                         (__nv_bfloat16*)out, n);
  return cudaGetLastError() == cudaSuccess ? NL2D_OK : NL2D_ERR_CUDA;
}

int nl2d_emu_mse(const float* pred, const float* target, const float* weight, void* grad,
                 float* loss, long long P, int nc, int cpad, void* stream) {
  if (!pred || !target || !grad || !loss || P < 1 || nc < 1 || cpad < nc) return NL2D_ERR_ARGS;
  k_mse<<<152 * 4, 256, 0, (cudaStream_t)stream>>>(pred, target, weight, (__nv_bfloat16*)grad,
                                                    loss, P, nc, cpad);
  return cudaGetLastError() == cudaSuccess ? NL2D_OK : NL2D_ERR_CUDA;
}

int nl2d_emu_adam(float* w, float* m, float* v, const float* g, void* w16, int n, float lr,
                  float b1, float b2, float eps, int step, void* stream) {
  const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
  k_adam<<<64, 256, 0, (cudaStream_t)stream>>>(w, m, v, g, (__nv_bfloat16*)w16, n, lr, b1, b2,
                                                eps, c1, c2);
  return cudaGetLastError() == cudaSuccess ? NL2D_OK : NL2D_ERR_CUDA;
}

int nl2d_emu_assemble(const float* snaps, const float* statics, const int* src,
                      const int* dom, const float* forcing, const float* scale12,
                      unsigned long long seed, void* x, float* target, int H, int W, int cpad,
                      int batch, void* stream) {
  if (!snaps || !statics || !src || !dom || !forcing || !scale12 || !x || cpad < 15 || H < 1 ||
      W < 1 || batch < 1)
    return NL2D_ERR_ARGS;
  k_assemble<<<152 * 8, 256, 0, (cudaStream_t)stream>>>(
      snaps, statics, src, dom, forcing, make_float3(scale12[0], scale12[1], scale12[2]),
      make_float3(scale12[3], scale12[4], scale12[5]),
      make_float3(scale12[6], scale12[7], scale12[8]),
      make_float3(scale12[9], scale12[10], scale12[11]), seed, (__nv_bfloat16*)x, target, H, W,
      cpad, batch);
  return cudaGetLastError() == cudaSuccess ? NL2D_OK : NL2D_ERR_CUDA;
}

int nl2d_emu_advance(float* state, const float* inc, const float* inc_scale3,
                     const float* statics, const int* dom, const float* forcing, long long HW,
                     long long P, int cpad, void* stream) {
  if (!state || !inc || !inc_scale3 || (statics && (!dom || !forcing || HW < 1)) || P < 0 ||
      cpad < 3)
    return NL2D_ERR_ARGS;
  k_advance<<<152 * 8, 256, 0, (cudaStream_t)stream>>>(
      state, inc, make_float3(inc_scale3[0], inc_scale3[1], inc_scale3[2]), statics, dom,
      forcing, HW, P, cpad);
  return cudaGetLastError() == cudaSuccess ? NL2D_OK : NL2D_ERR_CUDA;
}

}  // extern "C"
