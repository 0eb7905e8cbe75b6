// Surrogate convolutions on the 5th-generation tensor cores (tcgen05, sm_103a) for 128^3 boxes.
//
// The 3x3x3 circular convolution of a channels-last BF16 box [z][y][x][CIN] with weights
// [27][COUT][CIN] (tap (dz + 1) * 9 + (dy + 1) * 3 + (dx + 1)) is computed input-stationary.  One
// CTA per SM walks a contiguous range of output rows (z, y) of one z-plane at a time.  For each
// input row Y of the plane's three neighbours (z + dz) and each shift dx, one
// `tcgen05.mma.kind::f16` (BF16 x BF16 -> FP32, M = 128 voxels, K = 16 channels) multiplies the
// shifted row by the weights of the three taps (dz, dy = -1, 0, +1, dx) side by side in N:
// N = 3 * COUT columns land in the tensor-memory accumulators of output rows Y + 1, Y and Y - 1.
// Sharing the A operand (the shifted input row) between three output rows cuts the MMAs per output
// row from 27 * CIN / 16 with N = COUT to 9 * CIN / 16 with N = 3 * COUT; an N = COUT MMA pays
// for the whole 128 x 16 A tile from shared memory.
//
// Tensor memory holds S = 512 / COUT accumulators of COUT columns; output row o (the CTA's o-th)
// owns slot S - 1 - (o mod S), so rows Y + 1, Y, Y - 1 sit in ascending columns and one MMA covers
// them (two where the slot ring wraps).  Every MMA accumulates: the epilogue zeroes a slot after
// reading it, and all slots start zeroed.
//
// Shared memory holds every weight, per (dz, dx) as [ci / 8][dy, co][ci % 8] (K-major, no swizzle),
// and a ring of YS input-row groups; a group is the three rows (z - 1, z, z + 1) at one y.  A row lies as
// in memory, one voxel's channels (64 or 32 bytes) after another, swizzled over that span (K-major
// operand), with the circular neighbours of its ends before and behind it, so that shift dx starts the
// operand one voxel earlier or later.  A row comes by three TMA copies: its 128 voxels, and the 128 bytes
// that end (begin) the row once more in front of (behind) it.  A group is used by exactly one round of MMAs
// and released right after it.
//
// What bounds it: the operands' way out of shared memory, 7168 bytes per MMA of N = 96 at 128 bytes a
// cycle: 56 cycles, 1008 a row, 53 us a launch.  Copied by 16-byte cp.async into a layout of 8-channel
// chunks, as before, a group took its producers ~2000 cycles (the pieces land one by one, and each group needed
// a proxy fence): a 32 -> 32 layer 142 us, now 106.  The rest is the MMA
// warp's own work between rows (waits, commits, descriptors: ~700 cycles of dependent instructions).
//
// Roles: warp 0 issues the copies (one lane); warp 1 issues the MMAs (one elected lane) and commits
// completion to mbarriers; warps 2..9, two groups that take output rows in turn, read finished
// accumulators (tcgen05.ld, one TMEM lane = one voxel per thread), zero them, add the bias and apply
// ReLU / sigmoid / the input-gradient mask (read ahead of the accumulator), and store BF16 (or FP32)
// rows.  Every wait is bounded; on a timeout the CTA records the error, drains its copies and MMAs, frees
// its TMEM and leaves.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdio>
#include <mutex>
#include <string>
#include <type_traits>

#include "es_engine.h"

namespace sgtc {

constexpr int N = 128;                 // box side: one x-row is one M = 128 tile
constexpr int YS = 6;                  // input-row groups in the ring
constexpr int CONV_MMA_WARP = 1;
constexpr int EPI_GROUPS = 2;          // epilogue warpgroups of the convolutions, taking output rows in turn
constexpr int CONV_THREADS = 32 * (2 + 4 * EPI_GROUPS);
constexpr uint32_t TMEM_COLS = 512;
constexpr long kSpin = 1L << 24;       // mbarrier polls before a wait is declared hung
constexpr unsigned ERR_TIMEOUT = 1u;

enum Mode { FWD_RELU = 0, FWD_SIGMOID = 1, DGRAD_MASK = 2 };

__device__ unsigned g_err;

template <int CIN, int COUT> struct Layout {
  static constexpr int KC = CIN / 8;                  // 8-channel chunks
  static constexpr int S = TMEM_COLS / COUT;          // accumulator slots
  static constexpr int LBO_B = 3 * COUT * 16;         // B: K core matrices 3 * COUT rows apart
  static constexpr int PAIR_B = KC * LBO_B;           // B of one (dz, dx): 3 taps
  static constexpr int W_BYTES = 9 * PAIR_B;
  static constexpr int VOX = CIN * 2;                  // bytes of a voxel: the swizzle span
  static constexpr int PAD = 512;                      // before and between rows: 128 bytes of either neighbour's ends
  static constexpr int ROW = N * VOX + PAD;            // from row to row
  static constexpr int GROUP = 3 * ROW;
  static constexpr int HALO = 128 / VOX;               // voxels of an end copy (128 bytes)
  static constexpr uint32_t GROUP_TX = 3 * (N * VOX + 2 * 128);
  static constexpr int RING_BYTES = PAD + YS * GROUP;
  static constexpr int W_OFF = (RING_BYTES + 127) / 128 * 128;
  static constexpr int BAR_OFF = W_OFF + W_BYTES;
  static constexpr int NBARS = 2 * YS + 2 * S + 1;    // full[YS], sfree[YS], done[S], tfree[S], drain
  static constexpr int BYTES = BAR_OFF + NBARS * 8 + 16 + 1024;   // + tmem slot, abort, groups issued, alignment
  static_assert(VOX == 64 || VOX == 32, "a voxel is one swizzle span");
  static_assert(W_BYTES % 16 == 0, "16-byte aligned regions");
  static_assert(3 * COUT <= 256 && COUT % 16 == 0, "N = 3 COUT must be a valid M = 128 MMA width");
  static_assert(BYTES <= 232448, "shared memory per CTA");
};

// ------------------------------------------------------------------ PTX wrappers
__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void bar_init(uint64_t* b, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(saddr(b)) : "memory");
}
__device__ __forceinline__ bool bar_try(uint64_t* b, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(saddr(b)), "r"(parity)
      : "memory");
  return ok != 0;
}
// bounded wait; gives up (and raises the CTA's abort flag) after kSpin polls or once another role
// has aborted
__device__ __forceinline__ bool bar_wait(uint64_t* b, uint32_t parity, volatile int* abort) {
  for (long i = 0; i < kSpin; ++i) {
    if (bar_try(b, parity)) return true;
    if ((i & 255) == 255 && *abort) return false;
  }
  *abort = 1;
  atomicOr(&g_err, ERR_TIMEOUT);
  return false;
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void fence_bar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void bar_expect_tx(uint64_t* b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(saddr(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tma_load3(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(saddr(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(saddr(bar))
      : "memory");
}
__device__ __forceinline__ void tc_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(slot)), "r"(cols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}

// Shared-memory matrix descriptor, K-major without swizzle: core matrices of 8 rows x 16 bytes,
// `lbo` between core matrices along K, `sbo` between 8-row groups along M / N.
__device__ __forceinline__ uint64_t mdesc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
// The same, K-major with rows of VOX = 64 or 32 bytes swizzled over that span: 8-row groups one after
// another; the pattern goes by the address, so a start inside a group needs no more.
template <int VOX> __device__ __forceinline__ uint64_t mdesc_rows(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | (1ull << 16) | ((uint64_t)((8 * VOX) >> 4) << 32) | (1ull << 46) |
         ((VOX == 64 ? 4ull : 6ull) << 61);
}
// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both K-major, M x N.
__host__ __device__ constexpr uint32_t idesc_bf16(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
// D += A B; every MMA of this kernel accumulates into a zeroed or partly summed slot.  The whole
// warp runs the issue loop (its operands stay warp-uniform) and one elected lane issues.
__device__ __forceinline__ void mma_acc(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc) {
  asm volatile(
      "{\n .reg .pred p, e;\n setp.ne.b32 p, 1, 0;\n elect.sync _|e, 0xffffffff;\n"
      " @e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
      ::"r"(d), "l"(a), "l"(b), "r"(idesc)
      : "memory");
}
// completion of every MMA issued so far arrives once on `b` (one elected lane of a converged warp)
__device__ __forceinline__ void mma_commit(uint64_t* b) {
  asm volatile(
      "{\n .reg .pred e;\n elect.sync _|e, 0xffffffff;\n"
      " @e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(saddr(b))
      : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
// zero 16 columns of this warp's 32 lanes
__device__ __forceinline__ void tmem_zero16(uint32_t taddr) {
  const uint32_t z = 0;
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, "
      "%1};" ::"r"(taddr), "r"(z)
      : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Output rows [r0, r1) of this CTA, walked in segments of one z-plane each.
struct Range {
  int r0, r1;
};
__device__ __forceinline__ Range my_rows() {
  const int rows = N * N;
  return {(int)((long)rows * blockIdx.x / gridDim.x), (int)((long)rows * (blockIdx.x + 1) / gridDim.x)};
}

// The input-row groups of a CTA in order: per z-plane segment [yb, ye) of its output rows, y = yb - 1 .. ye.
struct GroupWalk {
  int r, r1, z, ye, yy;
  __device__ __forceinline__ GroupWalk(Range rg) : r(rg.r0), r1(rg.r1) { segment(); }
  __device__ __forceinline__ void segment() {
    z = r / N;
    ye = (z + 1) * N < r1 ? N : r1 - z * N;
    yy = r % N - 1;
  }
  __device__ __forceinline__ bool done() const { return r >= r1; }
  __device__ __forceinline__ void next() {
    if (++yy > ye) {
      r = z * N + ye;
      segment();
    }
  }
};

template <int CIN, int COUT, int MODE>
__global__ void __launch_bounds__(CONV_THREADS, 1) conv_tc_kernel(const __grid_constant__ CUtensorMap tm_row,
                                                                  const __grid_constant__ CUtensorMap tm_end,
                                                                  const __nv_bfloat16* __restrict__ w,
                                                                  const float* __restrict__ bias, void* out,
                                                                  const __nv_bfloat16* __restrict__ mask) {
  using L = Layout<CIN, COUT>;
  constexpr int KC = L::KC, S = L::S;
  constexpr int KSTEPS = CIN / 16;                    // MMA K steps per (dz, dx)
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char* sm = smem_raw + ((0u - saddr(smem_raw)) & 1023u);
  unsigned char* ring = sm + L::PAD;                  // first voxel of the first row
  unsigned char* sw = sm + L::W_OFF;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + L::BAR_OFF);
  uint64_t* full = bars;
  uint64_t* sfree = bars + YS;
  uint64_t* done = bars + 2 * YS;
  uint64_t* tfree = bars + 2 * YS + S;
  uint64_t* drain = bars + 2 * YS + 2 * S;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + L::NBARS);
  volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < YS; ++i) {
      bar_init(&full[i], 1);
      bar_init(&sfree[i], 1);
    }
    for (int i = 0; i < S; ++i) {
      bar_init(&done[i], 1);
      bar_init(&tfree[i], 128);
    }
    bar_init(drain, 1);
    *abort = 0;
    fence_bar_init();
  }
  if (warp == 0) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  __syncthreads();
  const Range rg = my_rows();
  GroupWalk walk(rg);
  int issued = 0;                                     // groups whose copies are under way
  auto issue_group = [&]() {
    const int slot = issued % YS;
    bar_expect_tx(&full[slot], L::GROUP_TX);
    unsigned char* gb = ring + slot * L::GROUP;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const int row = ((walk.z + d + N - 1) % N) * N + (walk.yy + N) % N;
      unsigned char* dst = gb + d * L::ROW;
      tma_load3(dst, &tm_row, &full[slot], 0, 0, row);
      tma_load3(dst - 128, &tm_end, &full[slot], 0, N - L::HALO, row);
      tma_load3(dst + N * L::VOX, &tm_end, &full[slot], 0, 0, row);
    }
    ++issued;
    walk.next();
  };
  // the first groups are on their way while the weights are staged
  if (threadIdx.x == 0)
    while (issued < YS && !walk.done()) issue_group();
  // weights -> per (dz, dx): [ci / 8][dy, co][ci % 8], 16-byte chunks; all loads of a thread in flight at once
  {
    constexpr int WCH = 27 * COUT * KC, Q = (WCH + CONV_THREADS - 1) / CONV_THREADS;
    uint4 v[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int c = threadIdx.x + q * CONV_THREADS;
      if (c < WCH) v[q] = __ldg(reinterpret_cast<const uint4*>(w) + c);   // [t][co][kc] is w's own order
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int c = threadIdx.x + q * CONV_THREADS;
      if (c < WCH) {
        const int kc = c % KC, co = (c / KC) % COUT, t = c / (KC * COUT);
        const int dz = t / 9, dy = (t / 3) % 3, dx = t % 3;
        *reinterpret_cast<uint4*>(sw + (dz * 3 + dx) * L::PAIR_B + kc * L::LBO_B + (dy * COUT + co) * 16) = v[q];
      }
    }
  }
  fence_proxy_async();                                // generic writes -> tensor-core reads
  tc_before();
  __syncthreads();
  tc_after();
  const uint32_t tmem = *tmem_slot;
  if (warp > CONV_MMA_WARP && warp <= CONV_MMA_WARP + 4) {
    // every accumulator slot starts at zero
    const uint32_t lanes = (uint32_t)(32 * (warp & 3)) << 16;
    for (int c = 0; c < (int)TMEM_COLS; c += 16) tmem_zero16(tmem + lanes + (uint32_t)c);
    tmem_wait_st();
  }
  tc_before();
  __syncthreads();
  tc_after();

  if (warp == 0) {
    // ------------------------------------------------------------------ copies
    if (lane == 0) {
      for (; !walk.done(); issue_group())
        if (issued >= YS && !bar_wait(&sfree[issued % YS], (uint32_t)((issued / YS - 1) & 1), abort)) break;
      abort[1] = issued;
    }
  } else if (warp == CONV_MMA_WARP) {
    {
      // ---------------------------------------------------------------- MMA issue
      // Descriptors are a base descriptor plus (byte offset >> 4) in the 14-bit address field.
      const uint64_t a_base = mdesc_rows<L::VOX>(saddr(ring));
      const uint64_t b_base = mdesc(saddr(sw), L::LBO_B, 128);
      int g = 0, o0 = 0;
      for (int r = rg.r0; r < rg.r1 && !__any_sync(0xFFFFFFFFu, *abort);) {
        const int z = r / N, yb = r % N;
        const int ye = (z + 1) * N < rg.r1 ? N : rg.r1 - z * N;
        // Input row Y's group has landed and output row Y + 1's slot is free.  Freed slots are looked for
        // eight rows at a time (a wait costs ~200 cycles even when there is nothing to wait for): the
        // epilogue groups take rows in order, so the last row of either group among the eight speaks for all.
        auto ready = [&](int Y, int gg) {
          bool k = bar_wait(&full[gg % YS], (uint32_t)((gg / YS) & 1), abort);
          const int o = o0 + Y + 1 - yb;
          if (Y + 1 < ye && o >= S && o % 8 == 0) {
#pragma unroll
            for (int e = 0; e < EPI_GROUPS; ++e) {
              const int q = o + 7 - e;
              k = k && bar_wait(&tfree[(S - 1) - q % S], (uint32_t)((q / S - 1) & 1), abort);
            }
          }
          return (bool)__all_sync(0xFFFFFFFFu, k);
        };
        bool ok = ready(yb - 1, g);
        for (int Y = yb - 1; Y <= ye && ok; ++Y, ++g) {
          // output rows this input row feeds: y in [ylo, yhi], tap dy = Y - y
          const int ylo = Y - 1 > yb ? Y - 1 : yb, yhi = Y + 1 < ye - 1 ? Y + 1 : ye - 1;
          const int ohi = o0 + (yhi - yb);
          tc_after();
          const int nrows = yhi - ylo + 1;
          const int s0 = (S - 1) - ohi % S;            // slot of row yhi; rows below follow upward
          const int n1 = nrows < S - s0 ? nrows : S - s0, n2 = nrows - n1;
          const uint32_t id1 = idesc_bf16(128, n1 * COUT), id2 = idesc_bf16(128, (n2 > 0 ? n2 : 1) * COUT);
          const uint32_t d1 = tmem + (uint32_t)(s0 * COUT);
          const uint64_t a_g = a_base + (uint64_t)((g % YS) * (L::GROUP / 16));
          const uint64_t b_blk = b_base + (uint64_t)((Y - yhi + 1) * COUT);   // first dy block, 16-byte units
// One straight run of MMAs per case: a test between the MMAs (whether the slot ring wraps)
          // would put a branch around every elected issue and slow the issue to ~90 cycles per MMA;
          // without it the issue keeps pace with the tensor pipe (~56 cycles at N = 96).
          auto issue = [&](auto two, auto from, auto to) {
            constexpr bool TWO = decltype(two)::value;
#pragma unroll
            for (int dz = decltype(from)::value; dz < decltype(to)::value; ++dz) {
#pragma unroll
              for (int dx = 0; dx < 3; ++dx) {
                const uint64_t ad = a_g + (uint64_t)(int64_t)((dz * L::ROW + (dx - 1) * L::VOX) / 16);
                const uint64_t bd = b_blk + (uint64_t)((dz * 3 + dx) * L::PAIR_B / 16);
#pragma unroll
                for (int k = 0; k < KSTEPS; ++k) {
                  const uint64_t ak = ad + (uint64_t)(2 * k);      // 16 channels: 32 bytes along the voxel
                  const uint64_t bk = bd + (uint64_t)(2 * k * L::LBO_B / 16);
                  mma_acc(d1, ak, bk, id1);
                  if (TWO) mma_acc(tmem, ak, bk + (uint64_t)(n1 * COUT), id2);
                }
              }
            }
          };
          // The waits for the next row stand between the second and the third dz: the MMAs queued so far run
          // meanwhile (waits between rows left the tensor pipe idle ~400 cycles a row)
          typedef std::integral_constant<int, 0> I0;
          typedef std::integral_constant<int, 2> I2;
          typedef std::integral_constant<int, 3> I3;
          if (n2 > 0) issue(std::true_type{}, I0{}, I2{}); else issue(std::false_type{}, I0{}, I2{});
          const bool next_ok = Y < ye ? ready(Y + 1, g + 1) : true;
          tc_after();
          if (n2 > 0) issue(std::true_type{}, I2{}, I3{}); else issue(std::false_type{}, I2{}, I3{});
          mma_commit(&sfree[g % YS]);                 // this input group is not read again
          if (Y - 1 >= yb && Y - 1 < ye) {
            const int od = o0 + (Y - 1 - yb);          // output row Y - 1 has all 27 taps
            mma_commit(&done[(S - 1) - od % S]);
          }
          ok = next_ok;
        }
        if (!ok) break;
        o0 += ye - yb;
        r = z * N + ye;
      }
      // every MMA this CTA issued has completed before its accumulators are freed
      __syncwarp();
      mma_commit(drain);
      for (long i = 0; i < kSpin && !bar_try(drain, 0); ++i) {
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    const int q = warp & 3;                            // TMEM lanes 32 q .. 32 q + 31
    const int x = 32 * q + lane;
    const uint32_t lanes = (uint32_t)(32 * q) << 16;
    float bv[COUT];
#pragma unroll
    for (int c = 0; c < COUT; ++c) bv[c] = bias ? bias[c] : 0.f;
    const int eg = (warp - CONV_MMA_WARP - 1) / 4;         // this warpgroup takes rows o = eg mod EPI_GROUPS
    for (int o = eg; o < rg.r1 - rg.r0; o += EPI_GROUPS) {
      const int r = rg.r0 + o;
      const int slot = (S - 1) - o % S;
      const size_t vox = (size_t)r * N + x;
      uint4 mrow[COUT / 8];                            // the mask's row, on its way while the MMAs finish
      if (MODE == DGRAD_MASK) {
#pragma unroll
        for (int j = 0; j < COUT / 8; ++j) mrow[j] = __ldg(reinterpret_cast<const uint4*>(mask + vox * COUT) + j);
      }
      const bool ok = bar_wait(&done[slot], (uint32_t)((o / S) & 1), abort);
      if (!__all_sync(0xFFFFFFFFu, ok)) break;        // tcgen05.ld / st need the whole warp
      tc_after();
      float v[COUT];
      const uint32_t ta = tmem + lanes + (uint32_t)(slot * COUT);
      if (COUT == 32) tmem_ld32(ta, v); else tmem_ld16(ta, v);
#pragma unroll
      for (int c = 0; c < COUT; c += 16) tmem_zero16(ta + (uint32_t)c);
      tmem_wait_st();
      tc_before();
      bar_arrive(&tfree[slot]);
      if (MODE == FWD_SIGMOID) {
        reinterpret_cast<float*>(out)[vox] = 1.0f / (1.0f + __expf(-(v[0] + bv[0])));
      } else {
        uint32_t mbits = 0xFFFFFFFFu;
        if (MODE == DGRAD_MASK) {
          mbits = 0;
#pragma unroll
          for (int j = 0; j < COUT / 8; ++j) {
            const uint4 m = mrow[j];
            const uint32_t wds[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
            for (int h = 0; h < 8; ++h) {
              const __nv_bfloat16 e = __ushort_as_bfloat16((unsigned short)(wds[h / 2] >> (16 * (h & 1))));
              if (__bfloat162float(e) > 0.f) mbits |= 1u << (8 * j + h);
            }
          }
        }
        uint4* op = reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(out) + vox * COUT);
#pragma unroll
        for (int j = 0; j < COUT / 8; ++j) {
          uint32_t pk[4];
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            const int c = 8 * j + 2 * h;
            float a0 = v[c] + bv[c], a1 = v[c + 1] + bv[c + 1];
            if (MODE == FWD_RELU) {
              a0 = fmaxf(a0, 0.f);
              a1 = fmaxf(a1, 0.f);
            } else {
              if (!((mbits >> c) & 1u)) a0 = 0.f;
              if (!((mbits >> (c + 1)) & 1u)) a1 = 0.f;
            }
            const __nv_bfloat162 p2 = __floats2bfloat162_rn(a0, a1);
            pk[h] = *reinterpret_cast<const uint32_t*>(&p2);
          }
          op[j] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        }
      }
    }
  }

  tc_before();
  __syncthreads();
  // No copy outlives the CTA: the MMA warp has seen every group land, or a role has aborted, which is known only
  // here (the producer may have left its loop before) and then they land first (bounded).  The number issued comes
  // through shared memory: kept in a register to here it changed the whole kernel's schedule (128^3 forward 953 -> 960 us)
  if (threadIdx.x == 0 && *abort) {
    const int groups = abort[1];
    for (int q = groups > YS ? groups - YS : 0; q < groups; ++q)
      for (long i = 0; i < kSpin && !bar_try(&full[q % YS], (uint32_t)((q / YS) & 1)); ++i) {
      }
  }
  if (warp == 0) {
    __syncwarp();
    tc_after();
    tmem_dealloc(tmem, TMEM_COLS);
  }
}

// ------------------------------------------------------------------ weight gradient
// dW[t][co][ci] = sum_v dZ[v][co] X[v + (dz, dy, dx)][ci] and db[co] = sum_v dZ[v][co] at 128^3.
// With u = v + (0, 0, dx): dW = sum_u dZ[u - dx][co] X[u + (dz, dy, 0)][ci], so for one output row
// (z, y) of dZ and one dy, one MMA per 16 voxels covers every (dz, ci) x (dx, co):
//   A (M = 128, MN-major): the input rows z - 1, z, z + 1 at y + dy, and a constant row of ones, whose
//     products are the bias gradient, CIN channels each (with CIN = 16 the upper half of M reads on into
//     whatever follows and is not used);
//   B (N = 3 COUT, MN-major): the dZ row (z, y) three times over, starting one voxel early, in place and one
//     late (dx = +1, 0, -1): with one voxel as the stride between the three, one copy of the row serves;
//   D: one accumulator per dy (3 COUT columns of tensor memory), summed over all of the CTA's rows.
// Staged rows lie as in memory, swizzled over a voxel's bytes (as in the convolutions), which is the
// MN-major layout of that swizzle: 8 voxels to a group along K, a row (or a voxel) from one span of
// channels to the next along M (N).  TMA brings them; a dZ row has its circular neighbours at either
// end.  Per-CTA partials [3][128][3 COUT] are summed in a fixed order by wgrad_tc_reduce.
// Bound by the operands' way out of shared memory, 1344 cycles a row, 70 us a launch; with 16-byte cp.async
// into 8-channel chunks, dZ three times, a 32 x 32 layer took 292 us (the copies, and a proxy fence each);
// now 112 us.
namespace wg {
constexpr int XS = 5;                      // input-row groups: y - 1, y, y + 1 in use, two landing
constexpr int DSL = 4;                     // dZ row slots
constexpr int PAD = 512;                   // before and between dZ rows: 128 bytes of either neighbour's ends
constexpr int WG_THREADS = 32 * 6;         // warp 0 copies, warp 1 MMAs, warps 2..5 partials
}  // namespace wg

template <int CIN, int COUT> struct WLayout {
  static constexpr int XV = CIN * 2, DV = COUT * 2;    // bytes of a voxel of X and of dZ: the swizzle spans
  static constexpr int XROW = N * XV;
  static constexpr int XGROUP = 4 * XROW;              // rows z - 1, z, z + 1 and the ones row
  static constexpr int DROW = N * DV + wg::PAD;
  static constexpr int HALO = 128 / DV;                // voxels of an end copy (128 bytes)
  static constexpr uint32_t X_TX = 3 * XROW, D_TX = N * DV + 2 * 128;
  static constexpr int NCOLS = 3 * COUT;               // N of one MMA
  static constexpr uint32_t TCOLS = 3 * NCOLS <= 256 ? 256u : 512u;
  static constexpr int ONES = 3 * CIN;                 // accumulator row of the bias gradient
  static constexpr int XRING = wg::XS * XGROUP;
  // with CIN = 16 an A operand reads 8 rows' worth from its group: up to a group past the ring
  static constexpr int D_OFF = XRING + wg::PAD, D_END = D_OFF + wg::DSL * DROW;
  static constexpr int A_END = XRING + (CIN == 16 ? XGROUP : 0);
  static constexpr int BAR_OFF = ((D_END > A_END ? D_END : A_END) + 15) / 16 * 16;
  static constexpr int NBARS = 2 * wg::XS + 2 * wg::DSL + 1;    // xfull, xfree, dfull, dfree, done
  static constexpr int BYTES = BAR_OFF + NBARS * 8 + 16 + 1024;   // + tmem slot, abort, items issued, alignment
  static_assert(NCOLS % 16 == 0 && NCOLS <= 256, "N = 3 COUT must be a valid M = 128 MMA width");
  static_assert(XGROUP % 512 == 0 && DROW % 512 == 0, "rows start on a whole swizzle pattern");
  static_assert(BYTES <= 232448, "shared memory per CTA");
};

// Where a weight-gradient wait gave up: {tag, sequence number, CTA, progress of the MMA warp};
// the first record wins.  Tags: 1 producer xfree, 2 producer dfree, 3 MMA xfull at a segment start,
// 4 MMA xfull per row, 5 MMA dfull, 6 partials-out done.
__device__ int g_wdiag[4];
constexpr long kWSpin = 1L << 20;
__device__ __forceinline__ bool wbar_wait(uint64_t* b, uint32_t parity, volatile int* abort, int tag, int seq, int prog) {
  for (long i = 0; i < kWSpin; ++i) {
    if (bar_try(b, parity)) return true;
    if ((i & 255) == 255 && *abort) return false;
  }
  *abort = 1;
  atomicOr(&g_err, ERR_TIMEOUT);
  if (atomicCAS(&g_wdiag[0], 0, tag) == 0) {
    g_wdiag[1] = seq;
    g_wdiag[2] = (int)blockIdx.x;
    g_wdiag[3] = prog;
  }
  return false;
}

// Shared-memory matrix descriptor, MN-major with rows of VOX = 64 or 32 bytes (VOX / 2 elements along M or
// N) swizzled over that span: 8 K-rows to a group, groups one after another, `lbo` from one span along M
// or N to the next.
template <int VOX> __device__ __forceinline__ uint64_t mdesc_mn(uint32_t addr, uint32_t lbo) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((8 * VOX) >> 4) << 32) | (1ull << 46) | ((VOX == 64 ? 4ull : 6ull) << 61);
}
// kind::f16 instruction descriptor with both operands MN-major (transpose bits 15 and 16)
__host__ __device__ constexpr uint32_t idesc_bf16_mn(int m, int n) { return idesc_bf16(m, n) | (1u << 15) | (1u << 16); }

template <int CIN, int COUT>
__global__ void __launch_bounds__(wg::WG_THREADS, 1) wgrad_tc_kernel(const __grid_constant__ CUtensorMap tm_x,
                                                                     const __grid_constant__ CUtensorMap tm_d,
                                                                     const __grid_constant__ CUtensorMap tm_dend,
                                                                     float* __restrict__ partials) {
  using L = WLayout<CIN, COUT>;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char* sm = smem_raw + ((0u - saddr(smem_raw)) & 1023u);
  unsigned char* xring = sm;
  unsigned char* dring = sm + L::D_OFF;              // first voxel of the first dZ row
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + L::BAR_OFF);
  uint64_t* xfull = bars;
  uint64_t* xfree = bars + wg::XS;
  uint64_t* dfull = bars + 2 * wg::XS;
  uint64_t* dfree = bars + 2 * wg::XS + wg::DSL;
  uint64_t* done = bars + 2 * wg::XS + 2 * wg::DSL;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + L::NBARS);
  volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < wg::XS; ++i) {
      bar_init(&xfull[i], 1);
      bar_init(&xfree[i], 1);
    }
    for (int i = 0; i < wg::DSL; ++i) {
      bar_init(&dfull[i], 1);
      bar_init(&dfree[i], 1);
    }
    bar_init(done, 1);
    *abort = 0;
    fence_bar_init();
  }
  if (warp == 0) {
    tmem_alloc(tmem_slot, L::TCOLS);
    tmem_relinquish();
  }
  // the ones row of every input-group slot (bf16 1.0 = 0x3F80), written once
  {
    const uint4 ones = make_uint4(0x3F803F80u, 0x3F803F80u, 0x3F803F80u, 0x3F803F80u);
    for (int i = threadIdx.x; i < wg::XS * (L::XROW / 16); i += wg::WG_THREADS) {
      const int slot = i / (L::XROW / 16), j = i % (L::XROW / 16);
      *reinterpret_cast<uint4*>(xring + slot * L::XGROUP + 3 * L::XROW + 16 * j) = ones;
    }
  }
  fence_proxy_async();
  tc_before();
  __syncthreads();
  tc_after();
  const uint32_t tmem = *tmem_slot;
  if (warp > CONV_MMA_WARP) {
    const uint32_t lanes = (uint32_t)(32 * (warp & 3)) << 16;
    for (int c = 0; c < (int)L::TCOLS; c += 16) tmem_zero16(tmem + lanes + (uint32_t)c);
    tmem_wait_st();
  }
  tc_before();
  __syncthreads();
  tc_after();
  const Range rg = my_rows();

  if (warp == 0) {
    // ------------------------------------------------------------------ copies
    // Per z-plane segment [yb, ye) of the CTA's rows: X(yb - 1), X(yb), then per output row y: X(y + 1), dZ(y).
    if (lane == 0) {
      int nx = 0, nd = 0;                           // items issued of each kind
      auto issue_x = [&](int z, int yw) -> bool {
        const int slot = nx % wg::XS;
        if (nx >= wg::XS && !wbar_wait(&xfree[slot], (uint32_t)((nx / wg::XS - 1) & 1), abort, 1, nx, nd)) return false;
        bar_expect_tx(&xfull[slot], L::X_TX);
#pragma unroll
        for (int d = 0; d < 3; ++d)
          tma_load3(xring + slot * L::XGROUP + d * L::XROW, &tm_x, &xfull[slot], 0, 0, ((z + d + N - 1) % N) * N + yw);
        ++nx;
        return true;
      };
      auto issue_d = [&](int r) -> bool {
        const int slot = nd % wg::DSL;
        if (nd >= wg::DSL && !wbar_wait(&dfree[slot], (uint32_t)((nd / wg::DSL - 1) & 1), abort, 2, nd, nx)) return false;
        bar_expect_tx(&dfull[slot], L::D_TX);
        unsigned char* dst = dring + slot * L::DROW;
        tma_load3(dst, &tm_d, &dfull[slot], 0, 0, r);
        tma_load3(dst - 128, &tm_dend, &dfull[slot], 0, N - L::HALO, r);
        tma_load3(dst + N * L::DV, &tm_dend, &dfull[slot], 0, 0, r);
        ++nd;
        return true;
      };
      bool ok = true;
      for (int r = rg.r0; r < rg.r1 && ok;) {
        const int z = r / N, yb = r % N;
        const int ye = (z + 1) * N < rg.r1 ? N : rg.r1 - z * N;
        ok = issue_x(z, (yb - 1 + N) % N) && issue_x(z, yb);
        for (int y = yb; y < ye && ok; ++y) ok = issue_x(z, (y + 1) % N) && issue_d(z * N + y);
        r = z * N + ye;
      }
      abort[1] = nx;
      abort[2] = nd;
    }
  } else if (warp == CONV_MMA_WARP) {
    // ---------------------------------------------------------------- MMA issue
    const uint64_t a_base = mdesc_mn<L::XV>(saddr(xring), L::XROW);
    const uint64_t b_base = mdesc_mn<L::DV>(saddr(dring) - L::DV, L::DV);   // dx = +1, 0, -1
    constexpr uint32_t idesc = idesc_bf16_mn(128, L::NCOLS);
    int gx = 0, gd = 0;
    bool ok = true;
    for (int r = rg.r0; r < rg.r1 && ok;) {
      const int z = r / N, yb = r % N;
      const int ye = (z + 1) * N < rg.r1 ? N : rg.r1 - z * N;
      const int nrows = ye - yb;
      auto x_here = [&](int g, int tag) {
        return __all_sync(0xFFFFFFFFu, wbar_wait(&xfull[g % wg::XS], (uint32_t)((g / wg::XS) & 1), abort, tag, g, gd));
      };
      auto row_here = [&](int i, int d) {
        return x_here(gx + i + 2, 4) &&
               __all_sync(0xFFFFFFFFu, wbar_wait(&dfull[d % wg::DSL], (uint32_t)((d / wg::DSL) & 1), abort, 5, d, gx + i + 2));
      };
      ok = x_here(gx, 3) && x_here(gx + 1, 3) && row_here(0, gd);
      for (int i = 0; i < nrows && ok; ++i) {
        tc_after();
        const uint64_t bd = b_base + (uint64_t)((gd % wg::DSL) * (L::DROW / 16));
        bool next_ok = true;
#pragma unroll
        for (int dyi = 0; dyi < 3; ++dyi) {
          // the waits for the next row's items stand before the last dy, beside the MMAs in the queue
          if (dyi == 2 && i + 1 < nrows) {
            next_ok = row_here(i + 1, gd + 1);
            tc_after();
          }
          const uint64_t ad = a_base + (uint64_t)(((gx + i + dyi) % wg::XS) * (L::XGROUP / 16));
          const uint32_t dcol = tmem + (uint32_t)(dyi * L::NCOLS);
#pragma unroll
          for (int ks = 0; ks < N / 16; ++ks) mma_acc(dcol, ad + (uint64_t)(ks * L::XV), bd + (uint64_t)(ks * L::DV), idesc);
        }
        mma_commit(&dfree[gd % wg::DSL]);           // this dZ row is not read again
        mma_commit(&xfree[(gx + i) % wg::XS]);      // nor is input group y - 1
        ++gd;
        ok = next_ok;
      }
      if (!ok) break;
      mma_commit(&xfree[(gx + nrows) % wg::XS]);    // groups ye - 1 and ye end with the segment
      mma_commit(&xfree[(gx + nrows + 1) % wg::XS]);
      gx += nrows + 2;
      r = z * N + ye;
    }
    __syncwarp();
    mma_commit(done);                               // every MMA of this CTA, also after an abort
    // the accumulators are freed only once every MMA issued has completed (bounded)
    for (long i = 0; i < kWSpin && !bar_try(done, 0); ++i) {
    }
  } else {
    // ------------------------------------------------------------------ partials out
    const int q = warp & 3;
    const uint32_t lanes = (uint32_t)(32 * q) << 16;
    const bool ok = wbar_wait(done, 0, abort, 6, 0, 0);
    if (__all_sync(0xFFFFFFFFu, ok)) {
      tc_after();
      const int m = 32 * q + lane;
      float* dst = partials + (size_t)blockIdx.x * 3 * 128 * L::NCOLS;
#pragma unroll
      for (int dyi = 0; dyi < 3; ++dyi) {
#pragma unroll
        for (int c0 = 0; c0 < L::NCOLS; c0 += COUT) {
          float v[COUT];
          const uint32_t ta = tmem + lanes + (uint32_t)(dyi * L::NCOLS + c0);
          if (COUT == 32) tmem_ld32(ta, v); else tmem_ld16(ta, v);
          if (m <= L::ONES) {                       // rows past the ones row's first are not read
            float* row = dst + ((size_t)dyi * 128 + m) * L::NCOLS + c0;
#pragma unroll
            for (int c = 0; c < COUT; c += 4) *reinterpret_cast<float4*>(row + c) = make_float4(v[c], v[c + 1], v[c + 2], v[c + 3]);
          }
        }
      }
    }
  }

  tc_before();
  __syncthreads();
  // no copy outlives the CTA (as in the convolutions)
  if (threadIdx.x == 0 && *abort) {
    const int nx = abort[1], nd = abort[2];
    for (int q = nx > wg::XS ? nx - wg::XS : 0; q < nx; ++q)
      for (long i = 0; i < kWSpin && !bar_try(&xfull[q % wg::XS], (uint32_t)((q / wg::XS) & 1)); ++i) {
      }
    for (int q = nd > wg::DSL ? nd - wg::DSL : 0; q < nd; ++q)
      for (long i = 0; i < kWSpin && !bar_try(&dfull[q % wg::DSL], (uint32_t)((q / wg::DSL) & 1)); ++i) {
      }
  }
  if (warp == 0) {
    __syncwarp();
    tc_after();
    tmem_dealloc(tmem, L::TCOLS);
  }
}

// dW[27][COUT][CIN] and db[COUT] from the per-CTA partials [cta][dy][(dz, ci) | ones][(dx, co)], summed
// over CTAs in a fixed order.  A block takes 32 neighbouring columns of one accumulator row, eight groups
// of CTAs beside each other: contiguous reads, ~20 in flight per thread.  A thread per element of dW, each
// reading its 152 partials one line apart, took 42 us; this 8 us (14.5 MB).
template <int CIN, int COUT>
__global__ void __launch_bounds__(256) wgrad_tc_reduce(const float* __restrict__ partials, int ctas, float* __restrict__ dw,
                                                       float* __restrict__ db) {
  using L = WLayout<CIN, COUT>;
  constexpr int NCOLS = L::NCOLS, PER = 3 * 128 * NCOLS, ROWS = L::ONES + 1;
  __shared__ float part[8][32];
  const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
  const int e = blockIdx.x * 32 + lane;               // element of [3][ROWS][NCOLS]
  const bool here = e < 3 * ROWS * NCOLS;
  const int n = e % NCOLS, m = (e / NCOLS) % ROWS, dyi = e / (NCOLS * ROWS);
  const float* src = partials + ((size_t)dyi * 128 + m) * NCOLS + n;
  const int per = (ctas + 7) / 8, c1 = min(ctas, (g + 1) * per);
  float s = 0.f;
  if (here) {
#pragma unroll 20
    for (int c = g * per; c < c1; ++c) s += __ldcg(src + (size_t)c * PER);
  }
  part[g][lane] = s;
  __syncthreads();
  if (g || !here) return;
  s = 0.f;
#pragma unroll
  for (int q = 0; q < 8; ++q) s += part[q][lane];
  const int dx = 2 - n / COUT, co = n % COUT;         // column blocks: dx = +1, 0, -1
  if (m < L::ONES) dw[((size_t)((m / CIN) * 9 + dyi * 3 + dx) * COUT + co) * CIN + m % CIN] = s;
  else if (dyi == 1 && dx == 1) db[co] = s;           // the ones row, the unshifted dZ
}

// TMA descriptor of a channels-last box [row = z N + y][x][cin]: boxes of `voxels` voxels of one row, swizzled
// over a voxel's bytes
bool row_map(CUtensorMap* m, const void* base, int cin, int voxels) {
  static PFN_cuTensorMapEncodeTiled_v12000 enc = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      enc = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
  });
  if (!enc) return false;
  cuuint64_t dims[3] = {(cuuint64_t)cin, (cuuint64_t)N, (cuuint64_t)N * N};
  cuuint64_t strides[2] = {(cuuint64_t)cin * 2, (cuuint64_t)N * cin * 2};
  cuuint32_t box[3] = {(cuuint32_t)cin, (cuuint32_t)voxels, 1u};
  cuuint32_t estr[3] = {1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, cin == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int CIN, int COUT>
int launch_wgrad(const void* x, const void* dz, float* dw, float* db, float* ws, size_t ws_bytes, cudaStream_t s,
                 std::string* err) {
  using L = WLayout<CIN, COUT>;
  auto kern = wgrad_tc_kernel<CIN, COUT>;
  static unsigned configured = 0u;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  if (!(configured & (1u << (dev & 31)))) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::BYTES) != cudaSuccess) {
      *err = "tcgen05 wgrad: shared memory opt-in failed";
      return ES_E_CUDA;
    }
    configured |= 1u << (dev & 31);
  }
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const size_t need = (size_t)sms * 3 * 128 * L::NCOLS * sizeof(float);
  if (!ws || ws_bytes < need) {
    *err = "tcgen05 wgrad: workspace needs " + std::to_string(need) + " bytes";
    return ES_E_ARG;
  }
  CUtensorMap mx, md, me;
  if (!row_map(&mx, x, CIN, N) || !row_map(&md, dz, COUT, N) || !row_map(&me, dz, COUT, L::HALO)) {
    *err = "tcgen05 wgrad: cuTensorMapEncodeTiled failed";
    return ES_E_CUDA;
  }
  kern<<<sms, wg::WG_THREADS, L::BYTES, s>>>(mx, md, me, ws);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) {
    constexpr int ELEMS = 3 * (L::ONES + 1) * L::NCOLS;
    wgrad_tc_reduce<CIN, COUT><<<(ELEMS + 31) / 32, 256, 0, s>>>(ws, sms, dw, db);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) {
    *err = std::string("tcgen05 wgrad launch: ") + cudaGetErrorString(e);
    return ES_E_CUDA;
  }
  return ES_OK;
}

// ------------------------------------------------------------------ host side
template <int CIN, int COUT, int MODE>
int launch(const void* in, const void* w, const float* bias, void* out, const void* mask, cudaStream_t s,
           std::string* err) {
  using L = Layout<CIN, COUT>;
  auto kern = conv_tc_kernel<CIN, COUT, MODE>;
  static unsigned configured = 0u;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  if (!(configured & (1u << (dev & 31)))) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::BYTES) != cudaSuccess) {
      *err = "tcgen05 conv: shared memory opt-in failed";
      return ES_E_CUDA;
    }
    configured |= 1u << (dev & 31);
  }
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  CUtensorMap row, end;
  if (!row_map(&row, in, CIN, N) || !row_map(&end, in, CIN, L::HALO)) {
    *err = "tcgen05 conv: cuTensorMapEncodeTiled failed";
    return ES_E_CUDA;
  }
  kern<<<sms, CONV_THREADS, L::BYTES, s>>>(row, end, (const __nv_bfloat16*)w, bias, out, (const __nv_bfloat16*)mask);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    *err = std::string("tcgen05 conv launch: ") + cudaGetErrorString(e);
    return ES_E_CUDA;
  }
  return ES_OK;
}

}  // namespace sgtc

// Dispatch for 128^3 boxes; returns ES_E_UNSUPPORTED for a combination that is not compiled.
__attribute__((visibility("hidden"))) int sg_tc_conv_fwd(int cin, int cout, int mode, const void* in, const void* w,
                                                         const float* bias, void* out, const void* mask,
                                                         cudaStream_t s, std::string* err) {
  using namespace sgtc;
  if ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(out) |
       reinterpret_cast<uintptr_t>(mask)) & 15u) {
    *err = "tcgen05 conv: tensors must be 16-byte aligned";
    return ES_E_ARG;
  }
  if (mode == FWD_RELU) {
    if (cin == 16 && cout == 32) return launch<16, 32, FWD_RELU>(in, w, bias, out, mask, s, err);
    if (cin == 32 && cout == 32) return launch<32, 32, FWD_RELU>(in, w, bias, out, mask, s, err);
  } else if (mode == FWD_SIGMOID) {
    if (cin == 32 && cout == 16) return launch<32, 16, FWD_SIGMOID>(in, w, bias, out, mask, s, err);
  } else if (mode == DGRAD_MASK) {
    if (cin == 32 && cout == 32) return launch<32, 32, DGRAD_MASK>(in, w, bias, out, mask, s, err);
    if (cin == 16 && cout == 32) return launch<16, 32, DGRAD_MASK>(in, w, bias, out, mask, s, err);
  }
  *err = "tcgen05 conv: combination not compiled";
  return ES_E_UNSUPPORTED;
}

// Device-side status of the tcgen05 convolutions: nonzero once a wait gave up; reading clears it.
__attribute__((visibility("hidden"))) int sg_tc_status(unsigned* status) {
  unsigned zero = 0;
  cudaError_t e = cudaMemcpyFromSymbol(status, sgtc::g_err, sizeof(unsigned));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(sgtc::g_err, &zero, sizeof(unsigned));
  return e == cudaSuccess ? ES_OK : ES_E_CUDA;
}

// Weight gradient at 128^3 on the tensor cores; ES_E_UNSUPPORTED for a combination not compiled.
__attribute__((visibility("hidden"))) int sg_tc_conv_wgrad(int cin, int cout, const void* x, const void* dz, float* dw,
                                                           float* db, float* ws, size_t ws_bytes, cudaStream_t s,
                                                           std::string* err) {
  using namespace sgtc;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(dz) | reinterpret_cast<uintptr_t>(ws)) & 15u) {
    *err = "tcgen05 wgrad: tensors must be 16-byte aligned";
    return ES_E_ARG;
  }
  if (cin == 16 && cout == 32) return launch_wgrad<16, 32>(x, dz, dw, db, ws, ws_bytes, s, err);
  if (cin == 32 && cout == 32) return launch_wgrad<32, 32>(x, dz, dw, db, ws, ws_bytes, s, err);
  if (cin == 32 && cout == 16) return launch_wgrad<32, 16>(x, dz, dw, db, ws, ws_bytes, s, err);
  *err = "tcgen05 wgrad: combination not compiled";
  return ES_E_UNSUPPORTED;
}

// Workspace of the tensor-core weight gradient (per-CTA partials).
__attribute__((visibility("hidden"))) size_t sg_tc_wgrad_workspace(int cout) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return (size_t)sms * 3 * 128 * 3 * cout * sizeof(float);
}

// The weight gradient's wait record (see g_wdiag); reading clears it.
__attribute__((visibility("hidden"))) int sg_tc_wgrad_diag(int* out4) {
  int zero[4] = {0, 0, 0, 0};
  cudaError_t e = cudaMemcpyFromSymbol(out4, sgtc::g_wdiag, sizeof(zero));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(sgtc::g_wdiag, zero, sizeof(zero));
  return e == cudaSuccess ? ES_OK : ES_E_CUDA;
}
