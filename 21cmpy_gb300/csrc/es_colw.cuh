// Column passes with one warp per few columns (sm_103a).  A tile of TI columns x N elements arrives by
// TMA in a ring of shared-memory buffers (swizzled, so that a warp reads 16-byte pieces of many rows
// without bank conflicts); each warp transforms CPW of the columns in place, with nothing but
// warp-level synchronisation between the Stockham stages, and a producer warp stores finished tiles
// and refills their buffers.
//
// What bounds it: the older form (es_tma.cuh) runs a stage of the whole tile between two CTA barriers
// with 16 warps per SM, and spends as long at barriers and waiting for its copies as issuing (issue
// active 47 % in the z inverse, 37 % in the y inverse at 256^3).  Here warps drift apart, so one
// warp's loads and shared-memory trips hide behind the others' arithmetic, and up to 192 KB of tiles
// are in flight per SM.  The arithmetic is the same operation for operation.  z inverse + filter / y inverse:
// 256^3 30.8 / 24.0 -> 23.1 / 16.9 us, 512^3 245 / 233 -> 205 / 186 us (DRAM).
#pragma once
#include "es_tma.cuh"

namespace es {

// TI columns per tile, CPW columns per warp, NG groups of TI / CPW warps taking tiles in turn, NBUF tile
// buffers.  TI = 0: the size keeps the older form.  Lines with odd factors do not fit the swizzle and
// 1024-point columns would need 64 elements per lane; up to 128 a pass is one or two tiles deep and
// nothing but latency, which the older form's wider split of a tile over threads shortens (z inverse
// / y inverse at 128^3: 7.3 / 5.3 us there, 8.1 / 5.5 us here at the best of five shapes).  512^3: three
// groups hold their 32 elements per lane in registers (four groups: spills, z inverse 295 us against
// 224); tiles twice as wide measured the same in z and 9 % slower in y.
template <int N> struct ColW { static constexpr int TI = 0,  CPW = 2, NG = 1, NBUF = 2; };
template <> struct ColW<256> { static constexpr int TI = 16, CPW = 2, NG = 3, NBUF = 6; };
template <> struct ColW<512> { static constexpr int TI = 8,  CPW = 2, NG = 3, NBUF = 6; };

template <int N, int MODE> struct ColWSmem {
  static constexpr int TI = ColW<N>::TI, CPW = ColW<N>::CPW;
  // z forward + binning: the warps' bins take the place of a tile (nothing is stored, so that a buffer is
  // refilled as soon as its tile is binned).  512^3: 420 us in the CTA-wide form, 282 us here (the plain
  // pass takes 190 us); delta_T and P(k) of a 256^3 box with 100 bins: 155 -> 150 us
  static constexpr int NBUF = ColW<N>::NBUF - (MODE == COL_Z_FWD_PK ? 1 : 0);
  static constexpr int WPT = TI ? TI / CPW : 1, NW = ColW<N>::NG * WPT, T = 32 * (NW + 1);
  static constexpr int tile = N * TI * 8;
  // per-warp filter weights, or per-warp bins and the thresholds
  static constexpr int wts = MODE == COL_Z_INV_FILTER ? NW * CPW * (N / 2 + 1) * 4
                             : MODE == COL_Z_FWD_PK   ? (NW * 3 + 1) * PK_MAX_BINS * 4 : 0;
  // [NBUF tiles | 2 NBUF mbarriers | twiddles by stage | filter weights or bins] after aligning the base to 1024
  static constexpr int bytes = NBUF * tile + 2 * NBUF * 8 + N * 8 + wts + 1024;
};

// The tiles one CTA takes, in order.  Plain passes: tiles blockIdx.x + k gridDim.x, groups in turn.  The
// z inverse + filter pass: the CTA's mirror-plane pairs (planes j and N - j of one column block have
// the same |k|^2 column by column, so the filter weights of the first serve the second) NG at a time,
// the NG first planes before the NG second ones, so that a group meets its pair in two tiles of its
// own; then its share of the remaining tiles (planes 0 and N/2, and the Nyquist plane), groups in
// turn, dealt from the last CTA, which has the fewest pairs.
struct ColWTile { int plane, c; bool nyq; };
template <int N, int MODE> struct ColWSeq {
  static constexpr int TI = ColW<N>::TI, CPR = (N / 2) / TI, NG = ColW<N>::NG;
  static constexpr bool ZPASS = MODE == COL_Z_FWD || MODE == COL_Z_INV_FILTER || MODE == COL_Z_INV || MODE == COL_Z_FWD_PK;
  static constexpr bool PAIRS = MODE == COL_Z_INV_FILTER;
  static constexpr int NPAIR = (N / 2 - 1) * CPR, NREST = 2 * CPR + N / TI;
  static constexpr int NTILES = N * CPR + (ZPASS ? N / TI : 0);
  int pairs = 0, count = 0;
  __device__ __forceinline__ ColWSeq() {
    const int b = blockIdx.x, G = gridDim.x, rb = G - 1 - b;
    if (PAIRS) {
      pairs = b < NPAIR ? (NPAIR - 1 - b) / G + 1 : 0;
      count = 2 * pairs + (rb < NREST ? (NREST - 1 - rb) / G + 1 : 0);
    } else {
      count = b < NTILES ? (NTILES - 1 - b) / G + 1 : 0;
    }
  }
  // plane `second` of the CTA's u-th pair
  __device__ __forceinline__ ColWTile pair(int u, bool second) const {
    const int unit = blockIdx.x + u * gridDim.x, j = unit / CPR + 1;
    return {second ? N - j : j, unit % CPR, false};
  }
  // its k-th tile besides the pairs
  __device__ __forceinline__ ColWTile single(int k) const {
    int tile = PAIRS ? (int)(gridDim.x - 1 - blockIdx.x) + k * (int)gridDim.x : (int)(blockIdx.x + k * gridDim.x);
    if (PAIRS) {
      if (tile < 2 * CPR) return {tile < CPR ? 0 : N / 2, tile % CPR, false};
      tile += N * CPR - 2 * CPR;
    }
    if (ZPASS && tile >= N * CPR) return {0, tile - N * CPR, true};
    return {tile / CPR, tile % CPR, false};
  }
  // its it-th tile (the order the producer moves them in)
  __device__ __forceinline__ ColWTile at(int it) const {
    if (!PAIRS || it >= 2 * pairs) return single(it - 2 * pairs);
    const int round = it / (2 * NG), off = it - round * 2 * NG, k = min(NG, pairs - round * NG);
    return pair(round * NG + (off >= k ? off - k : off), off >= k);
  }
};

// A wait that ends on completion, after the polls run out (recorded; the CTA aborts) or once another
// role has aborted.
__device__ __forceinline__ bool colw_wait(uint64_t* bar, uint32_t parity, const OpArgs& a, volatile int* abort) {
  const long limit = 1L << (a.wait_log2 > 0 ? a.wait_log2 : kWaitLog2);
  for (long i = 0; i < limit; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 15) == 15 && *abort) return false;
  }
  atomicOr(a.err, ES_DEV_ERR_TIMEOUT);
  *abort = 1;
  return false;
}

// The in-place transform of a warp's CPW columns of a swizzled tile.  A lane owns column l = lane & 1 of
// its 16-byte pieces (two columns each); piece q of the warp is the tile's piece `piece0 + q`.  Element e
// lies in row e; between stages 0 and 1 in row e ^ ((e / R0) mod 8), so that both the stride-R0 stores and
// the unit-stride loads touch eight different rows mod 8 in every eight lanes.
template <int N> struct WarpFft {
  static constexpr int TI = ColW<N>::TI, CPW = ColW<N>::CPW, ROWB = TI * 8;
  static constexpr int STAGES = Plan<N, 0>::stages, R0 = Plan<N, 0>::radix[0];
  static constexpr int LOG0 = R0 == 16 ? 4 : 3;
  static_assert(R0 == 16 || R0 == 8, "first radix 8 or 16");
  // byte offset of piece p of a row whose index mod 8 is x, relative to the row (TMA swizzle of
  // 16-byte pieces within 128 bytes: rows of 128, 64 or 32 bytes)
  static __device__ __forceinline__ int piece(int p, int x) {
    return (p ^ (ROWB == 128 ? x : ROWB == 64 ? (x >> 1) : (x >> 2))) << 4;
  }
  // change of a row's byte offset (piece included) when its index mod 8 is XORed with the constant x
  static __host__ __device__ constexpr int flip(int x) { return x * ROWB | ((ROWB == 128 ? x : ROWB == 64 ? (x >> 1) : (x >> 2)) << 4); }
  static __host__ __device__ constexpr int tw_offset(int s) {                // stage s's twiddles [r - 1][k] in the stage table
    int off = 0, ns = 1;
    for (int i = 0; i < s; ++i) { off += i ? (Plan<N, 0>::radix[i] - 1) * ns : 0; ns *= Plan<N, 0>::radix[i]; }
    return off;
  }
  static __device__ __forceinline__ void load_twiddles(float2* tws, const float2* tw, int tid, int nt) {
    stage_twiddles<1>(tws, tw, tid, nt);
  }
  template <int S> static __device__ __forceinline__ void stage_twiddles(float2* tws, const float2* tw, int tid, int nt) {
    if constexpr (S < STAGES) {
      constexpr int R = Plan<N, 0>::radix[S], Ns = StageNs<N, S, 0>::value;
      for (int i = tid; i < (R - 1) * Ns; i += nt) tws[tw_offset(S) + i] = tw[(i % Ns) * (i / Ns + 1) * (N / (Ns * R))];
      stage_twiddles<S + 1>(tws, tw, tid, nt);
    }
  }
  template <int S, bool INV, class Pre>
  static __device__ __forceinline__ void stage(unsigned char* buf, int piece0, const float2* tws, Pre pre) {
    constexpr int R = Plan<N, 0>::radix[S], Ns = StageNs<N, S, 0>::value, NR = N / R;
    constexpr int NBL = NR * (CPW / 2) / 16;             // butterflies per lane
    static_assert(NBL * 16 == NR * (CPW / 2) && NR % 8 == 0 && (S == 0 || Ns % 8 == 0), "whole octets of rows");
    const int lane = threadIdx.x & 31, l = lane & 1;
    float2 v[NBL][R];
#pragma unroll
    for (int i = 0; i < NBL; ++i) {
      const int bi = (lane >> 1) + 16 * i, j = bi % NR, q = bi / NR, p = piece0 + q;
      if (S == 1 && NR == R0) {                          // row (j ^ (r mod 8)) + r NR
        const unsigned char* at = buf + l * 8;
        const int base = j * ROWB + piece(p, j & 7);
#pragma unroll
        for (int r = 0; r < R; ++r)
          v[i][r] = *reinterpret_cast<const float2*>(at + (base ^ flip(r & 7)) + r * NR * ROWB);
      } else {
        const int row = S == 1 ? j ^ ((j >> LOG0) & 7) : j;
        const unsigned char* at = buf + l * 8 + row * ROWB + piece(p, row & 7);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          v[i][r] = *reinterpret_cast<const float2*>(at + r * NR * ROWB);
          if (S == 0) v[i][r] = pre(2 * q + l, j + r * NR, r >= R / 2, v[i][r]);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < NBL; ++i) {
      if (S > 0) {
        const int k = (((lane >> 1) + 16 * i) % NR) % Ns;
        const float2* t = tws + tw_offset(S) + k;
#pragma unroll
        for (int r = 1; r < R; ++r) {
          const float2 w = t[(r - 1) * Ns];
          v[i][r] = twid<INV>(v[i][r], w.x, w.y);
        }
      }
      Dft<R, INV>::run(v[i]);
    }
    __syncwarp();                                        // every lane has read: write in place
#pragma unroll
    for (int i = 0; i < NBL; ++i) {
      const int bi = (lane >> 1) + 16 * i, j = bi % NR, q = bi / NR, p = piece0 + q;
      if (S == 0 && STAGES > 1) {                        // row j R + (r ^ (j mod 8))
        unsigned char* at = buf + l * 8 + j * R * ROWB;
        const int base = (j & 7) * ROWB + piece(p, j & 7);
#pragma unroll
        for (int r = 0; r < R; ++r) *reinterpret_cast<float2*>(at + (base ^ flip(r & 7)) + (r >> 3) * 8 * ROWB) = v[i][r];
      } else {
        const int row = (j / Ns) * Ns * R + (j % Ns);
        unsigned char* at = buf + l * 8 + row * ROWB + piece(p, row & 7);
#pragma unroll
        for (int r = 0; r < R; ++r) *reinterpret_cast<float2*>(at + r * Ns * ROWB) = v[i][r];
      }
    }
    __syncwarp();
    if constexpr (S + 1 < STAGES) stage<S + 1, INV>(buf, piece0, tws, pre);
  }
};

template <int N, int MODE>
__global__ void __launch_bounds__(ColWSmem<N, MODE>::T, 1) col_warp(const __grid_constant__ typename ColArgs<MODE>::type a) {
  using SM = ColWSmem<N, MODE>;
  using F = WarpFft<N>;
  constexpr int M = N / 2, TI = SM::TI, CPW = SM::CPW, WPT = SM::WPT, NBUF = SM::NBUF, ROWB = TI * 8;
  constexpr int BOX = N < 256 ? N : 256;
  static_assert(NBUF >= 2, "a buffer is refilled only after the next tile's store is on its way");
  constexpr bool PK = MODE == COL_Z_FWD_PK;
  constexpr bool INV = MODE == COL_Z_INV_FILTER || MODE == COL_Y_INV || MODE == COL_Z_INV;
  constexpr bool ZPASS = ColWSeq<N, MODE>::ZPASS;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char* base = align_smem<1024>(smem_raw);
  uint64_t* full = reinterpret_cast<uint64_t*>(base + NBUF * SM::tile);
  uint64_t* done = full + NBUF;
  float2* tws = reinterpret_cast<float2*>(done + NBUF);
  float* wts = reinterpret_cast<float*>(tws + N);
  __shared__ int s_abort;
  volatile int* abort = &s_abort;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const ColWSeq<N, MODE> seq;

  auto load = [&](int it) {
    const ColWTile t = seq.at(it);
    uint64_t* bar = &full[it % NBUF];
    unsigned char* dst = base + (it % NBUF) * SM::tile;
    mbar_expect_tx(bar, (uint32_t)SM::tile + stall_bytes(a.stall, it));
    const uint64_t pol = l2_policy(a.hint_in);
#pragma unroll
    for (int h = 0; h < N / BOX; ++h) {
      unsigned char* d = dst + h * BOX * ROWB;
      if (t.nyq) tma_load2(d, &a.tm_in_nyq, bar, t.c * TI, h * BOX, pol);
      else if (ZPASS) tma_load3(d, &a.tm_in, bar, t.c * TI, t.plane, h * BOX, pol);
      else tma_load3(d, &a.tm_in, bar, t.c * TI, h * BOX, t.plane, pol);
    }
  };
  if (threadIdx.x == 32 * SM::NW) {
    s_abort = 0;
    for (int b = 0; b < NBUF; ++b) {
      mbar_init(&full[b], 1);
      mbar_init(&done[b], WPT);
    }
    fence_mbar_init();
    fence_async_smem();
  }
  F::load_twiddles(tws, a.tw, threadIdx.x, SM::T);
  int* sthr = reinterpret_cast<int*>(wts + SM::NW * 3 * PK_MAX_BINS);
  if constexpr (PK) {
    for (int i = threadIdx.x; i < SM::NW * 3 * PK_MAX_BINS; i += SM::T) wts[i] = 0.f;
    for (int i = threadIdx.x; i < a.nbins; i += SM::T) sthr[i] = a.thr[i];
  }
  if (!a.early) pdl_wait();
  if (threadIdx.x == 32 * SM::NW) {
    for (int it = 0; it < NBUF && it < seq.count; ++it) load(it);
    if (!a.early) pdl_trigger();
  }
  __syncthreads();

  if (warp == SM::NW) {
    // ------------------------------------------------------------------ producer: one lane
    if (lane == 0) {
      int loaded = seq.count < NBUF ? seq.count : NBUF;
      for (int it = 0; it < seq.count; ++it) {
        if (!colw_wait(&done[it % NBUF], (uint32_t)((it / NBUF) & 1), a, abort)) break;
        if (PK) {
          if (loaded < seq.count) load(loaded++);
          continue;
        }
        if (a.early && it == 0) {
          pdl_wait();
          pdl_trigger();
        }
        const ColWTile t = seq.at(it);
        const unsigned char* src = base + (it % NBUF) * SM::tile;
        const uint64_t pol = l2_policy(a.hint_out);
#pragma unroll
        for (int h = 0; h < N / BOX; ++h) {
          const unsigned char* s = src + h * BOX * ROWB;
          if (t.nyq) tma_store2(&a.tm_out_nyq, s, t.c * TI, h * BOX, pol);
          else if (ZPASS) tma_store3(&a.tm_out, s, t.c * TI, t.plane, h * BOX, pol);
          else tma_store3(&a.tm_out, s, t.c * TI, h * BOX, t.plane, pol);
        }
        bulk_commit();
        // tile it - 1 has left its buffer once all but the newest store have read theirs
        if (it >= 1 && loaded < seq.count) {
          asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
          load(loaded++);
        }
      }
      // no copy outlives the CTA: after an abort, the loads in flight land first (bounded)
      if (*abort)
        for (int it = loaded > NBUF ? loaded - NBUF : 0; it < loaded; ++it)
          mbar_wait(&full[it % NBUF], (uint32_t)((it / NBUF) & 1), a.wait_log2);
      if (a.early) pdl_wait();                           // also where this CTA has stored nothing
      bulk_wait0();
    }
    if constexpr (PK) {
      __syncwarp();
      pk_finish<SM::T, SM::NW>(wts, a);
    }
    return;
  }

  // -------------------------------------------------------------------- transforms
  const int group = warp / WPT, wt = warp % WPT, piece0 = wt * (CPW / 2);
  float* w = wts + warp * CPW * (M + 1);
  // W depends on |k|^2 = kz^2 + (ky^2 + kx^2 of the column): N/2 + 1 values per column, computed while the
  // tile is on its way
  auto weights = [&](const ColWTile& t) {
    const float scale = a.scale * a.inv_n3;
    auto put = [&](int cl, int kz) {
      const int col = t.c * TI + wt * CPW + cl;
      const int ck2 = !t.nyq ? wrap2<N>(t.plane) + col * col : wrap2<N>(col) + M * M;
      w[cl * (M + 1) + kz] = filter_weight(kz * kz + ck2, a.dk, a.fR, a.fk2cut, a.filter, a.ref_compat) * scale;
    };
    __syncwarp();
#pragma unroll 1
    for (int q = lane; q < CPW * M; q += 32) put(q / M, q % M);
    if (lane < CPW) put(lane, M);
    __syncwarp();
  };
  // meets the group's warps; true if all of them say so (they leave an aborted pass together)
  auto group_agrees = [&](int g, bool mine) {
    int r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\tbar.red.and.pred q, %2, %3, p;\n\tselp.s32 %0, 1, 0, q;\n\t}"
                 : "=r"(r) : "r"((int)mine), "r"(g + 1), "n"(32 * WPT) : "memory");
    return r != 0;
  };
  // transforms the CTA's it-th tile; false: aborted
  auto transform = [&](int it, const ColWTile& t) {
    unsigned char* buf = base + (it % NBUF) * SM::tile;
    const bool ok = colw_wait(&full[it % NBUF], (uint32_t)((it / NBUF) & 1), a, abort);
    const bool all_ok = __all_sync(0xffffffffu, ok);
    if (PK && !all_ok) return group_agrees(group, false);
    if (!all_ok) return false;
    if (MODE == COL_Z_INV_FILTER) {
      F::template stage<0, INV>(buf, piece0, tws, [&](int col, int k, bool upper, float2 v) {
        return cscale(v, w[col * (M + 1) + (upper ? N - k : k)]);
      });
    } else if (MODE == COL_Y_INV && t.c == 0 && wt == 0) {
      const float2* nyq = a.cin_nyq + (size_t)t.plane * N;
      F::template stage<0, INV>(buf, piece0, tws, [&](int col, int j, bool, float2 v) {
        if (col == 0) {                                  // u = y0 + i yM (both Hermitian columns)
          const float2 ym = nyq[j];
          v = make_float2(v.x - ym.y, v.y + ym.x);
        }
        return v;
      });
    } else {
      F::template stage<0, INV>(buf, piece0, tws, [](int, int, bool, float2 v) { return v; });
    }
    if (MODE == COL_Y_FWD && t.c == 0 && wt == 0) {
      // split the packed column 0: FFT(x0) stays, FFT(xM) goes to the Nyquist plane
      constexpr int Q = N / 32;
      float2 av[Q], bv[Q];
      auto at = [&](int row) { return reinterpret_cast<float2*>(buf + row * ROWB + F::piece(0, row & 7)); };
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int j = lane + 32 * q;
        const float2 v = *at(j), u = *at((N - j) % N);
        av[q] = make_float2(0.5f * (v.x + u.x), 0.5f * (v.y - u.y));
        bv[q] = make_float2(0.5f * (v.y + u.y), -0.5f * (v.x - u.x));
      }
      __syncwarp();
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int j = lane + 32 * q;
        *at(j) = av[q];
        a.cout_nyq[(size_t)t.plane * N + j] = bv[q];
      }
    }
    if constexpr (PK) {
      // all of the group's columns, TI neighbouring threads on a row: a warp sees few values of |kz| and so
      // few bins (its own columns from end to end would be all bins: 131 us at 256^3 with 100 bins)
      if (!group_agrees(group, true)) return false;
      constexpr int GT = 32 * WPT;
      const int tid = wt * 32 + lane, col = tid % TI, kx = t.c * TI + col;
      const int ck2 = t.nyq ? wrap2<N>(kx) + M * M : wrap2<N>(t.plane) + kx * kx;
      float* wb = wts + warp * 3 * PK_MAX_BINS;
      pk_bin_segment<N, (M * TI + GT - 1) / GT>(
          [&](int k) { return *reinterpret_cast<const float2*>(buf + k * ROWB + F::piece(col >> 1, k & 7) + (col & 1) * 8); },
          tid / TI, ck2, t.nyq || kx == 0 ? 1u : 2u, sthr, a.nbins, a.dk, a.volume, wb, wb + PK_MAX_BINS, pk_counts(wb));
    }
    fence_async_smem();
    __syncwarp();
    if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&done[it % NBUF])) : "memory");
    return true;
  };
  for (int u = group; u < seq.pairs; u += ColW<N>::NG) {
    const int round0 = u - group, k = min(ColW<N>::NG, seq.pairs - round0);
    const ColWTile t = seq.pair(u, false);
    weights(t);
    if (!transform(2 * round0 + group, t)) return;
    if (!transform(2 * round0 + k + group, seq.pair(u, true))) return;
  }
  for (int k = group; 2 * seq.pairs + k < seq.count; k += ColW<N>::NG) {
    const ColWTile t = seq.single(k);
    if (MODE == COL_Z_INV_FILTER) weights(t);
    if (!transform(2 * seq.pairs + k, t)) break;
  }
  if constexpr (PK) pk_finish<SM::T, SM::NW>(wts, a);
}

}  // namespace es
