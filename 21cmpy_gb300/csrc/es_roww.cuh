// Row C2R pass with one warp per few rows (sm_103a): half-spectrum rows -> real rows, with the
// excursion-set epilogue or a plain store.  A warp owns RW = 32 / NSL rows of every tile of its CTA (NSL:
// butterflies of the last stage), copies them in by itself (1-D bulk copies on its own mbarriers, the
// next tile's rows and previous-radius delta_R in flight), and takes them through the Hermitian split,
// both Stockham stages and the epilogue with warp-level synchronisation only:
//
//   * the split feeds the first stage in registers: a lane reads the elements of its butterfly and
//     their mirror images and forms Z[e] = (X[e] + conj X[M-e]) + U[e] (X[e] - conj X[M-e]) itself;
//   * the one exchange between the stages goes through the rows' own buffer, skewed so that neither
//     side has bank conflicts;
//   * the second stage's outputs stay in registers for the erfc sum, the previous radius' test and
//     the store.
//
// What bounds it: instruction issue (the erfc sum is half of it).  The older form (es_rows.cuh) spent
// 1018 warp instructions per tile and warp at 256^3, with four CTA barriers a tile (issue active 60 %).
// 256^3: 46.5 -> 38.8 us; 512^3: 395 -> 260 us, 1.6 GB at 0.91 of the copy rate.
// Thread for thread, the last stage, the running sums and the grid are the older form's, so the
// grid-wide sums come out the same bit for bit.
#pragma once
#include "es_rows.cuh"

namespace es {

// NP: previous-radius buffers per warp; 0: the size keeps the older form (two stages with whole
// warps of butterflies are needed; the small sizes are a single short tile per CTA).
template <int N> struct RowW { static constexpr int NP = 0; };
template <> struct RowW<128> { static constexpr int NP = 1; };   // one tile per CTA, mostly
template <> struct RowW<256> { static constexpr int NP = 2; };
template <> struct RowW<512> { static constexpr int NP = 2; };

template <int N> struct RowWCfg {
  static constexpr int M = N / 2, RL = Row2Cfg<N>::RL, NP = RowW<N>::NP;
  static constexpr int R0 = Plan<M, 0>::radix[0], R1 = Plan<M, 0>::radix[Plan<M, 0>::stages - 1];
  static constexpr int NSL = R0;                         // butterflies per row of the last of two stages
  static constexpr int RW = 32 / NSL;                    // rows per warp
  static constexpr int NW = RL / RW, T = 32 * NW;        // warps and threads of a CTA
  static constexpr bool HALF = RW * R1 * 2 == 32;        // first stage: two lanes per butterfly
  // rows of 64 elements: every other row starts half a bank cycle later, so 16 lanes on two rows
  // touch all 32 banks
  static constexpr int PITCH = M + (NSL == 8 ? 8 : 0);   // complex elements
  static constexpr int XBUF = RW * PITCH * 8;            // bytes of one buffer
  static constexpr int TW = (R1 - 1) * NSL;              // last stage's twiddles
  // [U | twiddles | per warp: 4 mbarriers | per warp: 2 spectrum, NP previous-radius buffers]
  static constexpr int BARS = (M + TW) * 8, BUFS = (BARS + NW * 32 + 127) / 128 * 128;
  static constexpr int bytes = BUFS + NW * (2 + NP) * XBUF + 128;
};

// Grid-wide sum with the summation order of a CTA of TV threads whose warps past NW hold zeros
// (grid_sum<TV>, es_kernels.cuh).
template <int TV, int NW>
__device__ __forceinline__ bool grid_sum_as(float mine, float* partials, unsigned* counter, float* sred, float* total) {
  __shared__ unsigned s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float v = warp_sum(mine);
  __syncthreads();
  if (lane == 0) sred[warp] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    float s = 0.f;
    for (int w = 0; w < NW; ++w) s += sred[w];
    partials[blockIdx.x] = s;
    __threadfence();
    s_last = (atomicAdd(counter, 1u) == gridDim.x - 1) ? 1u : 0u;
  }
  __syncthreads();
  if (!s_last) return false;
  __threadfence();
  for (int vw = warp; vw < TV / 32; vw += NW) {
    float acc = 0.f;
    for (int i = vw * 32 + lane; i < (int)gridDim.x; i += TV) acc += __ldcg(partials + i);
    acc = warp_sum(acc);
    if (lane == 0) sred[vw] = acc;
  }
  __syncthreads();
  float s = 0.f;
  for (int w = 0; w < TV / 32; ++w) s += sred[w];
  if (threadIdx.x == 0) *counter = 0u;
  *total = s;
  return true;
}

// First-stage butterfly of a lane (h: its half where two lanes share one).
template <class C, bool INV> __device__ __forceinline__ void row_first_dft(float2* v, int h) {
  if constexpr (C::HALF) {
    // radix 16 over two lanes: each takes the radix-8 DFT of the even or the odd samples, the odd
    // ones are turned by w_16^k, and the halves are combined across the pair (Dft<16>)
    static_assert(C::R0 == 16, "half butterflies are radix 8");
    constexpr float c1 = 0.92387953251128674f, s1 = 0.38268343236508978f, rt = 0.70710678118654752f;
    Dft<8, INV>::run(v);
    if (h) {
      v[1] = twid<INV>(v[1], c1, -s1);
      v[2] = twid<INV>(v[2], rt, -rt);
      v[3] = twid<INV>(v[3], s1, -c1);
      v[4] = rot<INV>(v[4]);
      v[5] = twid<INV>(v[5], -s1, -c1);
      v[6] = twid<INV>(v[6], -rt, -rt);
      v[7] = twid<INV>(v[7], -c1, -s1);
    }
    const float sg = h ? -1.0f : 1.0f;
#pragma unroll
    for (int k = 0; k < 8; ++k) {                      // even lane: e + o; odd lane: e - o (outputs 8 + k)
      const float ox = __shfl_xor_sync(0xffffffffu, v[k].x, 1), oy = __shfl_xor_sync(0xffffffffu, v[k].y, 1);
      v[k] = make_float2(fmaf(v[k].x, sg, ox), fmaf(v[k].y, sg, oy));
    }
  } else {
    Dft<C::R0, INV>::run(v);
  }
}

template <int N, int EPI>
__global__ void __launch_bounds__(RowWCfg<N>::T, RowOcc<N, 0>::MINB) row_warp_c2r(const __grid_constant__ OpArgs a) {
  using C = RowWCfg<N>;
  constexpr int M = C::M, RL = C::RL, RW = C::RW, R0 = C::R0, R1 = C::R1, NSL = C::NSL, NP = C::NP, PITCH = C::PITCH;
  constexpr int TV = Row2Cfg<N>::T;                      // threads of the older form's CTA
  constexpr bool HALF = C::HALF;
  constexpr int J0 = R1;                                 // butterflies per row of the first stage
  constexpr int V0 = HALF ? R0 / 2 : R0;                 // elements per lane in the first stage
  static_assert(Plan<M, 0>::stages == 2 && RW * NSL == 32 && (HALF || RW * J0 == 32) && RW * C::NW == RL, "two full stages");
  static_assert(R1 == 8 || R1 == 16, "skew of the exchange");
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char* base = align_smem<128>(smem_raw);
  float2* U = reinterpret_cast<float2*>(base);
  float2* tws = U + M;
  __shared__ float sred[TV / 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint64_t* bars = reinterpret_cast<uint64_t*>(base + C::BARS) + 4 * warp;   // [0, 1] spectrum, [2, 3] previous radius
  unsigned char* bufs = base + C::BUFS + warp * (2 + NP) * C::XBUF;

  constexpr int ntiles = N * N / RL;
  const int my_count = (int)blockIdx.x < ntiles ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  const bool has_prev = EPI == EPI_IONIZE && a.has_prev;
  // first pair of this warp's rows of its CTA's it-th tile (at most 512^3 / 2 pairs: 32 bits)
  auto pair_at = [&](int it) { return ((blockIdx.x + it * gridDim.x) * RL + warp * RW) * M; };
  auto copy_in = [&](const float2* src, unsigned char* dst, uint64_t* bar, uint32_t extra, int hint) {
    const uint64_t pol = l2_policy(hint);
    mbar_expect_tx(bar, (uint32_t)(RW * M * 8) + extra);
    if (PITCH == M) {
      bulk_load(dst, src, RW * M * 8, bar, pol);
    } else {
#pragma unroll
      for (int l = 0; l < RW; ++l) bulk_load(dst + l * PITCH * 8, src + l * M, M * 8, bar, pol);
    }
  };
  auto issue = [&](int it) {
    copy_in(a.cin + pair_at(it), bufs + (it & 1) * C::XBUF, &bars[it & 1], stall_bytes(a.stall, it), a.hint_in);
  };
  auto issue_prev = [&](int it) {
    copy_in(a.prev + pair_at(it), bufs + (2 + it % NP) * C::XBUF, &bars[2 + it % NP], 0u, ES_HINT_EVICT_FIRST);
  };
  if (lane == 0) {
    for (int b = 0; b < 4; ++b) mbar_init(&bars[b], 1);
    fence_mbar_init();
    fence_async_smem();
    if (has_prev && a.early)
      for (int it = 0; it < NP && it < my_count; ++it) issue_prev(it);
  }
  // U[e] = w^-e for e <= M/2, and -w^(M-e) (the same number as the split of the older form takes it) past it
  for (int e = threadIdx.x; e < M; e += C::T) {
    const float2 w = a.tw[e <= M / 2 ? e : M - e];
    U[e] = e <= M / 2 ? cconj(w) : make_float2(-w.x, -w.y);
  }
  for (int i = threadIdx.x; i < C::TW; i += C::T) tws[i] = a.tw[(i % NSL) * (i / NSL + 1) * 2];
  pdl_wait();
  if (lane == 0) {
    for (int it = 0; it < 2 && it < my_count; ++it) issue(it);
    if (has_prev && !a.early)
      for (int it = 0; it < NP && it < my_count; ++it) issue_prev(it);
  }
  pdl_trigger();
  // previous radius: erfc((dc - d) / denom_prev) * norm_prev >= 1/zeta  <=>  d >= thr_prev
  float thr_prev = __int_as_float(0x7f800000);
  if (has_prev) {
    const float y = a.inv_zeta / a.stats_prev[2];
    if (y < 2.0f) thr_prev = a.dc - a.denom_prev * erfcinvf(y);
  }
  const f32x2 DC = bc2(a.dc), INV = bc2(EPI == EPI_IONIZE ? 1.0f / a.denom : 0.f);
  f32x2 acc = bc2(0.0f);                                 // two running sums (even, odd voxels)
  __syncthreads();

  // first stage: lane = (row l0, butterfly j0[, half h]); last stage: lane = (row l, butterfly j)
  const int l0 = HALF ? lane / (2 * J0) : lane / J0, j0 = HALF ? (lane >> 1) % J0 : lane % J0, h = HALF ? lane & 1 : 0;
  const int l = lane / NSL, j = lane % NSL;
  bool ok = true;
  int it = 0;
  for (; it < my_count; ++it) {
    float2* X = reinterpret_cast<float2*>(bufs + (it & 1) * C::XBUF);
    const uint32_t pair0 = pair_at(it);
    ok = __all_sync(0xffffffffu, mbar_wait(&bars[it & 1], (uint32_t)((it >> 1) & 1), a.wait_log2));
    if (!ok) break;
    // element r of butterfly j0 is e = j0 + r M / R0; a half-butterfly takes r = 2 k + h
    float2 v[V0];
    {
      const float2* x = X + l0 * PITCH;
      const int e0 = j0 + h * (M / R0);
#pragma unroll
      for (int k = 0; k < V0; ++k) {
        const int e = e0 + k * (HALF ? 2 : 1) * (M / R0);
        const float2 own = x[e], u = U[e];
        const float2 oth = x[k == 0 ? (M - e) & (M - 1) : M - e];
        const float2 t1 = cmul(u, make_float2(own.x - oth.x, own.y + oth.y));
        v[k] = make_float2(own.x + oth.x - t1.y, own.y - oth.y + t1.x);
        if (k == 0 && e == 0) v[k] = make_float2(own.x + own.y, own.x - own.y);   // (X[0], X[N/2]), both real
      }
    }
    if (a.discard_in) {
      // the intermediate spectrum is dead once copied: drop its lines from L2 unwritten
      const float2* g = a.cin + pair0 + 16 * lane;
#pragma unroll
      for (int q = 0; q < RW * M / 16; q += 32)
        if (q + lane < RW * M / 16) l2_discard(g + 16 * q);
    }
    row_first_dft<C, true>(v, h);
    __syncwarp();                                        // every lane has read its rows
    // exchange: output r of butterfly j0 goes to slot j0 R0 + (r ^ j0)
    {
      float2* x = X + l0 * PITCH + j0 * R0 + h * V0;
#pragma unroll
      for (int k = 0; k < V0; ++k) x[k ^ (HALF ? (j0 & 7) : j0)] = v[k];
    }
    __syncwarp();
    float2 z[R1];
    {
      const float2* x = X + l * PITCH;
#pragma unroll
      for (int r = 0; r < R1; ++r) z[r] = x[r * R0 + (j ^ r)];
    }
    // the buffer takes the tile after next
    fence_async_smem();
    __syncwarp();
    if (lane == 0 && it + 2 < my_count) issue(it + 2);
#pragma unroll
    for (int r = 1; r < R1; ++r) {
      const float2 w = tws[(r - 1) * NSL + j];
      z[r] = twid<true>(z[r], w.x, w.y);
    }
    Dft<R1, true>::run(z);
    // element p = j + r NSL of row l
    const uint32_t row0 = pair0 + l * M;
    float2* out = a.rout + row0 + j;
    if (EPI == EPI_STORE) {
#pragma unroll
      for (int r = 0; r < R1; ++r) out[r * NSL] = cscale(z[r], a.scale);
      continue;
    }
    // the erfc sum first: the chains are independent and overlap
    {
      f32x2 e[R1];
#pragma unroll
      for (int r = 0; r < R1; ++r) e[r] = erfc_sum_pair(mul2(sub2(DC, pk2(z[r].x, z[r].y)), INV));
#pragma unroll
      for (int r = 0; r < R1; ++r) acc = add2(acc, e[r]);
    }
    // the previous radius' delta_R of this lane's elements
    const float2* pv = reinterpret_cast<const float2*>(bufs + (2 + it % NP) * C::XBUF) + l * PITCH + j;
    if (has_prev) {
      ok = __all_sync(0xffffffffu, mbar_wait(&bars[2 + it % NP], (uint32_t)((it / NP) & 1), a.wait_log2));
      if (!ok) break;
    }
    if (a.marker) {
      // centre mode: whether a cell passed at an earlier radius travels in the lowest mantissa bit of
      // delta_R (a change of at most one unit in the last place), so the next radius carries it on
#pragma unroll
      for (int r = 0; r < R1; ++r) {
        unsigned fx = 0u, fy = 0u;                       // flags in bit 0
        if (has_prev) {
          const float2 pp = pv[r * NSL];
          fx = pp.x >= thr_prev ? 1u : __float_as_uint(pp.x);
          fy = pp.y >= thr_prev ? 1u : __float_as_uint(pp.y);
        }
        __stcs(out + r * NSL, make_float2(__uint_as_float((__float_as_uint(z[r].x) & ~1u) | (fx & 1u)),
                                         __uint_as_float((__float_as_uint(z[r].y) & ~1u) | (fy & 1u))));
      }
    } else {
      // sphere mode: delta_R as it is, and the centres' bitmap, 8 consecutive pairs per store
      unsigned cnt = 0u;
#pragma unroll
      for (int r = 0; r < R1; ++r) {
        __stcs(out + r * NSL, z[r]);
        if (has_prev) {
          const float2 pp = pv[r * NSL];
          const unsigned bx = __ballot_sync(0xffffffffu, pp.x >= thr_prev);
          const unsigned by = __ballot_sync(0xffffffffu, pp.y >= thr_prev);
          cnt += __popc(bx) + __popc(by);
          if ((lane & 7) == 0) put_centres<N>(a.centres, row0 / M, j + r * NSL, bx >> lane, by >> lane);
        }
      }
      if (lane == 0 && cnt) atomicAdd(a.centre_count, cnt);
    }
    if (has_prev) {
      fence_async_smem();
      __syncwarp();
      if (lane == 0 && it + NP < my_count) issue_prev(it + NP);
    }
  }
  if (!ok) {
    // a wait ran out: record it; the copies in flight land (bounded waits) before the CTA leaves
    if (lane == 0) {
      atomicOr(a.err, ES_DEV_ERR_TIMEOUT);
      for (int q = it; q < it + 3 && q < my_count; ++q) mbar_wait(&bars[q & 1], (uint32_t)((q >> 1) & 1), a.wait_log2);
      if (has_prev)
        for (int q = it; q < it + NP && q < my_count; ++q)
          mbar_wait(&bars[2 + q % NP], (uint32_t)((q / NP) & 1), a.wait_log2);
    }
    __syncwarp();
  }
  if (EPI == EPI_IONIZE) {
    float total;
    const float2 acc2 = upk2(acc);
    if (grid_sum_as<TV, C::NW>(acc2.x + acc2.y, a.partials, a.counter, sred, &total) && threadIdx.x == 0) {
      const float mean = total / ((float)N * (float)N * (float)N);
      a.stats_out[0] = total;
      a.stats_out[1] = mean;
      a.stats_out[2] = a.normalize ? a.fc_mean / mean : 1.f;
    }
  }
}

// Row R2C pass in the same form: real rows -> half-spectrum rows (slot 0 holds (X[0], X[N/2])), with a scale
// or P(k) prologue.  The rows stay in one of the warp's NB buffers from their arrival to their stores: first
// stage out of it and back into it, last stage likewise in natural order, then the split by pairs (t, M - t)
// straight to global memory.  Arithmetic as row2_r2c, whose values pass through shared memory after the
// prologue: the scaling is kept out of the first butterfly's multiply-adds.
// 512^3: 235 -> 176 us, 1.07 GB at 0.90 of the copy rate, and so bound by DRAM.  256^3 keeps the older form:
// the pass alone takes 24 us against 27 us here, but a box 2746 us against 2736 and its products 160 against
// 156, with both neighbours overlapping the pass; at 128^3 there is nothing between them (911 us a box).
template <int N> struct RowWF {
  static constexpr bool ON = RowW<N>::NP > 0 && N >= 512;
  static constexpr int NB = 3;
  using C = RowWCfg<N>;
  static constexpr int TAB = (N / 4 + 1) + C::TW;        // split and last-stage twiddles
  static constexpr int BARS = (TAB * 8 + 15) / 16 * 16, BUFS = (BARS + C::NW * 32 + 127) / 128 * 128;
  static constexpr int bytes = BUFS + C::NW * NB * C::XBUF + 128;
};

template <int N, int PRO>
__global__ void __launch_bounds__(RowWCfg<N>::T) row_warp_r2c(const __grid_constant__ OpArgs a) {
  using C = RowWCfg<N>;
  using F = RowWF<N>;
  constexpr int M = C::M, RL = C::RL, RW = C::RW, R0 = C::R0, R1 = C::R1, NSL = C::NSL, NB = F::NB, PITCH = C::PITCH;
  constexpr bool HALF = C::HALF;
  constexpr int J0 = R1, V0 = HALF ? R0 / 2 : R0;
  static_assert(NB <= 4 && RW * (M / 2) % 32 == 0, "four mbarriers a warp; whole rounds of pairs");
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char* base = align_smem<128>(smem_raw);
  float2* wsp = reinterpret_cast<float2*>(base);         // w_N^t, t <= M/2
  float2* tws = wsp + M / 2 + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint64_t* bars = reinterpret_cast<uint64_t*>(base + F::BARS) + 4 * warp;
  unsigned char* bufs = base + F::BUFS + warp * NB * C::XBUF;

  constexpr int ntiles = N * N / RL;
  const int my_count = (int)blockIdx.x < ntiles ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  auto pair_at = [&](int it) { return ((blockIdx.x + it * gridDim.x) * RL + warp * RW) * M; };
  auto issue = [&](int it) {
    const uint64_t pol = l2_policy(a.hint_in);
    uint64_t* bar = &bars[it % NB];
    unsigned char* dst = bufs + (it % NB) * C::XBUF;
    const float2* src = a.rin + pair_at(it);
    mbar_expect_tx(bar, (uint32_t)(RW * M * 8) + stall_bytes(a.stall, it));
    if (PITCH == M) {
      bulk_load(dst, src, RW * M * 8, bar, pol);
    } else {
#pragma unroll
      for (int l = 0; l < RW; ++l) bulk_load(dst + l * PITCH * 8, src + l * M, M * 8, bar, pol);
    }
  };
  if (lane == 0) {
    for (int b = 0; b < NB; ++b) mbar_init(&bars[b], 1);
    fence_mbar_init();
    fence_async_smem();
  }
  for (int i = threadIdx.x; i <= M / 2; i += C::T) wsp[i] = a.tw[i];
  for (int i = threadIdx.x; i < C::TW; i += C::T) tws[i] = a.tw[(i % NSL) * (i / NSL + 1) * 2];
  pdl_wait();
  if (lane == 0)
    for (int it = 0; it < NB && it < my_count; ++it) issue(it);
  pdl_trigger();
  float sc = a.scale, sh = 0.f;
  if (PRO == PRO_PK) {
    const float ave = *a.ave;
    // g = (x / ave - 1) V / N^3  (delta_T.py:80-82), optionally times ave
    sc = a.pk_norm / ave;
    sh = -a.pk_norm;
    if (a.dimensional) { sc *= ave; sh *= ave; }
  }
  __syncthreads();

  const int l0 = HALF ? lane / (2 * J0) : lane / J0, j0 = HALF ? (lane >> 1) % J0 : lane % J0, h = HALF ? lane & 1 : 0;
  const int l = lane / NSL, j = lane % NSL;
  for (int it = 0; it < my_count; ++it) {
    float2* X = reinterpret_cast<float2*>(bufs + (it % NB) * C::XBUF);
    const uint32_t pair0 = pair_at(it);
    if (!__all_sync(0xffffffffu, mbar_wait(&bars[it % NB], (uint32_t)((it / NB) & 1), a.wait_log2))) {
      // a wait ran out: record it; the copies in flight land (bounded waits) before the warp leaves
      if (lane == 0) {
        atomicOr(a.err, ES_DEV_ERR_TIMEOUT);
        for (int q = it; q < it + NB && q < my_count; ++q) mbar_wait(&bars[q % NB], (uint32_t)((q / NB) & 1), a.wait_log2);
      }
      __syncwarp();
      break;
    }
    float2 v[V0];
    {
      const float2* x = X + l0 * PITCH + j0 + h * (M / R0);
#pragma unroll
      for (int k = 0; k < V0; ++k) {
        const float2 r = x[k * (HALF ? 2 : 1) * (M / R0)];
        v[k] = PRO == PRO_PK ? make_float2(fmaf(r.x, sc, sh), fmaf(r.y, sc, sh))
                             : make_float2(__fmul_rn(r.x, sc), __fmul_rn(r.y, sc));
      }
    }
    row_first_dft<C, false>(v, h);
    __syncwarp();                                        // every lane has read its rows
    {
      float2* x = X + l0 * PITCH + j0 * R0 + h * V0;
#pragma unroll
      for (int k = 0; k < V0; ++k) x[k ^ (HALF ? (j0 & 7) : j0)] = v[k];
    }
    __syncwarp();
    float2 z[R1];
    {
      const float2* x = X + l * PITCH;
#pragma unroll
      for (int r = 0; r < R1; ++r) z[r] = x[r * R0 + (j ^ r)];
    }
#pragma unroll
    for (int r = 1; r < R1; ++r) {
      const float2 w = tws[(r - 1) * NSL + j];
      z[r] = twid<false>(z[r], w.x, w.y);
    }
    Dft<R1, false>::run(z);
    __syncwarp();
#pragma unroll
    for (int r = 0; r < R1; ++r) X[l * PITCH + j + r * NSL] = z[r];
    __syncwarp();
    // X[m] = (Z[m] + conj Z[M-m]) / 2 - i w^m (Z[m] - conj Z[M-m]) / 2 by pairs (t, M - t); item 0 the packed
    // (X[0], X[N/2]) and the self-paired X[M/2]; w^(M-t) = -conj w^t
#pragma unroll 4
    for (int q = lane; q < RW * (M / 2); q += 32) {
      const int t = q % (M / 2), row = q / (M / 2);
      const float2* Z = X + row * PITCH;
      float2* out = a.cout + pair0 + row * M;
      if (t == 0) {
        const float2 z0 = Z[0];
        out[0] = make_float2(z0.x + z0.y, z0.x - z0.y);
        const float2 zh = Z[M / 2];
        const float2 th = cmul(wsp[M / 2], make_float2(0.f, zh.y + zh.y));
        out[M / 2] = make_float2(0.5f * (zh.x + zh.x + th.y), -0.5f * th.x);
      } else {
        const int m2 = M - t;
        const float2 zm = Z[t], zc = Z[m2], w = wsp[t];
        const float2 t1 = cmul(w, make_float2(zm.x - zc.x, zm.y + zc.y));
        out[t] = make_float2(0.5f * (zm.x + zc.x + t1.y), 0.5f * (zm.y - zc.y - t1.x));
        const float2 t2 = cmul(make_float2(-w.x, w.y), make_float2(zc.x - zm.x, zc.y + zm.y));
        out[m2] = make_float2(0.5f * (zc.x + zm.x + t2.y), 0.5f * (zc.y - zm.y - t2.x));
      }
    }
    fence_async_smem();
    __syncwarp();
    if (lane == 0 && it + NB < my_count) issue(it + NB);
  }
}

}  // namespace es
