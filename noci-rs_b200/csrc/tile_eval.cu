// One-kernel pair evaluation: each block takes a tile of consecutive pairs, groups them by rank class
// in shared memory and evaluates them, one class per warp at a time.
//
// The sorted pipeline (eval.cu) orders a whole request by (class, ket reference, bra) through global
// memory: five passes over 4-byte keys, ranks and indices and twelve dependent launches, so that the
// n^4 tables are read with locality.  Two kinds of request do not need that order:
//  * (F, S): the tables of one reference pair are four n^2 record arrays (100 KB at n = 40), L1 / L2
//    resident however the pairs come.  4 10^6 pairs at n = 28 (9 + 9 electrons, 3 references): 276 us
//    sorted, 207 us here (L1 gathers at 76 % of the L1TEX limit, hit rate 45 %, 24 warps per SM; 1000 pairs
//    31 -> 8.3 us); n = 40, 6 + 6 electrons, ranks 0-4: 158 us.  Reading the factors of single-single string
//    pairs from a table of all of them instead of the records was slower (252 us).
//  * small (H, S) requests: the chain of launches is longer than the work (512 pairs at n = 30: 37.7 ->
//    10.3 us).
// A tile of 1024 pairs holds some ten classes, so whole-warp padding costs about a sixth of the lanes.
#include <cuda_runtime.h>

#include <algorithm>

#include "internal.cuh"
#include "sort.cuh"
#include "wick_math.cuh"

namespace nw {
namespace {

constexpr int kTileThreads = 256;
constexpr int kTileItems = 4;                               // pairs per thread
constexpr int kTilePairs = kTileThreads * kTileItems;       // largest tile
constexpr int kSkipClass = 255;

// Classes of a tile: the 26 of the m = 0 evaluators, then (GEN) the same ranks of reference pairs with
// zero-overlap orbitals.
template <bool GEN>
constexpr int tile_classes() {
  return GEN ? 2 * kClasses : kClasses;
}

template <bool GEN>
__device__ __forceinline__ int tile_classify(const EvalParams& P, uint2 ab, uint64_t i, double* __restrict__ out,
                                             uint32_t* __restrict__ flag) {
  if (ab.x >= P.ndet || ab.y >= P.ndet) {
    atomicOr(flag, 1u);
    const double nan = __longlong_as_double(0x7FF8000000000000ll);
    store_hs(out, i, nan, nan);
    return kSkipClass;
  }
  const uint32_t dx = __ldg(P.desc + ab.x), dw = __ldg(P.desc + ab.y);
  const int px = (int)(dx & 0xFF), pw = (int)(dw & 0xFF);
  if (px == pw && far_same_parent(load_det(P.dets, ab.x), load_det(P.dets, ab.y))) {
    store_hs(out, i, 0.0, 0.0);
    return kSkipClass;
  }
  const int la = (int)((dx >> 8) & 15) + (int)((dw >> 8) & 15), lb = (int)(dx >> 12) + (int)(dw >> 12);
  const int ord = __ldg(P.order + px * P.nref + pw);
  if (ord < 0) return kSkipClass;  // reference pair outside the resident block: left unwritten
  const int c = rank_class(la, lb);
  if (GEN && ord >= P.nfast) return kClasses + c;
  return c;
}

// Groups the block's tile [base, base + count) by class and calls eval(class, request index, pair)
// for every pair to evaluate; the lanes of a warp always hold one class.  Chunks of 32 slots go to the
// warps from the last class down, so the ranks with the most work start first.
template <bool GEN, typename F>
__device__ __forceinline__ void tile_run(const EvalParams& P, const uint2* __restrict__ pairs, uint64_t base, int count,
                                         double* __restrict__ out, uint32_t* __restrict__ flag, F&& eval) {
  constexpr int NC = tile_classes<GEN>();
  constexpr int kSlots = kTilePairs + 32 * NC;
  __shared__ uint2 s_ab[kTilePairs];
  __shared__ uint16_t s_slot[kSlots];
  __shared__ uint32_t s_cnt[NC], s_first[NC + 1], s_next;
  const int tid = threadIdx.x, lane = tid & 31;
  for (int c = tid; c < NC; c += kTileThreads) s_cnt[c] = 0u;
  for (int k = tid; k < kSlots; k += kTileThreads) s_slot[k] = 0xFFFFu;
  if (tid == 0) s_next = 0u;
  __syncthreads();
  int cls[kTileItems], rk[kTileItems];
#pragma unroll
  for (int u = 0; u < kTileItems; ++u) {
    const int k = tid + u * kTileThreads;
    cls[u] = kSkipClass;
    if (k < count) {
      const uint2 ab = __ldg(pairs + base + k);
      s_ab[k] = ab;
      cls[u] = tile_classify<GEN>(P, ab, base + k, out, flag);
    }
  }
#pragma unroll
  for (int u = 0; u < kTileItems; ++u) {
    const uint32_t peers = __match_any_sync(0xFFFFFFFFu, cls[u]);
    const int leader = __ffs(peers) - 1;
    uint32_t first = 0u;
    if (lane == leader && cls[u] != kSkipClass) first = atomicAdd(&s_cnt[cls[u]], (uint32_t)__popc(peers));
    rk[u] = (int)(__shfl_sync(0xFFFFFFFFu, first, leader) + (uint32_t)__popc(peers & ((1u << lane) - 1u)));
  }
  __syncthreads();
  if (tid < 32) {
    // first slot of every class, each class padded to whole warps
    uint32_t carry = 0u;
#pragma unroll
    for (int c0 = 0; c0 < NC; c0 += 32) {
      const int c = c0 + lane;
      const uint32_t v = c < NC ? (s_cnt[c] + 31u) & ~31u : 0u;
      uint32_t x = v;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, d);
        if (lane >= d) x += y;
      }
      if (c < NC) s_first[c] = carry + x - v;
      carry += __shfl_sync(0xFFFFFFFFu, x, 31);
    }
    if (lane == 0) s_first[NC] = carry;
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kTileItems; ++u)
    if (cls[u] != kSkipClass) s_slot[s_first[cls[u]] + rk[u]] = (uint16_t)(tid + u * kTileThreads);
  __syncthreads();
  const uint32_t nchunk = s_first[NC] / 32u;
  for (;;) {
    uint32_t q = 0u;
    if (lane == 0) q = atomicAdd(&s_next, 1u);
    q = __shfl_sync(0xFFFFFFFFu, q, 0);
    if (q >= nchunk) break;
    const uint32_t slot0 = (nchunk - 1u - q) * 32u;
    // the chunk's class: the last one whose first slot is not beyond it (empty classes share the first
    // slot of their successor)
    int c = -1;
#pragma unroll
    for (int c0 = 0; c0 < NC; c0 += 32)
      c += __popc(__ballot_sync(0xFFFFFFFFu, c0 + lane < NC && s_first[min(c0 + lane, NC)] <= slot0));
    const uint32_t k = s_slot[slot0 + lane];
    if (k != 0xFFFFu) {
      const uint2 ab = s_ab[k];
      eval(c, base + k, ab);
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------------------
// (F, S).
// ---------------------------------------------------------------------------------------
template <int L>
__device__ __forceinline__ void spin_f_at(const double2* __restrict__ rec, double f0, int n, int nocc, int rx, uint64_t ix,
                                          uint64_t iw, double* det, double* f) {
  int r[L > 0 ? L : 1], c[L > 0 ? L : 1];
  det_labels_ct<L>(rx, ix, iw, nocc, n, r, c);
  spin_f_ct<L>(rec, rec + n * n, f0, n, r, c, det, f);
}

// One spin of an m = 0 pair; L is uniform over the warp.
__device__ __forceinline__ void spin_f_of(int L, const double2* __restrict__ rec, double f0, int n, int nocc, int rx,
                                          uint64_t ix, uint64_t iw, double* det, double* f) {
  switch (L) {
    case 0:
      spin_f_at<0>(rec, f0, n, nocc, rx, ix, iw, det, f);
      break;
    case 1:
      spin_f_at<1>(rec, f0, n, nocc, rx, ix, iw, det, f);
      break;
    case 2:
      spin_f_at<2>(rec, f0, n, nocc, rx, ix, iw, det, f);
      break;
    case 3:
      spin_f_at<3>(rec, f0, n, nocc, rx, ix, iw, det, f);
      break;
    default:
      spin_f_at<4>(rec, f0, n, nocc, rx, ix, iw, det, f);
      break;
  }
}

// The rare paths are calls that take everything by value and load the records themselves: a reference to a
// record or to the kernel's parameters would keep them in local memory on the common path too (4 10^6 (F, S)
// pairs: 235 us with references, 207 us without).
__device__ __noinline__ double2 fs_rt_one(const EvalParams* P, uint2 ab) {
  const DetRec x = load_det(P->dets, ab.x), w = load_det(P->dets, ab.y);
  const int p = (int)x.parent * P->nref + (int)w.parent;
  double2 r;
  eval_fs_m0_rt(P->fast[p], P->fock[p], x, w, P->n, P->nocc_a, P->nocc_b, &r.x, &r.y);
  return r;
}

__device__ __noinline__ double2 fs_gen_one(const EvalParams* P, uint2 ab) {
  const DetRec x = load_det(P->dets, ab.x), w = load_det(P->dets, ab.y);
  const int p = (int)x.parent * P->nref + (int)w.parent;
  double2 r;
  eval_fs_gen_any(P->gen[p], P->fock[p], x, w, P->n, P->nocc_a, P->nocc_b, P->tol, P->exact != 0, &r.x, &r.y);
  return r;
}

__device__ __forceinline__ void fs_fast(const EvalParams& P, int c, uint2 ab, double* f, double* s) {
  const DetRec x = load_det(P.dets, ab.x), w = load_det(P.dets, ab.y);
  const int p = (int)x.parent * P.nref + (int)w.parent;
  // the slab of the Fock records is regular: recx, recy of alpha, then of beta, per ordered pair
  const int la = c / 5, lb = c - 5 * la, n2 = P.n * P.n;
  const double* rec = P.fslab + (size_t)p * (8 * n2);
  const FsScalars* sc = reinterpret_cast<const FsScalars*>(P.fslab + (size_t)P.nref * P.nref * (8 * n2)) + p;
  double f0a, f0b, pa, pb;
  asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(f0a), "=d"(f0b), "=d"(pa), "=d"(pb) : "l"(sc));
  double deta, fa, detb, fb;
  spin_f_of(la, reinterpret_cast<const double2*>(rec), f0a, P.n, P.nocc_a, x.ra, x.ia, w.ia, &deta, &fa);
  spin_f_of(lb, reinterpret_cast<const double2*>(rec) + 2 * n2, f0b, P.n, P.nocc_b, x.rb, x.ib, w.ib, &detb, &fb);
  combine_fs(x.phase * w.phase, pa, deta, fa, pb, detb, fb, f, s);
}

template <bool GEN, int MINB>
__global__ void __launch_bounds__(kTileThreads, MINB) fs_tile_kernel(const __grid_constant__ EvalParams P, const uint2* __restrict__ pairs,
                                                                     uint64_t npairs, int tile,
                                                                     double* __restrict__ out,
                                                                     uint32_t* __restrict__ flag) {
  const uint64_t base = (uint64_t)blockIdx.x * (uint64_t)tile;
  const int count = (int)min((uint64_t)tile, npairs - base);
  tile_run<GEN>(P, pairs, base, count, out, flag, [&](int c, uint64_t i, uint2 ab) {
    double2 r;
    if (GEN && c >= kClasses)
      r = fs_gen_one(&P, ab);
    else if (c == kClasses - 1)
      r = fs_rt_one(&P, ab);
    else
      fs_fast(P, c, ab, &r.x, &r.y);
    store_hs(out, i, r.x, r.y);
  });
}

// ---------------------------------------------------------------------------------------
// (H, S) of small requests.
// ---------------------------------------------------------------------------------------
__device__ __noinline__ double2 hs_rt_one(const EvalParams* P, uint2 ab) {
  const DetRec x = load_det(P->dets, ab.x), w = load_det(P->dets, ab.y);
  double2 r;
  eval_m0_rt(P->fast[(int)x.parent * P->nref + (int)w.parent], x, w, P->n, P->nocc_a, P->nocc_b, P->enuc, &r.x, &r.y);
  return r;
}

__device__ __noinline__ double2 hs_gen_one(const EvalParams* P, uint2 ab) {
  const DetRec x = load_det(P->dets, ab.x), w = load_det(P->dets, ab.y);
  double2 r;
  eval_gen_any(P->gen[(int)x.parent * P->nref + (int)w.parent], x, w, P->n, P->nocc_a, P->nocc_b, P->enuc, P->tol,
               P->exact != 0, &r.x, &r.y);
  return r;
}

#define NW_HS_TILE_CASE(A, B)                                                       \
  case (A) * 5 + (B):                                                               \
    eval_m0_ct<A, B>(P.fast[p], x, w, P.n, P.nocc_a, P.nocc_b, P.enuc, &h, &s);     \
    break;

template <bool GEN>
__global__ void __launch_bounds__(kTileThreads, 1) hs_tile_kernel(const __grid_constant__ EvalParams P, const uint2* __restrict__ pairs,
                                                               uint64_t npairs, int tile, double* __restrict__ out,
                                                               uint32_t* __restrict__ flag) {
  const uint64_t base = (uint64_t)blockIdx.x * (uint64_t)tile;
  const int count = (int)min((uint64_t)tile, npairs - base);
  tile_run<GEN>(P, pairs, base, count, out, flag, [&](int c, uint64_t i, uint2 ab) {
    if (GEN && c >= kClasses) {
      const double2 r = hs_gen_one(&P, ab);
      store_hs(out, i, r.x, r.y);
      return;
    }
    if (c == kClasses - 1) {
      const double2 r = hs_rt_one(&P, ab);
      store_hs(out, i, r.x, r.y);
      return;
    }
    const DetRec x = load_det(P.dets, ab.x), w = load_det(P.dets, ab.y);
    const int p = (int)x.parent * P.nref + (int)w.parent;
    double h = 0.0, s = 0.0;
    switch (c) {
      NW_HS_TILE_CASE(0, 0) NW_HS_TILE_CASE(0, 1) NW_HS_TILE_CASE(0, 2) NW_HS_TILE_CASE(0, 3) NW_HS_TILE_CASE(0, 4)
      NW_HS_TILE_CASE(1, 0) NW_HS_TILE_CASE(1, 1) NW_HS_TILE_CASE(1, 2) NW_HS_TILE_CASE(1, 3) NW_HS_TILE_CASE(1, 4)
      NW_HS_TILE_CASE(2, 0) NW_HS_TILE_CASE(2, 1) NW_HS_TILE_CASE(2, 2) NW_HS_TILE_CASE(2, 3) NW_HS_TILE_CASE(2, 4)
      NW_HS_TILE_CASE(3, 0) NW_HS_TILE_CASE(3, 1) NW_HS_TILE_CASE(3, 2) NW_HS_TILE_CASE(3, 3) NW_HS_TILE_CASE(3, 4)
      NW_HS_TILE_CASE(4, 0) NW_HS_TILE_CASE(4, 1) NW_HS_TILE_CASE(4, 2) NW_HS_TILE_CASE(4, 3) NW_HS_TILE_CASE(4, 4)
    }
    store_hs(out, i, h, s);
  });
}
#undef NW_HS_TILE_CASE

}  // namespace

uint64_t tile_limit(const EvalParams& P, EvalMode mode, bool gen) {
  if (mode == EvalMode::kFS) return gen ? kTileSmall : ~0ull;
  const uint64_t reach = (uint64_t)P.span * P.span * P.n * P.n * P.n;
  if (gen || P.n > kTileLargeOrbitals || reach > kTileLargeReach) return kTileSmall;
  return P.span <= 3 ? kTileLarge : kTileTwoWaves;
}

cudaError_t eval_tiles(const EvalParams& P, const uint2* pairs, uint64_t npairs, double* out, EvalMode mode, bool gen,
                       uint32_t* flag, cudaStream_t stream) {
  // the tile of a small request: as many blocks as SMs before the tiles grow
  const uint64_t per = (npairs + 147) / 148;
  const int tile = (int)std::min<uint64_t>(kTilePairs, std::max<uint64_t>(32, (per + 31) / 32 * 32));
  const unsigned blocks = (unsigned)((npairs + tile - 1) / tile);
  if (mode == EvalMode::kFS) {
    if (gen)
      fs_tile_kernel<true, 1><<<blocks, kTileThreads, 0, stream>>>(P, pairs, npairs, tile, out, flag);
    else
      fs_tile_kernel<false, 3><<<blocks, kTileThreads, 0, stream>>>(P, pairs, npairs, tile, out, flag);
  } else if (gen) {
    hs_tile_kernel<true><<<blocks, kTileThreads, 0, stream>>>(P, pairs, npairs, tile, out, flag);
  } else {
    hs_tile_kernel<false><<<blocks, kTileThreads, 0, stream>>>(P, pairs, npairs, tile, out, flag);
  }
  return cudaGetLastError();
}

}  // namespace nw
