// Packed candidate matrix M = F - E0 S from single-spin string pairs.
//
// F and S of a pair of determinants are sums and products of per-spin factors (det, f) that depend only
// on the pair's alpha strings and its beta strings (combine_fs in wick_math.cuh), and a candidate list
// repeats its strings: 12000 of the 125685 singles and doubles of 9 + 9 electrons in 28 orbitals over 3
// references hold some 2300 strings per spin, 5 10^6 string pairs against 72 10^6 candidate pairs.  So the
// factors of every ordered string pair are evaluated once, and an entry of M costs two 16-byte reads.
//
// Those 12000 candidates: 2.4 ms of kernels through the pair pipeline, 0.56 ms here (string pairs 0.21 ms,
// rows 0.33 ms: 576 MB written, bound by the shared-memory gathers), the whole call 4.6 -> 1.07 ms.
//
//   string_insert_kernel   strings of the candidates, found in a hash table per spin
//   string_base_kernel     ids grouped by (parent, rank), so a warp of string pairs shares one rank
//   string_ids_kernel
//   string_pairs_kernel    {pref det, pref f} of every ordered string pair of one spin
//   packed_rows_kernel     the packed rows of M
#include <cuda_runtime.h>

#include <algorithm>

#include "internal.cuh"
#include "sort.cuh"
#include "wick_math.cuh"

namespace nw {
namespace {

constexpr int kRanks = 5;                        // ranks 0..4 per spin
constexpr int kStringClasses = 256 * kRanks;     // (parent, rank), parents as in the 8-bit descriptor
constexpr uint32_t kEmpty = 0xFFFFFFFFu;
constexpr uint64_t kMaxStrings = 65535ull * 8;   // ids share a word with the parent (24 bits); grid rows
constexpr uint64_t kStringMin = 1024;            // fewer candidates: the pair pipeline's launches are as short
constexpr size_t kRowStage = 220ull << 10;       // table rows staged in shared memory up to here
constexpr size_t kKeepTable = 512ull << 20;      // string-pair tables up to here stay with the context

struct StringRec {
  uint64_t idx;      // hole bytes 0..3, particle bytes 4..7, zero beyond the rank
  uint32_t parent;
  uint32_t rank;
};

__device__ __forceinline__ StringRec string_of(const DetRec& d, int spin) {
  const int r = spin ? d.rb : d.ra;
  const uint64_t half = r >= 4 ? 0xFFFFFFFFull : (1ull << (8 * r)) - 1ull;
  StringRec s;
  s.idx = (spin ? d.ib : d.ia) & (half | (half << 32));
  s.parent = d.parent;
  s.rank = (uint32_t)r;
  return s;
}

__device__ __forceinline__ bool same_string(const StringRec& a, const StringRec& b) {
  return a.idx == b.idx && a.parent == b.parent && a.rank == b.rank;
}

// First candidate that shows each string of a spin: rep[spin * n + i].  Slots hold candidate positions; a
// table has at least 2 n slots, so a probe ends at an empty or an equal one.
__global__ void string_insert_kernel(const nw_det* __restrict__ dets, const uint32_t* __restrict__ cand, uint32_t n,
                                     uint32_t cap, uint32_t* __restrict__ table, uint32_t* __restrict__ rep,
                                     uint32_t* __restrict__ pos, uint32_t* __restrict__ counts) {
  const uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (t >= 2ull * n) return;
  const int spin = t >= n;
  const uint32_t i = (uint32_t)(t - (spin ? n : 0u));
  const StringRec s = string_of(load_det(dets, cand[i]), spin);
  uint64_t h = s.idx ^ ((uint64_t)(s.parent * kRanks + s.rank) << 40) * 0x9E3779B97F4A7C15ull;
  h = (h ^ (h >> 32)) * 0xD6E8FEB86659FD93ull;
  uint32_t slot = (uint32_t)(h >> 32) & (cap - 1u);
  uint32_t* tab = table + (uint64_t)spin * cap;
  for (uint32_t probe = 0; probe < cap; ++probe, slot = (slot + 1u) & (cap - 1u)) {
    const uint32_t j = atomicCAS(tab + slot, kEmpty, i);
    if (j == kEmpty) {
      rep[t] = i;
      pos[t] = atomicAdd(counts + spin * kStringClasses + s.parent * kRanks + s.rank, 1u);
      return;
    }
    if (same_string(s, string_of(load_det(dets, cand[j]), spin))) {
      rep[t] = j;
      return;
    }
  }
}

// Exclusive sums of the class counts of both spins; total[spin].  One block, a thread per run of classes.
__global__ void __launch_bounds__(256) string_base_kernel(uint32_t* __restrict__ counts, uint32_t* __restrict__ total) {
  constexpr int kPer = kStringClasses / 256;
  __shared__ uint32_t sum[256];
  for (int spin = 0; spin < 2; ++spin) {
    uint32_t* c = counts + spin * kStringClasses + threadIdx.x * kPer;
    uint32_t s = 0;
    for (int k = 0; k < kPer; ++k) s += c[k];
    sum[threadIdx.x] = s;
    __syncthreads();
    for (int d = 1; d < 256; d <<= 1) {
      const uint32_t y = threadIdx.x >= d ? sum[threadIdx.x - d] : 0u;
      __syncthreads();
      sum[threadIdx.x] += y;
      __syncthreads();
    }
    uint32_t run = sum[threadIdx.x] - s;
    for (int k = 0; k < kPer; ++k) {
      const uint32_t v = c[k];
      c[k] = run;
      run += v;
    }
    if (threadIdx.x == 255) total[spin] = sum[255];
    __syncthreads();
  }
}

// sid[i] = {alpha id, beta id | parent << 24}, the candidates' phases and the string records.
__global__ void string_ids_kernel(const nw_det* __restrict__ dets, const uint32_t* __restrict__ cand, uint32_t n,
                                  const uint32_t* __restrict__ rep, const uint32_t* __restrict__ pos,
                                  const uint32_t* __restrict__ base, uint2* __restrict__ sid,
                                  double* __restrict__ phase, StringRec* __restrict__ rec, uint32_t ua) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const DetRec d = load_det(dets, cand[i]);
  uint32_t id[2];
#pragma unroll
  for (int spin = 0; spin < 2; ++spin) {
    const StringRec s = string_of(d, spin);
    const uint32_t j = rep[(uint64_t)spin * n + i];
    id[spin] = base[spin * kStringClasses + s.parent * kRanks + s.rank] + pos[(uint64_t)spin * n + j];
    if (j == i) rec[(spin ? ua : 0u) + id[spin]] = s;
  }
  sid[i] = make_uint2(id[0], id[1] | (d.parent << 24));
  phase[i] = d.phase;
}

// ---------------------------------------------------------------------------------------
// Factors of one string pair.
// ---------------------------------------------------------------------------------------
template <int L>
__device__ __forceinline__ void fast_factor(const FockSpinTab& t, int n, int nocc, int rx, uint64_t ix, uint64_t iw,
                                            double* det, double* f) {
  int r[L > 0 ? L : 1], c[L > 0 ? L : 1];
  det_labels_ct<L>(rx, ix, iw, nocc, n, r, c);
  spin_f_ct<L>(t.recx, t.recy, t.f0f[0], n, r, c, det, f);
}

template <int L>
__device__ __noinline__ void gen_factor(const GenSpin& g, const FockSpinTab& t, int n, int nocc, int rx, uint64_t ix,
                                        uint64_t iw, double tol, bool exact, double* det, double* f) {
  int r[L > 0 ? L : 1], c[L > 0 ? L : 1];
  det_labels_ct<L>(rx, ix, iw, nocc, n, r, c);
  double d0[Sq<L>::v], d1[Sq<L>::v];
  build_d_ct<L>(d0, g.x[0], g.y[0], n, r, c);
  build_d_ct<L>(d1, g.x[1], g.y[1], n, r, c);
  *det = overlap_spin_ct<L>(g.m, d0, d1);
  *f = spin_f_gen_ct<L>(g.m, t.ff_t, t.f0f, n, r, c, d0, d1, tol, exact);
}

__device__ __forceinline__ int labels_any(int rx, uint64_t ix, int rw, uint64_t iw, int nocc, int n, int* rows,
                                          int* cols) {
  uint8_t bx[8], bw[8];
  for (int k = 0; k < 8; ++k) {
    bx[k] = (uint8_t)ibyte(ix, k);
    bw[k] = (uint8_t)ibyte(iw, k);
  }
  return det_labels(rx, bx, rw, bw, nocc, n, rows, cols);
}

__device__ __noinline__ void fast_factor_rt(const FockSpinTab& t, int n, int nocc, int rx, uint64_t ix, int rw,
                                            uint64_t iw, double* det, double* f) {
  int r[kML], c[kML];
  const int L = labels_any(rx, ix, rw, iw, nocc, n, r, c);
  spin_f_rt(L, t.recx, t.recy, t.f0f[0], n, r, c, det, f);
}

__device__ __noinline__ void gen_factor_rt(const GenSpin& g, const FockSpinTab& t, int n, int nocc, int rx, uint64_t ix,
                                           int rw, uint64_t iw, double tol, bool exact, double* det, double* f) {
  int r[kML], c[kML];
  const int L = labels_any(rx, ix, rw, iw, nocc, n, r, c);
  double d0[kML * kML], d1[kML * kML];
  build_d_rt(d0, g.x[0], g.y[0], n, L, r, c);
  build_d_rt(d1, g.x[1], g.y[1], n, L, r, c);
  *det = overlap_spin_hd(g.m, L, d0, d1);
  *f = spin_f_gen_hd(g.m, t.ff_t, t.f0f, n, L, r, c, d0, d1, tol, exact);
}

// tab[i * u + j] = {pref det, pref f} of bra string i and ket string j of one spin (GEN: the string pairs
// of reference pairs with zero-overlap orbitals, else the others), and the excitation distance of strings
// of one parent.  A thread keeps its ket string for kRowsPer bra strings; a warp shares the bra string.
constexpr int kPairThreads = 128;
constexpr int kRowsPer = 8;

template <bool GEN>
__global__ void __launch_bounds__(kPairThreads, GEN ? 1 : 4)
    string_pairs_kernel(EvalParams P, int spin, const StringRec* __restrict__ rec, uint32_t u, double2* __restrict__ tab,
                        uint8_t* __restrict__ dist) {
  const uint32_t j = blockIdx.x * kPairThreads + threadIdx.x;
  if (j >= u) return;
  const StringRec w = rec[j];
  const int nocc = spin ? P.nocc_b : P.nocc_a;
  const uint32_t i1 = min(u, (blockIdx.y + 1u) * kRowsPer);
  for (uint32_t i = blockIdx.y * kRowsPer; i < i1; ++i) {
    const StringRec x = rec[i];
    const int p = (int)(x.parent * P.nref + w.parent);
    if ((P.order[p] >= P.nfast) != GEN) continue;
    const int L = (int)(x.rank + w.rank);
    double det, f, pref;
    if (GEN) {
      const GenSpin& g = spin ? P.gen[p].b : P.gen[p].a;
      const FockSpinTab& t = spin ? P.fock[p].b : P.fock[p].a;
      const bool exact = P.exact != 0;
      pref = g.pref;
      switch (L) {
        case 0:
          gen_factor<0>(g, t, P.n, nocc, x.rank, x.idx, w.idx, P.tol, exact, &det, &f);
          break;
        case 1:
          gen_factor<1>(g, t, P.n, nocc, x.rank, x.idx, w.idx, P.tol, exact, &det, &f);
          break;
        case 2:
          gen_factor<2>(g, t, P.n, nocc, x.rank, x.idx, w.idx, P.tol, exact, &det, &f);
          break;
        case 3:
          gen_factor<3>(g, t, P.n, nocc, x.rank, x.idx, w.idx, P.tol, exact, &det, &f);
          break;
        case 4:
          gen_factor<4>(g, t, P.n, nocc, x.rank, x.idx, w.idx, P.tol, exact, &det, &f);
          break;
        default:
          gen_factor_rt(g, t, P.n, nocc, x.rank, x.idx, w.rank, w.idx, P.tol, exact, &det, &f);
          break;
      }
    } else {
      const FockSpinTab& t = spin ? P.fock[p].b : P.fock[p].a;
      pref = spin ? P.fast[p].b.pref : P.fast[p].a.pref;
      switch (L) {
        case 0:
          fast_factor<0>(t, P.n, nocc, x.rank, x.idx, w.idx, &det, &f);
          break;
        case 1:
          fast_factor<1>(t, P.n, nocc, x.rank, x.idx, w.idx, &det, &f);
          break;
        case 2:
          fast_factor<2>(t, P.n, nocc, x.rank, x.idx, w.idx, &det, &f);
          break;
        case 3:
          fast_factor<3>(t, P.n, nocc, x.rank, x.idx, w.idx, &det, &f);
          break;
        case 4:
          fast_factor<4>(t, P.n, nocc, x.rank, x.idx, w.idx, &det, &f);
          break;
        default:
          fast_factor_rt(t, P.n, nocc, x.rank, x.idx, w.rank, w.idx, &det, &f);
          break;
      }
      if (x.parent == w.parent)
        dist[(uint64_t)i * u + j] = (uint8_t)(sym_diff(x.idx, (int)x.rank, w.idx, (int)w.rank, 0) +
                                              sym_diff(x.idx, (int)x.rank, w.idx, (int)w.rank, 4));
    }
    tab[(uint64_t)i * u + j] = make_double2(pref * det, pref * f);
  }
}

// Packed rows of M: row a holds M[a][a..n).  With STAGE the two table rows of candidate a are copied to
// shared memory first (16 (ua + ub) bytes): a random 16-byte read costs some 8 shared-memory cycles per
// warp there against 32 tag lookups in L1.  Rows are handed out longest first.
constexpr int kRowThreads = 512;

template <bool STAGE>
__global__ void __launch_bounds__(kRowThreads) packed_rows_kernel(const uint2* __restrict__ sid,
                                                                  const double* __restrict__ phase, uint32_t n,
                                                                  const double2* __restrict__ ta,
                                                                  const double2* __restrict__ tb,
                                                                  const uint8_t* __restrict__ da,
                                                                  const uint8_t* __restrict__ db, uint32_t ua,
                                                                  uint32_t ub, double e0, double* __restrict__ m,
                                                                  uint32_t* __restrict__ work) {
  extern __shared__ double2 rows[];
  __shared__ uint32_t next;
  for (;;) {
    if (threadIdx.x == 0) next = atomicAdd(work, 1u);
    __syncthreads();
    const uint32_t a = next;
    if (a >= n) break;
    const uint2 sa = sid[a];
    const uint32_t pa = sa.y >> 24, ib = sa.y & 0xFFFFFFu;
    const double2* ra = ta + (uint64_t)sa.x * ua;
    const double2* rb = tb + (uint64_t)ib * ub;
    if (STAGE) {
      for (uint32_t k = threadIdx.x; k < ua; k += kRowThreads) rows[k] = __ldg(ra + k);
      for (uint32_t k = threadIdx.x; k < ub; k += kRowThreads) rows[ua + k] = __ldg(rb + k);
      ra = rows;
      rb = rows + ua;
    }
    __syncthreads();
    const uint8_t* xa = da + (uint64_t)sa.x * ua;
    const uint8_t* xb = db + (uint64_t)ib * ub;
    const double ph_a = phase[a];
    double* row = m + ((uint64_t)a * (2ull * n - a + 1) / 2 - a);
    for (uint32_t b = a + threadIdx.x; b < n; b += kRowThreads) {
      const uint2 sb = __ldg(sid + b);
      const uint32_t jb = sb.y & 0xFFFFFFu;
      double v = 0.0;
      // determinants of one parent more than a double excitation apart: exact zeros
      if ((sb.y >> 24) != pa || (int)__ldg(xa + sb.x) + (int)__ldg(xb + jb) <= 4) {
        const double2 fa = STAGE ? ra[sb.x] : __ldg(ra + sb.x), fb = STAGE ? rb[jb] : __ldg(rb + jb);
        const double ph = ph_a * __ldg(phase + b);
        // combine_fs with the prefactors already in the factors
        double f = 0.0;
        if (fb.x != 0.0) f += fa.y * fb.x;
        if (fa.x != 0.0) f += fb.y * fa.x;
        v = ph * f - e0 * (ph * fa.x * fb.x);
      }
      row[b] = v;
    }
    __syncthreads();
  }
}

template <bool STAGE>
cudaError_t launch_rows(size_t shared, uint2* sid, double* phase, uint32_t n, double2* ta, double2* tb, uint8_t* da,
                        uint8_t* db, uint32_t ua, uint32_t ub, double e0, double* m, uint32_t* work) {
  auto k = packed_rows_kernel<STAGE>;
  cudaError_t e = cudaSuccess;
  if (STAGE) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared);
  int per_sm = 1;
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kRowThreads, shared);
  if (e != cudaSuccess) return e;
  k<<<148 * std::max(per_sm, 1), kRowThreads, shared>>>(sid, phase, n, ta, tb, da, db, ua, ub, e0, m, work);
  return cudaGetLastError();
}

inline size_t align256(size_t b) { return (b + 255) / 256 * 256; }

}  // namespace

nw_status fill_candidate_m(nw_ctx* ctx, const uint32_t* dcand, uint64_t n, double e0, double* m, bool* done) {
  *done = false;
  if (n < kStringMin || n >= (1ull << 28)) return NW_OK;
  const EvalParams P = make_params(ctx);
  uint32_t cap = 1u << 12;
  while (cap < 2 * n) cap <<= 1;
  // scratch: hash tables, representatives, positions, class counts, totals and the row counter, ids,
  // phases, string records
  const size_t o_rep = align256(8ull * cap), o_pos = o_rep + align256(8 * n), o_cnt = o_pos + align256(8 * n);
  const size_t o_tot = o_cnt + align256(8ull * kStringClasses), o_sid = o_tot + 256, o_ph = o_sid + align256(8 * n);
  const size_t o_rec = o_ph + align256(8 * n), bytes = o_rec + 2 * n * sizeof(StringRec);
  nw_status st = ensure(ctx, ctx->pt2_scratch, bytes);
  if (st != NW_OK) return st;
  char* s = static_cast<char*>(ctx->pt2_scratch.p);
  uint32_t* table = reinterpret_cast<uint32_t*>(s);
  uint32_t* rep = reinterpret_cast<uint32_t*>(s + o_rep);
  uint32_t* pos = reinterpret_cast<uint32_t*>(s + o_pos);
  uint32_t* counts = reinterpret_cast<uint32_t*>(s + o_cnt);
  uint32_t* total = reinterpret_cast<uint32_t*>(s + o_tot);
  uint2* sid = reinterpret_cast<uint2*>(s + o_sid);
  double* phase = reinterpret_cast<double*>(s + o_ph);
  StringRec* rec = reinterpret_cast<StringRec*>(s + o_rec);
  NW_CUDA(ctx, cudaMemsetAsync(table, 0xFF, 8ull * cap, nullptr));
  NW_CUDA(ctx, cudaMemsetAsync(counts, 0, o_sid - o_cnt, nullptr));
  const uint32_t nn = (uint32_t)n;
  string_insert_kernel<<<(unsigned)((2 * n + 255) / 256), 256>>>(P.dets, dcand, nn, cap, table, rep, pos, counts);
  string_base_kernel<<<1, 256>>>(counts, total);
  NW_CUDA(ctx, cudaGetLastError());
  uint32_t u[2] = {0, 0};
  NW_CUDA(ctx, cudaMemcpy(u, total, sizeof(u), cudaMemcpyDeviceToHost));
  const uint64_t ua = u[0], ub = u[1], sq = ua * ua + ub * ub;
  // worth it (and at most half of M's bytes) from four candidate pairs a string pair
  if (ua >= kMaxStrings || ub >= kMaxStrings || sq > n * (n + 1) / 8) return NW_OK;
  const size_t o_tb = align256(16 * ua * ua), o_da = o_tb + align256(16 * ub * ub);
  const size_t o_db = o_da + align256(ua * ua), tab_bytes = o_db + ub * ub;
  if (ctx->pt2_table.bytes < tab_bytes) {
    if (ctx->pt2_table.p) cudaFree(ctx->pt2_table.p);
    ctx->pt2_table = DevBuf{};
    if (ctx_malloc(ctx, &ctx->pt2_table.p, tab_bytes) != cudaSuccess) {
      cudaGetLastError();
      ctx->pt2_table.p = nullptr;
      return NW_OK;   // no room: the pair pipeline builds M
    }
    ctx->pt2_table.bytes = tab_bytes;
  }
  char* t = static_cast<char*>(ctx->pt2_table.p);
  double2* tab[2] = {reinterpret_cast<double2*>(t), reinterpret_cast<double2*>(t + o_tb)};
  uint8_t* dist[2] = {reinterpret_cast<uint8_t*>(t + o_da), reinterpret_cast<uint8_t*>(t + o_db)};
  string_ids_kernel<<<(unsigned)((n + 255) / 256), 256>>>(P.dets, dcand, nn, rep, pos, counts, sid, phase, rec, u[0]);
  for (int spin = 0; spin < 2; ++spin) {
    const uint32_t us = u[spin];
    const StringRec* rs = rec + (spin ? ua : 0);
    const dim3 grid((us + kPairThreads - 1) / kPairThreads, (us + kRowsPer - 1) / kRowsPer);
    string_pairs_kernel<false><<<grid, kPairThreads>>>(P, spin, rs, us, tab[spin], dist[spin]);
    if (ctx->nfast < ctx->nresident)
      string_pairs_kernel<true><<<grid, kPairThreads>>>(P, spin, rs, us, tab[spin], dist[spin]);
  }
  NW_CUDA(ctx, cudaGetLastError());
  const size_t shared = 16 * (ua + ub);
  const cudaError_t e = shared <= kRowStage
                            ? launch_rows<true>(shared, sid, phase, nn, tab[0], tab[1], dist[0], dist[1], u[0], u[1], e0,
                                                m, total + 2)
                            : launch_rows<false>(0, sid, phase, nn, tab[0], tab[1], dist[0], dist[1], u[0], u[1], e0, m,
                                                 total + 2);
  NW_CUDA(ctx, e);
  if (ctx->pt2_table.bytes > kKeepTable) {
    cudaFree(ctx->pt2_table.p);   // waits for the kernels
    ctx->pt2_table = DevBuf{};
  }
  *done = true;
  return NW_OK;
}

}  // namespace nw
