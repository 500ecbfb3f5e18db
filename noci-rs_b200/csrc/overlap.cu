// Spin-factorised overlap action y += S x over the resident basis (nw_apply_overlap_device and
// the direct-overlap NOCI-QMC propagator).
//
// The overlap of two determinants is the product of their alpha and beta single-spin overlaps,
// and the determinants of one parent reference share single-spin components (every determinant
// with the same alpha excitation has the same alpha string).  For a target parent Q and a source
// parent P != Q
//     S_{w Omega} = r_w r_Omega A^{QP}[a_w][a_Omega] B^{QP}[b_w][b_Omega],
// A^{QP}[i][j] = det(C_Q[:, occ(i)]^T S_AO C_P[:, occ(j)]) over the ascending occupied columns of
// the two alpha strings (B the same for beta), r = the record's phase times the canonical
// excitation phase of its holes and particles (1 for canonically phased records), so S x is two
// contractions per ordered parent pair (apply_overlap_sparse, src/noci/factorise/overlap.rs:434-498,
// 1276-1360).  With X the sources of P as a matrix over (a, b), the sources are split X = X1 + X2:
//   stage 1  U[a][bbar] = sum_b X1[a][b] B^{QP}[bbar][b]   for the rows R of X1 (b first)
//            W[abar][b] = sum_a A^{QP}[abar][a] X2[a][b]   for the columns C of X2 (a first)
//   stage 2  y_w += r_w sum_P { sum_{a in R} A[a_w][a] U[a][b_w] + sum_{b in C} W[a_w][b] B[b_w][b] }
// A source goes to X1 when its row is at least as long as its column, so that R and C are the few long
// rows and columns that cover the sources: for a singles-and-doubles space R is the parent's own alpha
// string and its singles and C the parent's own beta string, 146 terms a target instead of the 3925
// alpha strings (n = 40, 4 + 4 electrons), and U and W are 30 MB instead of 740.  All sources by rows
// or all by columns is taken where that costs less.  Determinants of one parent are orthonormal, so the
// same-parent block adds the sources with the same (a, b) pair (the determinant itself in a basis
// without duplicates).
//
// Layout: A^{QP} and B^{QP} are stored source-major (row a or b, contiguous over the target's strings,
// rows padded to an even length), so both stage-1 products read table rows coalesced.  Rows of X1
// (columns of X2) with mostly the same entries form dense tiles of kOvlTile rows whose sources are
// staged in shared memory: one 16-byte load of a table row feeds 2 kOvlTile multiply-adds.  The
// other rows go one by one in chunks of at most kOvlChunk sources, chunks of a long row adding into it
// atomically.  Stage 2 is one thread per (target, quarter of the terms) in sorted (a, b) order, so
// a warp reads equal or neighbouring a_w and b_w.  No allocation and no host synchronisation per
// apply, so the QMC report block keeps it inside its CUDA graph.
//
// Bound: HBM, every factor table read once (n = 40, 4 + 4 electrons, 3 references: 1.48 GB, 226 us at the
// copy bandwidth).  Measured there (B200): 1326 -> 390 us an apply against all sources by rows (stage 1
// 323 us for all parents, stage 2 52 us; before, 172 and 255 us for each of the three target parents).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <map>
#include <new>
#include <string>
#include <utility>
#include <vector>

#include "internal.cuh"
#include "wick_math.cuh"

namespace nw {

// Stage 1, rows one by one: a chunk is a run of sources of one row of X1 (or column of X2); `out` is
// stored by the row's only chunk, or added into atomically by each chunk of a longer row (cleared first).
// A block takes a group of consecutive chunks of one table (at most kOvlGroup sources).
struct OvlChunk {
  uint64_t tab;     // table (source-major) in the factor buffer
  uint64_t out;     // row of U or W in the work buffer
  uint32_t k0, k1;  // source list positions
  uint32_t atomic;  // the row has several chunks
  uint32_t pad;
};
struct OvlGroup {
  uint32_t c0, c1;  // chunks
  uint32_t k0, k1;  // their sources
  uint32_t ld;      // row length of the table and of the output
};
// Stage 1, dense tiles: nrow consecutive output rows over nk common table rows.
struct OvlTile {
  uint64_t tab, out;
  uint64_t x0;      // kOvlTile source entries per table row (the last entry + 1: none)
  uint32_t k0, nk;  // table rows
  uint32_t nrow, ld;
};
// One source of a row: table row and position among the distinct (parent, a, b) entries.
struct OvlSource {
  uint32_t row, entry;
};
// Terms of one ordered parent pair in stage 2.
struct OvlPair {
  uint64_t a_tab, b_tab;  // factor tables
  uint64_t u, w;          // first rows of U and W
  uint32_t r0, nr;        // rows R of the source parent (positions in the row list)
  uint32_t c0, nc;        // columns C
};

namespace {

constexpr int kOvlMaxOcc = 16;    // occupied orbitals per spin of the factor kernel
constexpr int kOvlThreads = 256;
constexpr uint32_t kOvlChunk = 64;    // sources per stage-1 chunk
constexpr uint32_t kOvlGroup = 64;    // sources per stage-1 block
constexpr uint32_t kOvlTile = 16;     // rows of a dense stage-1 tile
constexpr uint32_t kOvlTileK = 160;   // table rows of a dense tile held at once (20 KB of sources)
constexpr uint32_t kOvlTargets = 64;  // targets of a stage-2 block (kOvlThreads / kOvlTargets term segments)
constexpr uint64_t kOvlWork = 1ull << 27;  // doubles of U and W per batch of target parents (1 GB)

// One entry of a (source-major) single-spin factor table per thread; MAXO bounds nocc (the LU scratch lives in
// the thread's stack frame, MAXO^2 doubles).
template <int MAXO>
__global__ void __launch_bounds__(kOvlThreads) ovl_factor_kernel(const double* __restrict__ o, int nmo,
                                                                  const uint8_t* __restrict__ occ_t,
                                                                  const uint8_t* __restrict__ occ_s, int nocc,
                                                                  uint32_t nt, uint32_t ns, uint32_t ld,
                                                                  double* __restrict__ out) {
  const uint64_t total = (uint64_t)nt * ns;
  for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < total; e += (uint64_t)gridDim.x * blockDim.x) {
    // consecutive threads write consecutive entries of the output row
    const uint32_t i = (uint32_t)(e % nt), j = (uint32_t)(e / nt);
    const uint8_t* oi = occ_t + (uint64_t)i * nocc;
    const uint8_t* oj = occ_s + (uint64_t)j * nocc;
    double m[MAXO * MAXO];
    for (int r = 0; r < nocc; ++r)
      for (int c = 0; c < nocc; ++c) m[r * nocc + c] = o[(uint64_t)oi[r] * nmo + oj[c]];
    out[(uint64_t)j * ld + i] = det_lu_inplace(m, nocc);
  }
}

// xs[e] = sum of r x over the determinants of distinct entry e (xs[nent] = 0 stands for no source).
__global__ void __launch_bounds__(kOvlThreads) ovl_gather_kernel(uint64_t nent, const uint32_t* __restrict__ first,
                                                                  const uint32_t* __restrict__ ord_det,
                                                                  const double* __restrict__ ord_r,
                                                                  const double* __restrict__ x,
                                                                  double* __restrict__ xs) {
  for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e <= nent; e += (uint64_t)gridDim.x * blockDim.x) {
    double v = 0.0;
    if (e < nent)
      for (uint32_t t = first[e]; t < first[e + 1]; ++t) v += ord_r[t] * x[ord_det[t]];
    xs[e] = v;
  }
}

// Zeros in the output rows that several chunks add into.
__global__ void __launch_bounds__(kOvlThreads) ovl_zero_kernel(const ulonglong2* __restrict__ rows,
                                                                double* __restrict__ u) {
  const ulonglong2 r = rows[blockIdx.x];  // offset, length
  for (uint64_t i = threadIdx.x; i < r.y; i += blockDim.x) u[r.x + i] = 0.0;
}

// Stage 1: blockIdx.x < ntile takes a dense tile (bound by FP64 FMA), the others a group of chunks (bound by
// reading the table); both in one launch, so the tiles' arithmetic runs beside the others' loads.
// blockIdx.y takes 512 columns, two neighbouring ones per thread.
__global__ void __launch_bounds__(kOvlThreads, 3)
    ovl_stage1_kernel(const OvlTile* __restrict__ tiles, uint32_t ntile, const OvlGroup* __restrict__ groups,
                      const OvlChunk* __restrict__ chunks, const OvlSource* __restrict__ src,
                      const uint32_t* __restrict__ trow, const uint32_t* __restrict__ tent,
                      const double* __restrict__ xs, const double* __restrict__ fac, double* __restrict__ u) {
  __shared__ __align__(16) double sx[kOvlTileK * kOvlTile];
  __shared__ uint32_t sb[kOvlTileK];
  const uint32_t col = 2 * (blockIdx.y * blockDim.x + threadIdx.x);
  if (blockIdx.x < ntile) {
    const OvlTile t = tiles[blockIdx.x];
    if (2 * blockIdx.y * blockDim.x >= t.ld) return;
    double2 acc[kOvlTile];
#pragma unroll
    for (uint32_t i = 0; i < kOvlTile; ++i) acc[i] = make_double2(0.0, 0.0);
    for (uint32_t kb = 0; kb < t.nk; kb += kOvlTileK) {
      const uint32_t nk = min(kOvlTileK, t.nk - kb);
      __syncthreads();
      for (uint32_t i = threadIdx.x; i < nk * kOvlTile; i += blockDim.x) sx[i] = xs[tent[t.x0 + kb * kOvlTile + i]];
      for (uint32_t i = threadIdx.x; i < nk; i += blockDim.x) sb[i] = trow[t.k0 + kb + i];
      __syncthreads();
      if (col < t.ld) {
        const double* tab = fac + t.tab + col;
        double2 next = __ldg(reinterpret_cast<const double2*>(tab + (uint64_t)sb[0] * t.ld));
#pragma unroll 2
        for (uint32_t k = 0; k < nk; ++k) {
          const double2 b = next;
          if (k + 1 < nk) next = __ldg(reinterpret_cast<const double2*>(tab + (uint64_t)sb[k + 1] * t.ld));
          const double2* xr = reinterpret_cast<const double2*>(sx + k * kOvlTile);
#pragma unroll
          for (uint32_t i = 0; i < kOvlTile / 2; ++i) {
            const double2 xv = xr[i];
            acc[2 * i].x = fma(xv.x, b.x, acc[2 * i].x);
            acc[2 * i].y = fma(xv.x, b.y, acc[2 * i].y);
            acc[2 * i + 1].x = fma(xv.y, b.x, acc[2 * i + 1].x);
            acc[2 * i + 1].y = fma(xv.y, b.y, acc[2 * i + 1].y);
          }
        }
      }
    }
    if (col >= t.ld) return;
#pragma unroll
    for (uint32_t i = 0; i < kOvlTile; ++i)
      if (i < t.nrow) *reinterpret_cast<double2*>(u + t.out + (uint64_t)i * t.ld + col) = acc[i];
    return;
  }
  const OvlGroup g = groups[blockIdx.x - ntile];
  for (uint32_t i = threadIdx.x; i < g.k1 - g.k0; i += blockDim.x) {
    const OvlSource s = src[g.k0 + i];
    sx[i] = xs[s.entry];
    sb[i] = s.row;
  }
  __syncthreads();
  if (col >= g.ld) return;
  for (uint32_t c = g.c0; c < g.c1; ++c) {
    const OvlChunk ch = chunks[c];
    const double* bt = fac + ch.tab + col;
    auto row = [&](uint32_t k) { return __ldg(reinterpret_cast<const double2*>(bt + (uint64_t)sb[k] * g.ld)); };
    const uint32_t k1 = ch.k1 - g.k0;
    uint32_t k = ch.k0 - g.k0;
    double2 a0 = make_double2(0.0, 0.0), a1 = a0, a2 = a0, a3 = a0;
    for (; k + 4 <= k1; k += 4) {
      const double2 b0 = row(k), b1 = row(k + 1), b2 = row(k + 2), b3 = row(k + 3);
      a0.x += sx[k] * b0.x;
      a0.y += sx[k] * b0.y;
      a1.x += sx[k + 1] * b1.x;
      a1.y += sx[k + 1] * b1.y;
      a2.x += sx[k + 2] * b2.x;
      a2.y += sx[k + 2] * b2.y;
      a3.x += sx[k + 3] * b3.x;
      a3.y += sx[k + 3] * b3.y;
    }
    for (; k < k1; ++k) {
      const double2 b0 = row(k);
      a0.x += sx[k] * b0.x;
      a0.y += sx[k] * b0.y;
    }
    const double s0 = (a0.x + a1.x) + (a2.x + a3.x), s1 = (a0.y + a1.y) + (a2.y + a3.y);
    double* dst = u + ch.out + col;
    if (ch.atomic) {
      atomicAdd(dst, s0);
      atomicAdd(dst + 1, s1);
    } else {
      *reinterpret_cast<double2*>(dst) = make_double2(s0, s1);
    }
  }
}

// y_t += r_t (sum of the stage-2 terms + same-parent sources) for kOvlTargets sorted targets of one
// parent per block; each of the kOvlThreads / kOvlTargets thread rows sums one segment of the terms
// (all P != Q, R then C), added in a fixed order through shared memory.
__global__ void __launch_bounds__(kOvlThreads)
    ovl_stage2_kernel(int q0, int nref, const uint32_t* __restrict__ blk, const uint64_t* __restrict__ pstart,
                      const OvlPair* __restrict__ pairs, const uint32_t* __restrict__ rlist,
                      const uint32_t* __restrict__ clist, const uint32_t* __restrict__ lda,
                      const uint32_t* __restrict__ ldb, const uint32_t* __restrict__ ord_det,
                      const uint32_t* __restrict__ ord_a, const uint32_t* __restrict__ ord_b,
                      const uint32_t* __restrict__ ord_e, const double* __restrict__ ord_r,
                      const double* __restrict__ xs, const double* __restrict__ fac, const double* __restrict__ u,
                      double* __restrict__ y) {
  constexpr int kSeg = kOvlThreads / kOvlTargets;
  __shared__ double part[kSeg][kOvlTargets];
  int q = q0;
  const uint32_t b0 = blk[q0] + blockIdx.x;
  while (b0 >= blk[q + 1]) ++q;
  const int tl = threadIdx.x % kOvlTargets, seg = threadIdx.x / kOvlTargets;
  const uint64_t t = pstart[q] + (uint64_t)(b0 - blk[q]) * kOvlTargets + tl;
  const bool live = t < pstart[q + 1];
  double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
  if (live) {
    const uint32_t at = ord_a[t], bt = ord_b[t];
    const uint64_t la = lda[q], lb = ldb[q];
    for (int p = 0; p < nref; ++p) {
      if (p == q) continue;
      const OvlPair pr = pairs[(uint64_t)q * nref + p];
      {
        const uint32_t k1 = (uint32_t)((uint64_t)pr.nr * (seg + 1) / kSeg);
        uint32_t k = (uint32_t)((uint64_t)pr.nr * seg / kSeg);
        const uint32_t* rl = rlist + pr.r0;
        const double* av = fac + pr.a_tab + at;
        const double* uv = u + pr.u + bt;
        for (; k + 4 <= k1; k += 4) {
          const uint64_t r0 = __ldg(rl + k), r1 = __ldg(rl + k + 1), r2 = __ldg(rl + k + 2), r3 = __ldg(rl + k + 3);
          a0 += __ldg(av + r0 * la) * uv[k * lb];
          a1 += __ldg(av + r1 * la) * uv[(k + 1) * lb];
          a2 += __ldg(av + r2 * la) * uv[(k + 2) * lb];
          a3 += __ldg(av + r3 * la) * uv[(k + 3) * lb];
        }
        for (; k < k1; ++k) a0 += __ldg(av + (uint64_t)__ldg(rl + k) * la) * uv[k * lb];
      }
      {
        const uint32_t k1 = (uint32_t)((uint64_t)pr.nc * (seg + 1) / kSeg);
        uint32_t k = (uint32_t)((uint64_t)pr.nc * seg / kSeg);
        const uint32_t* cl = clist + pr.c0;
        const double* bv = fac + pr.b_tab + bt;
        const double* wv = u + pr.w + at;
        for (; k + 4 <= k1; k += 4) {
          const uint64_t c0 = __ldg(cl + k), c1 = __ldg(cl + k + 1), c2 = __ldg(cl + k + 2), c3 = __ldg(cl + k + 3);
          a0 += __ldg(bv + c0 * lb) * wv[k * la];
          a1 += __ldg(bv + c1 * lb) * wv[(k + 1) * la];
          a2 += __ldg(bv + c2 * lb) * wv[(k + 2) * la];
          a3 += __ldg(bv + c3 * lb) * wv[(k + 3) * la];
        }
        for (; k < k1; ++k) a0 += __ldg(bv + (uint64_t)__ldg(cl + k) * lb) * wv[k * la];
      }
    }
  }
  part[seg][tl] = (a0 + a1) + (a2 + a3);
  __syncthreads();
  if (seg == 0 && live) {
    double v = 0.0;
#pragma unroll
    for (int s = 0; s < kSeg; ++s) v += part[s][tl];
    y[ord_det[t]] += ord_r[t] * (v + xs[ord_e[t]]);
  }
}

inline int grid_of(uint64_t work) {
  const uint64_t g = (work + kOvlThreads - 1) / kOvlThreads;
  return (int)std::max<uint64_t>(1, std::min<uint64_t>(g, 148ull * 16));
}

// Fermionic sign of the excitation (excitation_phase_bits, src/basis/excitation.rs:110-146):
// holes removed from the highest down, particles added from the lowest up, each contributing
// the parity of the occupied orbitals below it.
double excitation_sign(int nocc, int rank, const uint8_t* idx) {
  char occ[256] = {};  // orbital indices are bytes
  for (int i = 0; i < nocc && i < 256; ++i) occ[i] = 1;
  auto below = [&](int p) {
    int c = 0;
    for (int i = 0; i < p; ++i) c += occ[i];
    return c & 1;
  };
  int odd = 0;
  for (int k = rank - 1; k >= 0; --k) {
    odd ^= below(idx[k]);
    occ[idx[k]] = 0;
  }
  for (int k = 0; k < rank; ++k) {
    odd ^= below(idx[4 + k]);
    if (k + 1 != rank) occ[idx[4 + k]] = 1;
  }
  return odd ? -1.0 : 1.0;
}

using SpinKey = std::pair<int, uint64_t>;

SpinKey spin_key(int rank, const uint8_t* idx) {
  uint64_t v = 0;
  for (int k = 0; k < rank; ++k) {
    v |= (uint64_t)idx[k] << (8 * k);
    v |= (uint64_t)idx[4 + k] << (8 * (4 + k));
  }
  return {rank, v};
}

}  // namespace

struct OverlapPlan {
  // Target parents [q0, q1) whose U and W fit the work buffer together, with their stage-1 work.
  struct Batch {
    int q0, q1;
    uint64_t tile0, ntile, group0, ngroup, zero0, nzero;
    uint32_t ldmax;
    uint32_t nblk;  // stage-2 blocks
  };
  int nref = 0, oa = 0, ob = 0;
  uint64_t ndet = 0, nent = 0;
  std::vector<uint32_t> na, nb;
  std::vector<uint32_t> lda, ldb;       // alpha / beta strings per parent rounded up to even: table row lengths
  std::vector<uint64_t> pstart;         // per parent: first sorted position (nref + 1)
  std::vector<Batch> batches;
  void* mem = nullptr;
  uint32_t* ord_det = nullptr;
  uint32_t* ord_a = nullptr;
  uint32_t* ord_b = nullptr;
  uint32_t* ord_e = nullptr;
  double* ord_r = nullptr;
  uint32_t* first = nullptr;            // first sorted position of each distinct entry (nent + 1)
  OvlTile* tiles = nullptr;
  OvlGroup* groups = nullptr;
  OvlChunk* chunks = nullptr;
  OvlSource* src = nullptr;
  uint32_t* trow = nullptr;
  uint32_t* tent = nullptr;
  ulonglong2* zero_rows = nullptr;
  OvlPair* pairs = nullptr;
  uint32_t* rlist = nullptr;
  uint32_t* clist = nullptr;
  uint32_t* d_lda = nullptr;
  uint32_t* d_ldb = nullptr;
  uint32_t* d_blk = nullptr;
  uint64_t* d_pstart = nullptr;
  double* fac = nullptr;
  double* u = nullptr;
  double* xs = nullptr;
};

namespace {

// The sources of one parent by rows (or columns): for each line its id and its (table row, entry) list.
struct Lines {
  std::vector<uint32_t> id;
  std::vector<std::vector<OvlSource>> src;
};

// Split of one parent's distinct entries into lines by rows (R) and by columns (C), see the header.  `rows` and
// `cols` count each alpha and beta string's entries; targets, nb and na are the other parents' averages.
void split_sources(const std::vector<uint32_t>& ea, const std::vector<uint32_t>& eb, uint32_t na, uint32_t nb,
                   uint64_t e0, double targets, double tna, double tnb, Lines* R, Lines* C) {
  const size_t ne = ea.size();
  std::vector<uint32_t> rows(na, 0), cols(nb, 0);
  for (size_t e = 0; e < ne; ++e) {
    ++rows[ea[e]];
    ++cols[eb[e]];
  }
  auto by_row = [&](int mode, size_t e) { return mode == 0 ? rows[ea[e]] >= cols[eb[e]] : mode == 1; };
  int best = 0;
  double best_cost = 0.0;
  for (int mode = 0; mode < 3; ++mode) {  // the rule, all by rows, all by columns
    std::vector<char> r(na, 0), c(nb, 0);
    double cost = 0.0;
    for (size_t e = 0; e < ne; ++e) {
      if (by_row(mode, e)) {
        r[ea[e]] = 1;
        cost += tnb;
      } else {
        c[eb[e]] = 1;
        cost += tna;
      }
    }
    for (char k : r) cost += k ? targets : 0.0;
    for (char k : c) cost += k ? targets : 0.0;
    if (mode == 0 || cost < best_cost) {
      best = mode;
      best_cost = cost;
    }
  }
  std::vector<std::vector<OvlSource>> lr(na), lc(nb);
  // entries come in (a, b) order, so every line's list is in table-row order
  for (size_t e = 0; e < ne; ++e) {
    if (by_row(best, e))
      lr[ea[e]].push_back(OvlSource{eb[e], (uint32_t)(e0 + e)});
    else
      lc[eb[e]].push_back(OvlSource{ea[e], (uint32_t)(e0 + e)});
  }
  auto collect = [](std::vector<std::vector<OvlSource>>& l, Lines* out) {
    std::vector<uint32_t> id;
    for (uint32_t i = 0; i < l.size(); ++i)
      if (!l[i].empty()) id.push_back(i);
    // lines of equal length next to each other, so that lines with the same entries share a tile
    std::stable_sort(id.begin(), id.end(), [&](uint32_t x, uint32_t y) { return l[x].size() > l[y].size(); });
    for (uint32_t i : id) {
      out->id.push_back(i);
      out->src.push_back(std::move(l[i]));
    }
  };
  collect(lr, R);
  collect(lc, C);
}

}  // namespace

void overlap_plan_free(OverlapPlan* pl) {
  if (!pl) return;
  if (pl->mem) cudaFree(pl->mem);
  delete pl;
}

nw_status overlap_plan_get(nw_ctx* ctx, cudaStream_t stream, OverlapPlan** out) {
  if (ctx->ovl) {
    *out = ctx->ovl;
    return NW_OK;
  }
  if (!ctx->d_dets || ctx->ndet == 0) return fail(ctx, NW_ERR_STATE, "the overlap action needs a resident basis");
  if (ctx->nocc_a > kOvlMaxOcc || ctx->nocc_b > kOvlMaxOcc)
    return fail(ctx, NW_ERR_UNSUPPORTED, "the overlap action supports at most 16 occupied orbitals per spin");
  const int nref = ctx->nref, nmo = ctx->nmo, nao = ctx->nao;
  const uint64_t nd = ctx->ndet;
  std::vector<nw_det> dets(nd);
  NW_CUDA(ctx, cudaMemcpyAsync(dets.data(), ctx->d_dets, nd * sizeof(nw_det), cudaMemcpyDeviceToHost, stream));
  NW_CUDA(ctx, cudaStreamSynchronize(stream));

  OverlapPlan* pl = new (std::nothrow) OverlapPlan;
  if (!pl) return NW_ERR_ALLOC;
  pl->nref = nref;
  pl->oa = ctx->nocc_a;
  pl->ob = ctx->nocc_b;
  pl->ndet = nd;
  // parent-local single-spin components
  std::vector<std::map<SpinKey, uint32_t>> ca(nref), cb(nref);
  std::vector<uint32_t> aid(nd), bid(nd);
  std::vector<double> rr(nd);
  for (uint64_t d = 0; d < nd; ++d) {
    const nw_det& r = dets[d];
    const SpinKey ka = spin_key(r.rank_a, r.idx_a), kb = spin_key(r.rank_b, r.idx_b);
    auto ia = ca[r.parent].emplace(ka, (uint32_t)ca[r.parent].size()).first;
    auto ib = cb[r.parent].emplace(kb, (uint32_t)cb[r.parent].size()).first;
    aid[d] = ia->second;
    bid[d] = ib->second;
    rr[d] = r.phase * excitation_sign(ctx->nocc_a, r.rank_a, r.idx_a) * excitation_sign(ctx->nocc_b, r.rank_b, r.idx_b);
  }
  pl->na.resize(nref);
  pl->nb.resize(nref);
  pl->lda.resize(nref);
  pl->ldb.resize(nref);
  std::vector<uint64_t> ca_off(nref + 1, 0), cb_off(nref + 1, 0);
  for (int p = 0; p < nref; ++p) {
    pl->na[p] = (uint32_t)ca[p].size();
    pl->nb[p] = (uint32_t)cb[p].size();
    pl->lda[p] = (pl->na[p] + 1) & ~1u;
    pl->ldb[p] = (pl->nb[p] + 1) & ~1u;
    ca_off[p + 1] = ca_off[p] + pl->na[p];
    cb_off[p + 1] = cb_off[p] + pl->nb[p];
  }
  // occupied orbitals of every component, ascending
  std::vector<uint8_t> occ_a(std::max<uint64_t>(1, ca_off[nref] * pl->oa)), occ_b(std::max<uint64_t>(1, cb_off[nref] * pl->ob));
  auto fill_occ = [&](const SpinKey& k, int nocc, uint8_t* dst) {
    const int rank = k.first;
    std::vector<int> o;
    for (int i = 0; i < nocc; ++i) {
      bool hole = false;
      for (int h = 0; h < rank; ++h) hole |= ((k.second >> (8 * h)) & 0xFF) == (uint64_t)i;
      if (!hole) o.push_back(i);
    }
    for (int h = 0; h < rank; ++h) o.push_back((int)((k.second >> (8 * (4 + h))) & 0xFF));
    std::sort(o.begin(), o.end());
    for (int i = 0; i < nocc; ++i) dst[i] = (uint8_t)o[i];
  };
  for (int p = 0; p < nref; ++p) {
    for (const auto& kv : ca[p]) fill_occ(kv.first, pl->oa, occ_a.data() + (ca_off[p] + kv.second) * pl->oa);
    for (const auto& kv : cb[p]) fill_occ(kv.first, pl->ob, occ_b.data() + (cb_off[p] + kv.second) * pl->ob);
  }
  // sorted order (parent, a, b)
  std::vector<uint32_t> order(nd);
  for (uint64_t d = 0; d < nd; ++d) order[d] = (uint32_t)d;
  std::sort(order.begin(), order.end(), [&](uint32_t x, uint32_t y) {
    if (dets[x].parent != dets[y].parent) return dets[x].parent < dets[y].parent;
    if (aid[x] != aid[y]) return aid[x] < aid[y];
    if (bid[x] != bid[y]) return bid[x] < bid[y];
    return x < y;
  });
  std::vector<uint32_t> o_a(nd), o_b(nd), o_e(nd), first;
  std::vector<double> o_r(nd);
  pl->pstart.assign(nref + 1, nd);
  // distinct (parent, a, b) entries in sorted order
  std::vector<std::vector<uint32_t>> ea(nref), eb(nref);
  std::vector<uint64_t> estart(nref + 1, 0);
  for (uint64_t t = 0; t < nd; ++t) {
    const uint32_t d = order[t];
    const uint32_t p = dets[d].parent;
    o_a[t] = aid[d];
    o_b[t] = bid[d];
    o_r[t] = rr[d];
    const bool np = t == 0 || dets[order[t - 1]].parent != p;
    if (np) pl->pstart[p] = t;
    if (np || o_a[t - 1] != o_a[t] || o_b[t - 1] != o_b[t]) {
      first.push_back((uint32_t)t);
      ea[p].push_back(o_a[t]);
      eb[p].push_back(o_b[t]);
    }
    o_e[t] = (uint32_t)first.size() - 1;
  }
  pl->nent = first.size();
  first.push_back((uint32_t)nd);
  for (int p = 0; p < nref; ++p) estart[p + 1] = estart[p] + ea[p].size();
  for (int p = nref - 1; p >= 0; --p)
    if (pl->pstart[p] > pl->pstart[p + 1]) pl->pstart[p] = pl->pstart[p + 1];  // parents without determinants
  // rows and columns of every source parent
  std::vector<Lines> R(nref), C(nref);
  std::vector<uint32_t> rlist, clist, r0(nref), c0(nref);
  for (int p = 0; p < nref && nref > 1; ++p) {
    double targets = 0.0, tna = 0.0, tnb = 0.0;
    for (int q = 0; q < nref; ++q)
      if (q != p) {
        targets += (double)(pl->pstart[q + 1] - pl->pstart[q]);
        tna += pl->na[q];
        tnb += pl->nb[q];
      }
    split_sources(ea[p], eb[p], pl->na[p], pl->nb[p], estart[p], targets, tna, tnb, &R[p], &C[p]);
    r0[p] = (uint32_t)rlist.size();
    c0[p] = (uint32_t)clist.size();
    rlist.insert(rlist.end(), R[p].id.begin(), R[p].id.end());
    clist.insert(clist.end(), C[p].id.begin(), C[p].id.end());
  }
  // factor tables, U and W rows and the stage-1 work per batch of target parents
  std::vector<uint64_t> a_off((size_t)nref * nref, 0), bt_off((size_t)nref * nref, 0);
  std::vector<OvlPair> pairs((size_t)nref * nref, OvlPair{});
  uint64_t nfac = 0, nu = 0;
  std::vector<OvlTile> tiles;
  std::vector<OvlGroup> groups;
  std::vector<OvlChunk> chunks;
  std::vector<OvlSource> src;
  std::vector<uint32_t> trow, tent, blk(nref + 1, 0);
  std::vector<ulonglong2> zero_rows;
  for (int q = 0; q < nref; ++q)
    blk[q + 1] = blk[q] + (uint32_t)((pl->pstart[q + 1] - pl->pstart[q] + kOvlTargets - 1) / kOvlTargets);
  // the lists of one source parent's lines are shared by all its targets: tile and chunk shapes per line set
  struct Shape {
    bool tile;
    uint32_t l0, nl;     // lines
    uint32_t k0, nk;     // tile: table rows; line: sources in `src`
    uint64_t x0;
  };
  auto shapes_of = [&](const Lines& L, uint32_t nrows) {
    std::vector<Shape> out;
    std::vector<uint32_t> rows, seen(nrows, 0), place(nrows);  // distinct table rows of a window of lines
    uint32_t window = 0;
    for (uint32_t l = 0; l < L.id.size();) {
      // a tile where the lines share their entries: at most 1.5 times the work of the lines one by one
      const uint32_t nl = std::min<uint32_t>(kOvlTile, (uint32_t)L.id.size() - l);
      rows.clear();
      ++window;
      uint64_t nnz = 0;
      for (uint32_t i = 0; i < nl; ++i) {
        nnz += L.src[l + i].size();
        for (const OvlSource& s : L.src[l + i])
          if (seen[s.row] != window) {
            seen[s.row] = window;
            rows.push_back(s.row);
          }
      }
      if (nl >= 4 && 2 * rows.size() * nl <= 3 * nnz) {
        std::sort(rows.begin(), rows.end());
        for (uint32_t k = 0; k < rows.size(); ++k) place[rows[k]] = k;
        const Shape sh{true, l, nl, (uint32_t)trow.size(), (uint32_t)rows.size(), tent.size()};
        trow.insert(trow.end(), rows.begin(), rows.end());
        tent.resize(sh.x0 + rows.size() * kOvlTile, (uint32_t)pl->nent);
        for (uint32_t i = 0; i < nl; ++i)
          for (const OvlSource& s : L.src[l + i]) tent[sh.x0 + (uint64_t)place[s.row] * kOvlTile + i] = s.entry;
        out.push_back(sh);
        l += nl;
      } else {
        out.push_back(Shape{false, l, 1, (uint32_t)src.size(), (uint32_t)L.src[l].size(), 0});
        src.insert(src.end(), L.src[l].begin(), L.src[l].end());
        ++l;
      }
    }
    return out;
  };
  std::vector<std::vector<Shape>> rshape(nref), cshape(nref);
  for (int p = 0; p < nref; ++p) {
    rshape[p] = shapes_of(R[p], pl->nb[p]);
    cshape[p] = shapes_of(C[p], pl->na[p]);
  }
  auto work_of = [&](int q) {
    uint64_t w = 0;
    for (int p = 0; p < nref; ++p)
      if (p != q) w += (uint64_t)R[p].id.size() * pl->ldb[q] + (uint64_t)C[p].id.size() * pl->lda[q];
    return w;
  };
  for (int q = 0; q < nref && nref > 1;) {
    OverlapPlan::Batch bt{q, q, tiles.size(), 0, groups.size(), 0, zero_rows.size(), 0, 2, 0};
    uint64_t uq = 0;
    while (bt.q1 < nref && (bt.q1 == bt.q0 || uq + work_of(bt.q1) <= kOvlWork)) {
      const int qq = bt.q1++;
      bt.nblk += blk[qq + 1] - blk[qq];
      if (pl->pstart[qq + 1] == pl->pstart[qq]) continue;
      bt.ldmax = std::max(bt.ldmax, std::max(pl->lda[qq], pl->ldb[qq]));
      for (int p = 0; p < nref; ++p) {
        if (p == qq) continue;
        const size_t i = (size_t)qq * nref + p;
        nfac = (nfac + 1) & ~1ull;  // 16-byte aligned table rows
        a_off[i] = nfac;
        nfac += (uint64_t)pl->na[p] * pl->lda[qq];
        bt_off[i] = nfac;
        nfac += (uint64_t)pl->nb[p] * pl->ldb[qq];
        OvlPair& pr = pairs[i];
        pr = OvlPair{a_off[i], bt_off[i], 0, 0, r0[p], (uint32_t)R[p].id.size(), c0[p], (uint32_t)C[p].id.size()};
        for (int side = 0; side < 2; ++side) {
          const uint32_t ld = side ? pl->lda[qq] : pl->ldb[qq];
          const uint64_t tab = side ? a_off[i] : bt_off[i];
          (side ? pr.w : pr.u) = uq;
          bool open = false;  // a group never spans two tables
          for (const Shape& sh : side ? cshape[p] : rshape[p]) {
            const uint64_t out = uq + (uint64_t)sh.l0 * ld;
            if (sh.tile) {
              tiles.push_back(OvlTile{tab, out, sh.x0, sh.k0, sh.nk, sh.nl, ld});
              continue;
            }
            const bool multi = sh.nk > kOvlChunk;
            if (multi) zero_rows.push_back(make_ulonglong2(out, ld));
            for (uint32_t k = 0; k < sh.nk; k += kOvlChunk) {
              const uint32_t ka = sh.k0 + k, kb = sh.k0 + std::min(sh.nk, k + kOvlChunk);
              // a group's sources are consecutive in the list (a tile between two lines does not break that)
              if (!open || kb - groups.back().k0 > kOvlGroup || ka != groups.back().k1) {
                groups.push_back(OvlGroup{(uint32_t)chunks.size(), (uint32_t)chunks.size(), ka, ka, ld});
                open = true;
              }
              chunks.push_back(OvlChunk{tab, out, ka, kb, multi ? 1u : 0u, 0u});
              groups.back().c1 = (uint32_t)chunks.size();
              groups.back().k1 = kb;
            }
          }
          uq += (uint64_t)(side ? C[p].id.size() : R[p].id.size()) * ld;
        }
      }
    }
    bt.ntile = tiles.size() - bt.tile0;
    bt.ngroup = groups.size() - bt.group0;
    bt.nzero = zero_rows.size() - bt.zero0;
    nu = std::max(nu, uq);
    pl->batches.push_back(bt);
    q = bt.q1;
  }
  if (nref == 1) pl->batches.push_back(OverlapPlan::Batch{0, 1, 0, 0, 0, 0, 0, 0, 2, blk[1]});
  // one allocation: device arrays, factor tables, work buffers and the MO overlaps of the set-up
  const size_t n2 = (size_t)nmo * nmo;
  const size_t nrr = (size_t)nref * nref;
  size_t off = 0;
  auto carve = [&](size_t bytes) {
    const size_t at = off;
    off += (bytes + 255) & ~(size_t)255;
    return at;
  };
  auto some = [](size_t n) { return std::max<size_t>(1, n); };
  const size_t o_det = carve(nd * 4), o_a_ = carve(nd * 4), o_b_ = carve(nd * 4), o_e_ = carve(nd * 4);
  const size_t o_r_ = carve(nd * 8), o_first = carve(first.size() * 4);
  const size_t o_tiles = carve(some(tiles.size()) * sizeof(OvlTile));
  const size_t o_groups = carve(some(groups.size()) * sizeof(OvlGroup));
  const size_t o_chunks = carve(some(chunks.size()) * sizeof(OvlChunk));
  const size_t o_src = carve(some(src.size()) * sizeof(OvlSource));
  const size_t o_trow = carve(some(trow.size()) * 4), o_tent = carve(some(tent.size()) * 4);
  const size_t o_zero = carve(some(zero_rows.size()) * sizeof(ulonglong2));
  const size_t o_pairs = carve(nrr * sizeof(OvlPair));
  const size_t o_rl = carve(some(rlist.size()) * 4), o_cl = carve(some(clist.size()) * 4);
  const size_t o_lda = carve(nref * 4), o_ldb = carve(nref * 4), o_blk = carve((nref + 1) * 4);
  const size_t o_ps = carve((nref + 1) * 8);
  const size_t o_occa = carve(occ_a.size()), o_occb = carve(occ_b.size());
  const size_t o_fac = carve(some(nfac) * 8), o_u = carve(some(nu) * 8);
  const size_t o_xs = carve((pl->nent + 1) * 8);
  const size_t o_t = carve((size_t)nref * nao * nmo * 8), o_o = carve(2 * nrr * n2 * 8);
  if (ctx_malloc(ctx, reinterpret_cast<void**>(&pl->mem), off) != cudaSuccess) {
    pl->mem = nullptr;
    overlap_plan_free(pl);
    return fail(ctx, NW_ERR_ALLOC,
                "the overlap factor tables need " + std::to_string(off >> 20) + " MiB, more than the free device memory");
  }
  char* base = static_cast<char*>(pl->mem);
  pl->ord_det = reinterpret_cast<uint32_t*>(base + o_det);
  pl->ord_a = reinterpret_cast<uint32_t*>(base + o_a_);
  pl->ord_b = reinterpret_cast<uint32_t*>(base + o_b_);
  pl->ord_e = reinterpret_cast<uint32_t*>(base + o_e_);
  pl->ord_r = reinterpret_cast<double*>(base + o_r_);
  pl->first = reinterpret_cast<uint32_t*>(base + o_first);
  pl->tiles = reinterpret_cast<OvlTile*>(base + o_tiles);
  pl->groups = reinterpret_cast<OvlGroup*>(base + o_groups);
  pl->chunks = reinterpret_cast<OvlChunk*>(base + o_chunks);
  pl->src = reinterpret_cast<OvlSource*>(base + o_src);
  pl->trow = reinterpret_cast<uint32_t*>(base + o_trow);
  pl->tent = reinterpret_cast<uint32_t*>(base + o_tent);
  pl->zero_rows = reinterpret_cast<ulonglong2*>(base + o_zero);
  pl->pairs = reinterpret_cast<OvlPair*>(base + o_pairs);
  pl->rlist = reinterpret_cast<uint32_t*>(base + o_rl);
  pl->clist = reinterpret_cast<uint32_t*>(base + o_cl);
  pl->d_lda = reinterpret_cast<uint32_t*>(base + o_lda);
  pl->d_ldb = reinterpret_cast<uint32_t*>(base + o_ldb);
  pl->d_blk = reinterpret_cast<uint32_t*>(base + o_blk);
  pl->d_pstart = reinterpret_cast<uint64_t*>(base + o_ps);
  uint8_t* d_occa = reinterpret_cast<uint8_t*>(base + o_occa);
  uint8_t* d_occb = reinterpret_cast<uint8_t*>(base + o_occb);
  pl->fac = reinterpret_cast<double*>(base + o_fac);
  pl->u = reinterpret_cast<double*>(base + o_u);
  pl->xs = reinterpret_cast<double*>(base + o_xs);
  double* d_t = reinterpret_cast<double*>(base + o_t);
  double* d_o = reinterpret_cast<double*>(base + o_o);
  auto up = [&](void* dst, const void* src, size_t bytes) {
    return bytes == 0 || cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, stream) == cudaSuccess;
  };
  // the padding column of an odd-length table row is summed by stage 1 into a column nobody reads
  const bool ok_up =
      up(pl->ord_det, order.data(), nd * 4) && up(pl->ord_a, o_a.data(), nd * 4) && up(pl->ord_b, o_b.data(), nd * 4) &&
      up(pl->ord_e, o_e.data(), nd * 4) && up(pl->ord_r, o_r.data(), nd * 8) &&
      up(pl->first, first.data(), first.size() * 4) && up(pl->tiles, tiles.data(), tiles.size() * sizeof(OvlTile)) &&
      up(pl->groups, groups.data(), groups.size() * sizeof(OvlGroup)) &&
      up(pl->chunks, chunks.data(), chunks.size() * sizeof(OvlChunk)) &&
      up(pl->src, src.data(), src.size() * sizeof(OvlSource)) && up(pl->trow, trow.data(), trow.size() * 4) &&
      up(pl->tent, tent.data(), tent.size() * 4) &&
      up(pl->zero_rows, zero_rows.data(), zero_rows.size() * sizeof(ulonglong2)) &&
      up(pl->pairs, pairs.data(), nrr * sizeof(OvlPair)) && up(pl->rlist, rlist.data(), rlist.size() * 4) &&
      up(pl->clist, clist.data(), clist.size() * 4) && up(pl->d_lda, pl->lda.data(), nref * 4) &&
      up(pl->d_ldb, pl->ldb.data(), nref * 4) && up(pl->d_blk, blk.data(), blk.size() * 4) &&
      up(pl->d_pstart, pl->pstart.data(), pl->pstart.size() * 8) && up(d_occa, occ_a.data(), occ_a.size()) &&
      up(d_occb, occ_b.data(), occ_b.size());
  bool ok = ok_up && cudaMemsetAsync(pl->fac, 0, some(nfac) * 8, stream) == cudaSuccess;
  // O^{QP}_sigma = C_Q^T (S C_P): nmo x nmo per ordered pair and spin, then the factor tables
  for (int spin = 0; ok && spin < 2 && nref > 1; ++spin) {
    const double* c = spin ? ctx->d_cb : ctx->d_ca;
    const long long cs = (long long)nao * nmo;
    ok = dgemm_strided(stream, false, false, nao, nmo, nao, 1.0, ctx->d_s, nao, 0, c, nmo, cs, 0.0, d_t, nmo, cs,
                       nref) == cudaSuccess;
    for (int q = 0; ok && q < nref; ++q)
      ok = dgemm_strided(stream, true, false, nmo, nmo, nao, 1.0, c + q * cs, nmo, 0, d_t, nmo, cs, 0.0,
                         d_o + ((size_t)spin * nrr + (size_t)q * nref) * n2, nmo, (long long)n2, nref) == cudaSuccess;
  }
  auto factors = [&](const double* o, const uint8_t* ot, const uint8_t* os, int nocc, uint32_t nt, uint32_t ns,
                     uint32_t ld, double* out) {
    const uint64_t e = (uint64_t)nt * ns;
    if (e == 0) return;
    if (nocc <= 4)
      ovl_factor_kernel<4><<<grid_of(e), kOvlThreads, 0, stream>>>(o, nmo, ot, os, nocc, nt, ns, ld, out);
    else if (nocc <= 8)
      ovl_factor_kernel<8><<<grid_of(e), kOvlThreads, 0, stream>>>(o, nmo, ot, os, nocc, nt, ns, ld, out);
    else
      ovl_factor_kernel<kOvlMaxOcc><<<grid_of(e), kOvlThreads, 0, stream>>>(o, nmo, ot, os, nocc, nt, ns, ld, out);
  };
  for (int q = 0; ok && q < nref; ++q)
    for (int p = 0; ok && p < nref; ++p) {
      if (p == q || pl->pstart[q + 1] == pl->pstart[q]) continue;
      const size_t i = (size_t)q * nref + p;
      factors(d_o + i * n2, d_occa + ca_off[q] * pl->oa, d_occa + ca_off[p] * pl->oa, pl->oa, pl->na[q], pl->na[p],
              pl->lda[q], pl->fac + a_off[i]);
      factors(d_o + (nrr + i) * n2, d_occb + cb_off[q] * pl->ob, d_occb + cb_off[p] * pl->ob, pl->ob, pl->nb[q],
              pl->nb[p], pl->ldb[q], pl->fac + bt_off[i]);
      ok = cudaGetLastError() == cudaSuccess;
    }
  if (ok) ok = cudaStreamSynchronize(stream) == cudaSuccess;
  if (!ok) {
    overlap_plan_free(pl);
    return fail(ctx, NW_ERR_CUDA, "overlap factor table set-up failed");
  }
  ctx->ovl = pl;
  *out = pl;
  return NW_OK;
}

nw_status overlap_apply(nw_ctx* ctx, const OverlapPlan* pl, const double* x, double* y, cudaStream_t stream) {
  ovl_gather_kernel<<<grid_of(pl->nent + 1), kOvlThreads, 0, stream>>>(pl->nent, pl->first, pl->ord_det, pl->ord_r, x,
                                                                       pl->xs);
  for (const OverlapPlan::Batch& b : pl->batches) {
    if (b.nzero > 0)
      ovl_zero_kernel<<<(unsigned)b.nzero, kOvlThreads, 0, stream>>>(pl->zero_rows + b.zero0, pl->u);
    if (b.ntile + b.ngroup > 0)
      ovl_stage1_kernel<<<dim3((unsigned)(b.ntile + b.ngroup), (b.ldmax + 2 * kOvlThreads - 1) / (2 * kOvlThreads)),
                          kOvlThreads, 0, stream>>>(pl->tiles + b.tile0, (uint32_t)b.ntile, pl->groups + b.group0,
                                                    pl->chunks, pl->src, pl->trow, pl->tent, pl->xs, pl->fac, pl->u);
    if (b.nblk > 0)
      ovl_stage2_kernel<<<b.nblk, kOvlThreads, 0, stream>>>(b.q0, pl->nref, pl->d_blk, pl->d_pstart, pl->pairs,
                                                            pl->rlist, pl->clist, pl->d_lda, pl->d_ldb, pl->ord_det,
                                                            pl->ord_a, pl->ord_b, pl->ord_e, pl->ord_r, pl->xs,
                                                            pl->fac, pl->u, y);
  }
  NW_CUDA(ctx, cudaGetLastError());
  return NW_OK;
}

}  // namespace nw

extern "C" {

nw_status nw_apply_overlap_device(nw_ctx* ctx, const double* x_dev, double* y_dev, void* stream) {
  if (!ctx || !x_dev || !y_dev) return NW_ERR_INVALID;
  const cudaStream_t s = static_cast<cudaStream_t>(stream);
  nw::CtxGuard guard(ctx, s);
  NW_CUDA(ctx, cudaSetDevice(ctx->device));
  nw::OverlapPlan* pl = nullptr;
  const nw_status st = nw::overlap_plan_get(ctx, s, &pl);
  if (st != NW_OK) return st;
  return nw::overlap_apply(ctx, pl, x_dev, y_dev, s);
}

}  // extern "C"
