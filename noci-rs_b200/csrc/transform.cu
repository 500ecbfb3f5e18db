// Four-index transforms of the build for orbital spaces up to 64, in two fused half transforms.
//
// A tensor of the build is N[pq][rs] = sum A[mu,p] B[nu,q] (mu nu|lam sig) C[lam,r] D[sig,s].  Each
// half is a batch of two-sided products  out = A^T In B  with one n x n matrix In per batch entry:
//   first half   In = (lam sig| . .), lam >= sig only (the tensor is symmetric under lam <-> sig and
//                under exchange of the pairs): H[pq][u], u = lam (lam + 1) / 2 + sig;
//   second half  In = H[pq][.] unpacked to its symmetric square: N[pq][rs] in natural order.
// Both quarter transforms of a half run in one kernel: the first product's DMMA accumulators are the
// second product's A fragments as they lie in registers (thread tig of a quad holds columns 2 tig and
// 2 tig + 1 of each 8-column tile; the second operand's rows are stored permuted to match), so the
// intermediate never leaves the register file.
//
// Bound: the FP64 tensor pipe (n = 64: 4 n^3 flops per 32 KB read and 32 KB written).  A block keeps
// A and B and a group of 4 matrices in shared memory (n = 64: 209 KB, one block of 8 warps per SM;
// smaller n pack 6 to 16 matrices); a warp owns 16 rows of two matrices, so an A or B fragment is loaded
// once for both, and the next group's cp.async runs under the second product, which no longer
// reads the matrices.  The four separate quarter transforms this replaces (a GEMM with K = n each,
// 64 x 64 tiles) moved the n^4 intermediate through memory four times, computed both (lam sig) and
// (sig lam), and repeated the first half for every tensor that shares it.
//
// Measured (B200): the second half at n = 64 runs at 28 TFLOP/s (FP64 tensor pipe 79 % active, ncu), the
// quarter transforms at 21; a build of 3 references with one zero-overlap reference pair, 31.7 -> 12.5 ms
// at n = 64 and, without one, 3.36 -> 0.91 ms at n = 30 (11.2 and 0.475 ms since the other products of the build
// share launches).  Larger n (matrices beyond shared memory) and tensors
// without the symmetry keep the quarter transforms.
#include <cuda_runtime.h>

#include "internal.cuh"

namespace nw {
namespace {

template <int N8>
struct TwoSided {
  static constexpr int RG = (N8 + 1) / 2;                             // 16-row groups of a matrix
  static constexpr int PAIRS = RG == 1 ? 8 : RG == 2 ? 4 : RG == 3 ? 3 : 2;  // matrix pairs of a block
  static constexpr int WARPS = RG * PAIRS;
  static constexpr int THREADS = 32 * WARPS;
  static constexpr int MATS = 2 * PAIRS;
  static constexpr int NP = 8 * N8;
  static constexpr int LD = NP + 4;                // = 4 mod 8: conflict-free fragment loads
  static constexpr int MSZ = NP * LD;              // doubles of one matrix
  static constexpr int BSZ = MSZ + 16;             // A is read up to column 16 RG - 1 of its last row
  static constexpr int BLOCKS = N8 <= 4 ? 2 : 1;   // resident blocks per SM
  static constexpr size_t smem(int npack) {
    return sizeof(double) * ((size_t)MATS * MSZ + 2 * BSZ) + sizeof(uint32_t) * (size_t)npack;
  }
};

__device__ __forceinline__ void dmma1688(double (&d)[4], const double (&a)[4], double b0, double b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};\n"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b0), "d"(b1));
}

__device__ __forceinline__ void cp8(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp16(double* dst, const double* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// u -> (lam, sig), lam >= sig, u = lam (lam + 1) / 2 + sig  (u < 2080)
__device__ __forceinline__ void unpack_pair(int u, int* lam, int* sig) {
  int l = (int)((sqrtf(8.0f * (float)u + 1.0f) - 1.0f) * 0.5f);
  while (l * (l + 1) / 2 > u) --l;
  while ((l + 1) * (l + 2) / 2 <= u) ++l;
  *lam = l;
  *sig = u - l * (l + 1) / 2;
}

// Blocks walk a contiguous range of (task, group of MATS matrices).  HALF: In is row (lam sig) of the
// Coulomb tensor and out is transposed to H[pq][u]; else In is unpacked from H and out is natural
// (kStore) or subtracted in the J order (kSubtract).
template <int N8, bool HALF>
__global__ void __launch_bounds__(TwoSided<N8>::THREADS, TwoSided<N8>::BLOCKS)
    two_sided_kernel(const TransformTask* __restrict__ tasks, int ntask, int n, int nmat, int npack, int ldu) {
  using T = TwoSided<N8>;
  extern __shared__ __align__(16) double tsm[];
  double* in = tsm;
  double* as = in + (size_t)T::MATS * T::MSZ;
  double* bs = as + T::BSZ;
  uint32_t* tab = reinterpret_cast<uint32_t*>(bs + T::BSZ);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int grp = lane >> 2, tig = lane & 3;
  const int rg = warp % T::RG, pr = warp / T::RG;
  const long long n2 = (long long)n * n;
  const long long ngroup = (nmat + T::MATS - 1) / T::MATS, total = ngroup * ntask;
  const long long it0 = total * blockIdx.x / gridDim.x, it1 = total * (blockIdx.x + 1) / gridDim.x;
  if (it0 >= it1) return;

  // rows and columns past n stay zero: the copies never touch them
  for (int i = tid; i < T::MATS * T::MSZ + 2 * T::BSZ; i += T::THREADS) tsm[i] = 0.0;
  if (!HALF)
    for (int u = tid; u < npack; u += T::THREADS) {
      int l, s;
      unpack_pair(u, &l, &s);
      tab[u] = (uint32_t)(l * T::LD + s) | ((uint32_t)(s * T::LD + l) << 16);
    }
  __syncthreads();

  auto load_ab = [&](const TransformTask& t) {
    for (int i = tid; i < (int)n2; i += T::THREADS) {
      const int r = i / n, c = i % n;
      as[r * T::LD + c] = t.a[i];
      bs[((r & ~7) | ((r & 1) << 2) | ((r & 7) >> 1)) * T::LD + c] = t.b[i];
    }
  };
  // the RG warps of a matrix pair copy their own two matrices and synchronise among themselves only
  const int ptid = rg * 32 + lane;
  constexpr int PT = 32 * T::RG;
  auto pair_sync = [&]() {
    if (T::RG == 1)
      __syncwarp();
    else
      asm volatile("bar.sync %0, %1;\n" ::"r"(1 + pr), "n"(PT) : "memory");
  };
  auto load_in = [&](const TransformTask& t, int m0) {
    double* in = tsm + (2 * pr) * T::MSZ;
    m0 += 2 * pr;
    if (HALF) {
#pragma unroll 1
      for (int j = 0; j < 2; ++j) {
        if (m0 + j >= nmat) break;
        int l, s;
        unpack_pair(m0 + j, &l, &s);
        const double* src = t.in + ((long long)l * n + s) * n2;
        double* dst = in + j * T::MSZ;
        if ((n & 1) == 0) {
          const int nh = n >> 1;
          for (int i = ptid; i < n * nh; i += PT) {
            const int r = i / nh, c = i % nh;
            cp16(dst + r * T::LD + 2 * c, src + 2 * i);
          }
        } else {
          for (int i = ptid; i < (int)n2; i += PT) cp8(dst + (i / n) * T::LD + i % n, src + i);
        }
      }
    } else {
      for (int u = ptid; u < npack; u += PT) {
        const uint32_t d = tab[u];
        const double* src = t.in + (long long)m0 * ldu + u;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          if (m0 + j < nmat) {
            cp8(in + j * T::MSZ + (d & 0xFFFF), src + (long long)j * ldu);
            cp8(in + j * T::MSZ + (d >> 16), src + (long long)j * ldu);
          }
        }
      }
    }
    cp_commit();
  };

  int task = (int)(it0 / ngroup);
  load_ab(tasks[task]);
  load_in(tasks[task], (int)(it0 % ngroup) * T::MATS);
  cp_wait_all();
  __syncthreads();
  const double* in0 = in + (2 * pr) * T::MSZ;
  const double* in1 = in0 + T::MSZ;
  for (long long it = it0; it < it1; ++it) {
    const int m0 = (int)(it % ngroup) * T::MATS;
    // first product: 16 rows of A^T In for both matrices
    double z[2][N8][4];
#pragma unroll
    for (int j = 0; j < N8; ++j)
#pragma unroll
      for (int h = 0; h < 4; ++h) z[0][j][h] = z[1][j][h] = 0.0;
#pragma unroll
    for (int k = 0; k < N8; ++k) {
      const int k0 = 8 * k + tig;
      double af[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) af[i] = as[(k0 + 4 * (i >> 1)) * T::LD + rg * 16 + grp + 8 * (i & 1)];
#pragma unroll
      for (int j = 0; j < N8; ++j) {
        const int o = k0 * T::LD + 8 * j + grp;
        dmma1688(z[0][j], af, in0[o], in0[o + 4 * T::LD]);
        dmma1688(z[1][j], af, in1[o], in1[o + 4 * T::LD]);
      }
    }
    pair_sync();  // the matrices are consumed: the next group's copies may start
    const bool more = it + 1 < it1;
    const int ntk = more ? (int)((it + 1) / ngroup) : task;
    if (more) load_in(tasks[ntk], (int)((it + 1) % ngroup) * T::MATS);
    // second product: the accumulators are A fragments (k slot tig <-> column 2 tig, tig + 4 <-> 2 tig + 1)
    const TransformTask t = tasks[task];
    const int ma = m0 + 2 * pr;
#pragma unroll 1
    for (int j0 = 0; j0 < N8; j0 += 2) {
      double acc[2][2][4];
#pragma unroll
      for (int g = 0; g < 2; ++g)
#pragma unroll
        for (int h = 0; h < 4; ++h) acc[0][g][h] = acc[1][g][h] = 0.0;
#pragma unroll
      for (int k = 0; k < N8; ++k) {
        const double a0[4] = {z[0][k][0], z[0][k][2], z[0][k][1], z[0][k][3]};
        const double a1[4] = {z[1][k][0], z[1][k][2], z[1][k][1], z[1][k][3]};
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          if (N8 % 2 == 0 || j0 + g < N8) {
            const double* b = bs + (8 * k + tig) * T::LD + 8 * (j0 + g) + grp;
            const double b0 = b[0], b1 = b[4 * T::LD];
            dmma1688(acc[0][g], a0, b0, b1);
            dmma1688(acc[1][g], a1, b0, b1);
          }
        }
      }
      // rows grp, grp + 8 of the warp's 16; columns 2 tig, 2 tig + 1 of each 8-column tile
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        const int q0 = 8 * (j0 + g) + 2 * tig;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int r = rg * 16 + grp + 8 * h;
          if (r >= n || q0 >= n || ma >= nmat) continue;
          const bool two = q0 + 1 < n;
          if (HALF) {
            // H[pq][u], u = ma and ma + 1 (ldu is even and ma is even: 16-byte stores)
            double* o = t.out + ((long long)r * n + q0) * ldu + ma;
            *reinterpret_cast<double2*>(o) = make_double2(acc[0][g][2 * h], acc[1][g][2 * h]);
            if (two) *reinterpret_cast<double2*>(o + ldu) = make_double2(acc[0][g][2 * h + 1], acc[1][g][2 * h + 1]);
          } else if (t.mode == kStore) {
#pragma unroll
            for (int m = 0; m < 2; ++m) {
              if (ma + m >= nmat) continue;
              double* o = t.out + (ma + m) * n2 + (long long)r * n + q0;
              if ((n & 1) == 0) {
                *reinterpret_cast<double2*>(o) = make_double2(acc[m][g][2 * h], acc[m][g][2 * h + 1]);
              } else {
                o[0] = acc[m][g][2 * h];
                if (two) o[1] = acc[m][g][2 * h + 1];
              }
            }
          } else {
            // J[a][b][c][d] -= value, matrix (a, c), row b, column d
#pragma unroll
            for (int m = 0; m < 2; ++m) {
              if (ma + m >= nmat) continue;
              const int a = (ma + m) / n, c = (ma + m) % n;
              double* o = t.out + (((long long)a * n + r) * n + c) * n + q0;
              o[0] -= acc[m][g][2 * h];
              if (two) o[1] -= acc[m][g][2 * h + 1];
            }
          }
        }
      }
    }
    if (more) {
      cp_wait_all();
      if (ntk != task) {
        __syncthreads();  // every warp has read the old A and B
        task = ntk;
        load_ab(tasks[task]);
        __syncthreads();
      } else {
        pair_sync();
      }
    }
  }
}

template <int N8, bool HALF>
cudaError_t launch_two_sided(cudaStream_t st, const TransformTask* tasks, int ntask, int n) {
  using T = TwoSided<N8>;
  const int npack = n * (n + 1) / 2, nmat = HALF ? npack : n * n;
  const size_t smem = T::smem(HALF ? 0 : npack);
  cudaError_t e = cudaFuncSetAttribute(two_sided_kernel<N8, HALF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const long long total = (long long)((nmat + T::MATS - 1) / T::MATS) * ntask;
  const int grid = (int)(total < 148 * T::BLOCKS ? total : 148 * T::BLOCKS);
  two_sided_kernel<N8, HALF><<<grid, T::THREADS, smem, st>>>(tasks, ntask, n, nmat, npack, (int)packed_ld(n));
  return cudaGetLastError();
}

// jas = T - T^T over (b, d) for every (a, c), in place: N[ab|cd] - N[ad|cb].  One block per (a, c);
// bound by memory, the tensor read and written once (n = 64: 268 MB).
__global__ void __launch_bounds__(256) antisymmetrise_kernel(double* const* __restrict__ tensors, int n) {
  extern __shared__ double tile[];
  const int ld = n | 1;
  const long long n2 = (long long)n * n;
  const int a = blockIdx.x / n, c = blockIdx.x % n;
  double* t = tensors[blockIdx.y] + (long long)a * n * n2 + (long long)c * n;   // + b n^2 + d
  for (int i = threadIdx.x; i < (int)n2; i += blockDim.x) tile[(i / n) * ld + i % n] = t[(i / n) * n2 + i % n];
  __syncthreads();
  for (int i = threadIdx.x; i < (int)n2; i += blockDim.x) {
    const int b = i / n, d = i % n;
    t[b * n2 + d] = tile[b * ld + d] - tile[d * ld + b];
  }
}

// Tensor of the reversed reference pair: out[a,b,c,d] = in[rho1(b), pi1(a), rho2(d), pi2(c)] with
// pi(r) = r + o mod n and rho(c) = c - o mod n (the row space of (w, x) is the column space of (x, w),
// rotated, and the other way round).  One block per (a, b): both tiles are contiguous.
__global__ void __launch_bounds__(256) mirror_kernel(const MirrorTask* __restrict__ tasks, int n) {
  extern __shared__ double tile[];
  const MirrorTask t = tasks[blockIdx.y];
  const int ld = n | 1;
  const long long n2 = (long long)n * n;
  const int a = blockIdx.x / n, b = blockIdx.x % n;
  const int i1 = (b + n - t.o1) % n, j1 = (a + t.o1) % n;
  const double* src = t.in + ((long long)i1 * n + j1) * n2;
  double* dst = t.out + ((long long)a * n + b) * n2;
  for (int i = threadIdx.x; i < (int)n2; i += blockDim.x) tile[(i / n) * ld + i % n] = src[i];
  __syncthreads();
  for (int i = threadIdx.x; i < (int)n2; i += blockDim.x) {
    const int c = i / n, d = i % n;
    int r = d - t.o2, k = c + t.o2;
    if (r < 0) r += n;
    if (k >= n) k -= n;
    dst[i] = tile[r * ld + k];
  }
}

// Largest |E| and largest violation of (mu nu|lam sig) = (mu nu|sig lam) = (lam sig|mu nu), as the bits
// of non-negative doubles (their order is the integers' order).
__global__ void __launch_bounds__(256) eri_symmetry_kernel(const double* __restrict__ eri, int n,
                                                           unsigned long long* __restrict__ out) {
  __shared__ double tile[32][33];
  const int n2 = n * n;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  double big = 0.0, off = 0.0;
  const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
  for (int k = ty; k < 32; k += 8)
    tile[k][tx] = (c0 + k < n2 && r0 + tx < n2) ? eri[(long long)(c0 + k) * n2 + r0 + tx] : 0.0;
  __syncthreads();
  for (int k = ty; k < 32; k += 8) {
    const int r = r0 + k, c = c0 + tx;
    if (r >= n2 || c >= n2) continue;
    const double v = eri[(long long)r * n2 + c];
    const double w = eri[(long long)r * n2 + (long long)(c % n) * n + c / n];
    big = fmax(big, fabs(v));
    off = fmax(off, fmax(fabs(v - w), fabs(v - tile[tx][k])));
  }
  for (int d = 16; d > 0; d >>= 1) {
    big = fmax(big, __shfl_xor_sync(0xFFFFFFFFu, big, d));
    off = fmax(off, __shfl_xor_sync(0xFFFFFFFFu, off, d));
  }
  if (tx == 0) {
    atomicMax(out, (unsigned long long)__double_as_longlong(big));
    atomicMax(out + 1, (unsigned long long)__double_as_longlong(off));
  }
}

}  // namespace

#define NW_TWO_SIDED(K)                                                    \
  case K:                                                                  \
    return half ? launch_two_sided<K, true>(st, tasks, ntask, n)           \
                : launch_two_sided<K, false>(st, tasks, ntask, n);

cudaError_t two_sided(cudaStream_t st, bool half, const TransformTask* tasks, int ntask, int n) {
  if (ntask <= 0) return cudaSuccess;
  switch ((n + 7) / 8) {
    NW_TWO_SIDED(1)
    NW_TWO_SIDED(2)
    NW_TWO_SIDED(3)
    NW_TWO_SIDED(4)
    NW_TWO_SIDED(5)
    NW_TWO_SIDED(6)
    NW_TWO_SIDED(7)
    NW_TWO_SIDED(8)
  }
  return cudaErrorInvalidValue;
}
#undef NW_TWO_SIDED

cudaError_t antisymmetrise(cudaStream_t st, double* const* tensors, int count, int n) {
  if (count <= 0) return cudaSuccess;
  antisymmetrise_kernel<<<dim3(n * n, count), 256, sizeof(double) * n * (n | 1), st>>>(tensors, n);
  return cudaGetLastError();
}

cudaError_t mirror_tensors(cudaStream_t st, const MirrorTask* tasks, int count, int n) {
  if (count <= 0) return cudaSuccess;
  mirror_kernel<<<dim3(n * n, count), 256, sizeof(double) * n * (n | 1), st>>>(tasks, n);
  return cudaGetLastError();
}

cudaError_t eri_symmetry(cudaStream_t st, const double* eri, int n, double* scratch2, double* big, double* off) {
  cudaError_t e = cudaMemsetAsync(scratch2, 0, 2 * sizeof(double), st);
  if (e != cudaSuccess) return e;
  const unsigned t = (unsigned)((n * n + 31) / 32);
  eri_symmetry_kernel<<<dim3(t, t), 256, 0, st>>>(eri, n, reinterpret_cast<unsigned long long*>(scratch2));
  double h[2];
  e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(h, scratch2, sizeof(h), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  *big = h[0];
  *off = h[1];
  return e;
}

}  // namespace nw
