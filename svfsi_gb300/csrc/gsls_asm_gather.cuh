// Assembly through an element buffer: one launch over all elements writes
// their matrices and residuals, then every CSR block and every node adds its
// contributions in element order (DOASSEM, Code/Source/svFSI/LHSA.f:266-298,
// from the other side).  Included by gsls_assemble.cu.
//
// The colour launches that scatter into the matrix are a chain of ~30 launches
// of a few hundred blocks each: the element work after a colour's wait runs
// with one or two warps per scheduler, every thread waits for its 16 loads of
// the matrix one after the other, and each colour touches the whole matrix
// (6.3 GB of DRAM traffic for a 188 MB matrix on the neo-Hookean beam).  The
// buffer is written and read once, in whole sectors.  The elements are stored
// in colour order, so a block's sum takes the colours' order: the same sum.
// A buffer above kElemBuf is filled and added in parts; the map is one list per
// window of kInvEl elements, so that its entries fit in 31 bits.
#pragma once

namespace gsls {

constexpr size_t kElemBuf = (size_t)4 << 30;
constexpr int kInvEl = 1 << 26;

// One warp's rows of N values per lane, staged in shared memory so that the
// rows leave in whole 16-byte vectors, each row contiguous.  PAD: an odd
// number of vectors per lane keeps the staging free of bank conflicts.
template <class T, int N>
struct EmitRow {
  static constexpr int NV = N * (int)sizeof(T) / 16, PAD = NV | 1;
  static constexpr int kBytes = 32 * PAD * 16;  // per warp
  static_assert(N * sizeof(T) % 16 == 0, "whole vectors");
  // lane l's row goes to dst + l * stride; rows of lanes >= n are dropped
  static __device__ __forceinline__ void out(const T *row, unsigned char *buf, unsigned char *dst,
                                             size_t stride, int n) {
    const int lane = threadIdx.x & 31;
    uint4 *b = reinterpret_cast<uint4 *>(buf);
#pragma unroll
    for (int q = 0; q < NV; q++) b[lane * PAD + q] = reinterpret_cast<const uint4 *>(row)[q];
    __syncwarp();
#pragma unroll 4
    for (int t = lane; t < n * NV; t += 32) {
      const int el = t / NV, q = t - el * NV;
      reinterpret_cast<uint4 *>(dst + (size_t)el * stride)[q] = b[el * PAD + q];
    }
    __syncwarp();
  }
};

// this warp's part of the element buffer
struct EmitAt {
  unsigned char *buf;  // staging
  unsigned char *lK;   // first element's matrix, 16 blocks of DD values
  double *lR;          // first element's residual, 4 x dof
  int n;               // elements of this warp
};
__device__ __forceinline__ EmitAt emit_at(const AsmArgs &A, unsigned char *smem, int bytes,
                                          size_t kbytes, int dof) {
  const int w = threadIdx.x >> 5, t0 = blockIdx.x * blockDim.x + w * 32;
  EmitAt E;
  E.buf = smem + (size_t)w * bytes;
  E.lK = reinterpret_cast<unsigned char *>(A.lK) + (size_t)t0 * kbytes;
  E.lR = A.lR + (size_t)t0 * 4 * dof;
  E.n = max(0, min(32, A.nColorEl - t0));
  return E;
}
template <class VT, int DOF>
constexpr int emit_bytes() {
  return EmitRow<VT, 4 * DOF * DOF>::kBytes > EmitRow<double, 4 * DOF>::kBytes
             ? EmitRow<VT, 4 * DOF * DOF>::kBytes
             : EmitRow<double, 4 * DOF>::kBytes;
}
template <int DOF>
__device__ __forceinline__ void emit_res(const EmitAt &E, const double *lR) {
  EmitRow<double, 4 * DOF>::out(lR, E.buf, reinterpret_cast<unsigned char *>(E.lR),
                                sizeof(double) * 4 * DOF, E.n);
}
// the four blocks (a, 0..3)
template <class VT, int DOF>
__device__ __forceinline__ void emit_row(const EmitAt &E, int a, const VT *row) {
  constexpr int N = 4 * DOF * DOF;
  EmitRow<VT, N>::out(row, E.buf, E.lK + (size_t)a * N * sizeof(VT), sizeof(VT) * 4 * N, E.n);
}

// ---- the inverse of the element -> CSR map: ent[ptr[p] .. ptr[p+1]) = 16 e + 4
// a + b of the element blocks that CSR block p receives, ascending
__global__ void k_inv_count(size_t n, const int *__restrict__ map, int *__restrict__ cnt) {
  for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n;
       k += (size_t)gridDim.x * blockDim.x)
    atomicAdd(cnt + map[k], 1);
}
// exclusive scan in three launches: sums of chunks of kScan, of the chunk
// sums (one block), and within the chunks
constexpr int kScan = 2048;
__global__ void __launch_bounds__(256) k_scan_sums(int n, const int *__restrict__ cnt,
                                                   int *__restrict__ sums) {
  __shared__ int sh[32];
  int s = 0, tot;
  for (int k = threadIdx.x; k < kScan; k += 256) {
    const int i = blockIdx.x * kScan + k;
    if (i < n) s += cnt[i];
  }
  block_scan_excl(s, sh, tot);
  if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}
__global__ void __launch_bounds__(1024) k_scan_top(int n, int *sums) {
  __shared__ int sh[32];
  int run = 0;
  for (int k0 = 0; k0 < n; k0 += 1024) {
    const int k = k0 + threadIdx.x;
    int tot;
    const int ex = block_scan_excl(k < n ? sums[k] : 0, sh, tot);
    if (k < n) sums[k] = run + ex;
    run += tot;
    __syncthreads();
  }
}
__global__ void __launch_bounds__(256) k_scan_fill(int n, const int *__restrict__ cnt,
                                                   const int *__restrict__ sums,
                                                   int *__restrict__ ptr, int total) {
  __shared__ int sh[32];
  int run = sums[blockIdx.x];
  for (int k0 = 0; k0 < kScan; k0 += 256) {
    const int i = blockIdx.x * kScan + k0 + threadIdx.x;
    int tot;
    const int ex = block_scan_excl(i < n ? cnt[i] : 0, sh, tot);
    if (i < n) ptr[i] = run + ex;
    run += tot;
    __syncthreads();
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) ptr[n] = total;
}
// cnt counts down: the slots of a list in any order, sorted afterwards
__global__ void k_inv_fill(size_t n, const int *__restrict__ map, const int *__restrict__ ptr,
                           int *__restrict__ cnt, int *__restrict__ ent) {
  for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n;
       k += (size_t)gridDim.x * blockDim.x)
    ent[ptr[map[k]] + atomicSub(cnt + map[k], 1) - 1] = (int)k;
}
__global__ void k_inv_sort(int nnz, const int *__restrict__ ptr, int *__restrict__ ent) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < nnz; p += gridDim.x * blockDim.x) {
    const int b = ptr[p], e = ptr[p + 1];
    for (int i = b + 1; i < e; i++) {
      const int v = ent[i];
      int j = i - 1;
      for (; j >= b && ent[j] > v; j--) ent[j + 1] = ent[j];
      ent[j + 1] = v;
    }
  }
}

// Values per thread.  The index work is done once per thread: with one value
// each, 3x3 blocks in FP32 took 270 M warp instructions (342 us for 1,022,208
// tets), and a row each is faster (neo-Hookean beam, FP32: assembly 1.85 -> 1.67
// ms).  Of 4x4 blocks in FP64, which are whole sectors, two values each are
// slower (VMS fluid, 371,520 tets: 1.38 -> 1.49 ms; 48 registers and half the
// loads in flight).
template <int DD, class VT>
constexpr int gather_width() {
  return DD == 9 && sizeof(VT) == 4 ? 3 : 1;
}
// Val[p] = sum of the element blocks e0 <= e < e1 of its list (added to Val
// unless first), V values per thread, four blocks in flight; PART: the list may
// hold elements outside e0 .. e1.  Bound by the sectors of the scattered blocks.
template <int DD, class VT, bool PART>
__global__ void __launch_bounds__(256) k_gather_val(size_t n, const int *__restrict__ ptr,
                                                    const int *__restrict__ ent,
                                                    const VT *__restrict__ lK, int e0, int e1,
                                                    int first, VT *__restrict__ Val) {
  constexpr int V = gather_width<DD, VT>(), T = DD / V;
  for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n;
       k += (size_t)gridDim.x * blockDim.x) {
    const size_t p = k / T;
    const int c = (int)(k - p * T) * V;
    const int b = __ldg(ptr + p), e = __ldg(ptr + p + 1);
    VT *__restrict__ out = Val + p * DD + c;
    VT s[V];
#pragma unroll
    for (int q = 0; q < V; q++) s[q] = first ? VT(0) : out[q];
    const VT *__restrict__ src = lK + c - (size_t)e0 * 16 * DD;
    for (int i = b; i < e; i += 4) {
      int id[4];
      VT v[4][V];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        id[u] = i + u < e ? __ldg(ent + i + u) : -1;
        if (PART && id[u] >= 0 && ((id[u] >> 4) < e0 || (id[u] >> 4) >= e1)) id[u] = -1;
      }
#pragma unroll
      for (int u = 0; u < 4; u++) {
        if (id[u] >= 0) {
          const VT *__restrict__ w = src + (size_t)id[u] * DD;
#pragma unroll
          for (int q = 0; q < V; q++) v[u][q] = __ldcs(w + q);
        }
      }
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (id[u] >= 0)
#pragma unroll
          for (int q = 0; q < V; q++) s[q] += v[u][q];
    }
#pragma unroll
    for (int q = 0; q < V; q++) out[q] = s[q];
  }
}
// Residual values of an element in the buffer: 4 per degree of freedom; a scalar
// element's are not weighted yet, its weight is the fifth of 6
template <int DOF>
constexpr int kResRow = DOF == 1 ? 6 : 4 * DOF;

// R of a node from the list of its diagonal block, whose entries are (e, a, a)
template <int DOF>
__global__ void __launch_bounds__(256) k_gather_res(int nNo, const int *__restrict__ diagPtr,
                                                    const int *__restrict__ ptr,
                                                    const int *__restrict__ ent,
                                                    const double *__restrict__ lR, int e0, int e1,
                                                    int first, double *__restrict__ R) {
  const size_t n = (size_t)nNo * DOF;
  for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n;
       k += (size_t)gridDim.x * blockDim.x) {
    const size_t i = k / DOF;
    const int c = (int)(k - i * DOF), p = __ldg(diagPtr + i);
    const int b = __ldg(ptr + p), e = __ldg(ptr + p + 1);
    double s = first ? 0.0 : R[k];
    for (int q = b; q < e; q += 4) {
      int id[4];
      double v[4], w[4] = {};
#pragma unroll
      for (int u = 0; u < 4; u++) {
        id[u] = q + u < e ? __ldg(ent + q + u) : -1;
        if (id[u] >= 0 && ((id[u] >> 4) < e0 || (id[u] >> 4) >= e1)) id[u] = -1;
      }
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const double *__restrict__ r =
            lR + (size_t)((id[u] >= 0 ? id[u] >> 4 : e0) - e0) * kResRow<DOF>;
        v[u] = id[u] >= 0 ? __ldcs(r + (id[u] & 3) * DOF + c) : 0.0;
        if constexpr (DOF == 1) w[u] = id[u] >= 0 ? __ldcs(r + 4) : 0.0;
      }
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (id[u] >= 0) s = DOF == 1 ? fma(w[u], v[u], s) : s + v[u];
    }
    R[k] = s;
  }
}

}  // namespace gsls
