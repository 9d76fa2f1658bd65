// Row partition of the matrix over the thread blocks of a persistent Krylov
// kernel (one block per SM), with the matrix in a per-warp stream layout.
//
// Block b owns a compact set of rows.  Every vector entry that its rows
// multiply is either its own or in its halo list, so a block that keeps both
// in shared memory (its window) reads no vector entry from L2 inside the
// product: one coalesced pass over the halo replaces ~15 scattered gathers
// per row.  Columns become 16-bit window indices.
//
// Order: a block's rows, sorted by decreasing length, fill slices of
// RW = 32/L rows; lane g*L + l of a slice's warp takes the blocks l, l+L, ...
// of row g.  Vectors of the kernel live in this slot order (slot = slice*RW +
// g over all blocks; empty slots hold zeros).  Slice s of a block belongs to
// warp s % kPartWarps, and a warp's steps are those of its slices one after another.
#pragma once

#include "gsls_internal.cuh"

namespace gsls {

// Warps per block: FP64 instructions issue at one per ~64 cycles and
// scheduler whatever the number of warps, and each warp pays for its own
// share of every reduction; in FP32, 16 warps of 128 registers spill and were
// 12 % slower on the beam than 8 (122 against 107 ms a step).
constexpr int kPartWarps = 8;
constexpr int kPartThreads = 32 * kPartWarps;
constexpr int kPartMaxBlocks = 256;

struct PartArgs {
  const int *wbase;   // first step of each (block, warp), nblk * kPartWarps + 1
  const int *sst;     // first step of each slice
  const int *soff;    // the same with every slice starting at a multiple of 8
  const int *sbase;   // first slice of each block, nblk + 1
  const int *slen;    // steps of each slice (>= 1)
  const int *hoff;    // halo offsets, nblk + 1
  const int *halo;    // halo entries: slots of other blocks
  const int *slotRow; // row of each slot or -1
  const int *src;     // CSR block of each (step, lane) or -1
  const unsigned short *lcol;  // window index of each (step, lane)
  int nblk, L;
  int winMax, nslMax, stMax;  // largest window, slices of a block, steps of a warp
  int nS, grpMax;             // all slices; groups of 8 steps of a warp
  long long nslots, nsteps, nsteps8;  // slots; steps, and those of soff
};

// Partitions of the lhs over at most num_sms() blocks, each once per lhs: [0] of
// the rows as the mesh numbers them, [1] in an order of the graph's own, for a
// kernel whose windows do not fit in [0] of a mesh with scattered numbers.  part_setup orders the rows and sizes
// the windows, part_fill makes the tables of the halos and steps for a caller
// whose windows fit.  ok is false when a window has more than 65,535 entries or
// there is no memory for the tables: the callers then have kernels without them.
int part_setup(gsls_lhs *lhs, bool graph);
int part_fill(gsls_lhs *lhs, RowPart &p);
// The first of the two on which `fits` is true, its tables filled; *p null when
// there is none.
//
// The windows of a scattered numbering are several times as wide as those of a
// mesh numbered plane by plane; the order of the graph makes them as narrow
// (358,425 nodes at random: 31,063 -> 3,982 entries) for a search of 0.1 s on the
// host, once.  Where the windows of [0] fit, an iteration on them is at most
// 1.6 times as long as on a mesh numbered plane by plane, and they are taken.
template <class Fits>
int part_for(gsls_lhs *lhs, RowPart **p, const Fits &fits) {
  *p = nullptr;
  for (int k = 0; k < 2; k++) {
    RowPart &q = lhs->ws.part[k];
    if (k == 1 && !lhs->ws.part[0].scattered) break;
    GSLS_TRY(part_setup(lhs, k == 1));
    if (!q.ok) continue;
    if (!fits(q)) {
      q.tmp.release();
      continue;
    }
    GSLS_TRY(part_fill(lhs, q));
    if (!q.ok) continue;
    *p = &q;
    return GSLS_OK;
  }
  return GSLS_OK;
}
PartArgs part_args(const RowPart &p);
// least rows of the largest block: where these alone do not fit, nothing is built
inline long long part_rows(const gsls_lhs *lhs) {
  const long long nblk = num_sms() < kPartMaxBlocks ? num_sms() : kPartMaxBlocks;
  return (lhs->nNo + nblk - 1) / nblk;
}

// Most dynamic shared memory of a block of the kernel on this device
inline size_t smem_cap(const void *kernel) {
  int dev = 0, opt = 0;
  cudaFuncAttributes fa{};
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&opt, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (cudaFuncGetAttributes(&fa, kernel) != cudaSuccess) return 0;
  return (size_t)opt - fa.sharedSizeBytes;
}

// Cooperative launch with smem bytes of dynamic shared memory.  The attribute
// that allows them belongs to the kernel, not to the launch: it is always set
// to the same value, the most there is (cap), so that of two host threads with
// systems of different size neither lowers it between the other's two calls.
inline int coop_launch(const void *kernel, size_t cap, int nblk, void **args, size_t smem,
                       cudaStream_t st) {
  GSLS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap));
  GSLS_CUDA(cudaLaunchCooperativeKernel(kernel, dim3(nblk), dim3(kPartThreads), args, smem, st));
  return GSLS_OK;
}

// A node's D values in global memory, read and written through L2; stride VD
// (3-vectors are padded to 4 values: whole 16-byte accesses)
template <int D, class XT>
struct NodeL2 {
  static constexpr int VD = D == 3 ? 4 : D;
  static __device__ __forceinline__ void ld(const XT *p, XT o[D]) {
    if constexpr (sizeof(XT) == 4) {
      if constexpr (D == 1) {
        o[0] = __ldcg(p);
      } else if constexpr (D == 2) {
        const float2 v = __ldcg(reinterpret_cast<const float2 *>(p));
        o[0] = v.x;
        o[1] = v.y;
      } else {
        const float4 v = __ldcg(reinterpret_cast<const float4 *>(p));
        o[0] = v.x;
        o[1] = v.y;
        o[2] = v.z;
        if constexpr (D == 4) o[3] = v.w;
      }
    } else {
      if constexpr (D == 1) {
        o[0] = __ldcg(p);
      } else {
        const double2 v = __ldcg(reinterpret_cast<const double2 *>(p));
        o[0] = v.x;
        o[1] = v.y;
        if constexpr (D > 2) {
          const double2 u = __ldcg(reinterpret_cast<const double2 *>(p) + 1);
          o[2] = u.x;
          if constexpr (D == 4) o[3] = u.y;
        }
      }
    }
  }
  static __device__ __forceinline__ void st(XT *p, const XT o[D]) {
    if constexpr (sizeof(XT) == 4) {
      if constexpr (D == 1)
        __stcg(p, o[0]);
      else if constexpr (D == 2)
        __stcg(reinterpret_cast<float2 *>(p), make_float2(o[0], o[1]));
      else
        __stcg(reinterpret_cast<float4 *>(p), make_float4(o[0], o[1], o[2], D == 4 ? o[D - 1] : 0.f));
    } else {
      if constexpr (D == 1) {
        __stcg(p, o[0]);
      } else {
        __stcg(reinterpret_cast<double2 *>(p), make_double2(o[0], o[1]));
        if constexpr (D > 2)
          __stcg(reinterpret_cast<double2 *>(p) + 1, make_double2(o[2], D == 4 ? o[D - 1] : 0.0));
      }
    }
  }
};

// use(k, load(k)) for the nodes k of this thread, B loads in flight
template <int D, class XT>
constexpr int kB = sizeof(XT) == 4 ? 6 : D > 2 ? 3 : 5;
template <int B, int D, class XT, class Ld, class Use>
__device__ __forceinline__ void for_nodes(int n, const Ld &load, const Use &use) {
#pragma unroll 1
  for (int k0 = threadIdx.x; k0 < n; k0 += B * kPartThreads) {
    XT v[B][D];
#pragma unroll
    for (int u = 0; u < B; u++)
      if (k0 + u * kPartThreads < n) load(k0 + u * kPartThreads, v[u]);
#pragma unroll
    for (int u = 0; u < B; u++)
      if (k0 + u * kPartThreads < n) use(k0 + u * kPartThreads, v[u]);
  }
}

// Groups of G (at most 8) steps that never hold steps of two slices, as a
// table of each warp in shared memory: the group's first
// step (soff) relative to the block's, the steps of it that belong to the
// slice, and whether it is the slice's first or last.  Written by the warp's lane 0
// (table of at least nslMax / kPartWarps + 1 + grpMax * 8 / G entries); the
// number of groups on every lane.
constexpr int kGrpOff = (1 << 20) - 1, kGrpLast = 1 << 24, kGrpFirst = 1 << 25;
__device__ __forceinline__ int grp_valid(int e) { return (e >> 20) & 15; }
__host__ __device__ __forceinline__ int grp_cap(int nslMax, int grpMax, int G) {
  return nslMax / kPartWarps + 1 + grpMax * (8 / G);
}
template <int G>
static __device__ __noinline__ int part_groups(const int *__restrict__ soff,
                                               const int *__restrict__ slen, int nsl, int w,
                                               int *tab) {
  int n = 0;
  if ((threadIdx.x & 31) == 0)
    for (int s = w; s < nsl; s += kPartWarps) {
      const int len = __ldg(slen + s), at = __ldg(soff + s) - __ldg(soff);
      for (int t = 0; t < len; t += G)
        tab[n++] = (at + t) | min(G, len - t) << 20 | (t + G >= len ? kGrpLast : 0) |
                   (t == 0 ? kGrpFirst : 0);
    }
  __syncwarp();
  return __shfl_sync(0xffffffffu, n, 0);
}

}  // namespace gsls
