// CG (CGRADS/CGRADV, Code/Source/svFSILS/CGRAD.f:125-242) as one cooperative
// launch per solve on the row partition of gsls_part.cuh.
//
// A block keeps the direction P of its window (own rows and halo) in shared
// memory and reads its share of the matrix as one sequential stream per warp,
// the next group of steps always in flight in registers, so the product
// touches L2/HBM only for the matrix itself, in order and in whole 16-byte
// vectors.  Iteration k:
//  1. KP = K P of the own rows from the window; block partials of P.KP;
//  2. grid sum (gsls_gridbar.cuh): alpha; R -= alpha KP for the own rows, R
//     published; partials of |R|^2; X += alpha P while they travel;
//  3. grid sum: err, beta, CGRAD's stopping tests; P = R + beta P for the
//     own rows and, from the published R, for the halo: every block forms
//     the same P entries as their owners, so P itself never travels.
// Odd iterations walk the stream from the end: what L2 (or, for a small
// share, L1) still holds of the matrix is met first.
//
// Measured (GB300): the FP32 solves of the neo-Hookean beam (358,425 nodes,
// 3x3 blocks, 188 MB of matrix) take 36 us per iteration against 74 us for
// the three batched kernels (an iteration reads 134 MB from DRAM, 20 us at
// the measured copy rate; the rest is L2 and two grid sums of ~3.5 us); the
// FP64 3x3 solves of 15,616 nodes 13 us against 21 us (FP64 pipe 5 us); the
// 20^3 heat cube 8 us against 12 us per iteration (two grid sums).
//
// Staging the stream in shared memory by bulk copies (a ring per warp with an
// mbarrier per slot, or one ring per block with a producer warp) was slower:
// with ~100 KB left for the ring a warp waits for, releases and addresses a
// chunk every one or two steps, 120-160 instructions per step of 22 loads
// and FMAs (beam: 84,000-119,000 cycles a product).
#include <algorithm>

#include "gsls_gridbar.cuh"
#include "gsls_part.cuh"
#include "gsls_spmv.cuh"

namespace gsls {

static_assert(sizeof(GridRedBuf) + kScalRed <= kScalBytes, "scalar buffer");

template <class XT>
struct WcgArgs {
  PartArgs P;
  const unsigned char *stream;
  double *R;          // in: right-hand side (row order), out: W X
  const double *W;
  XT *Xg, *Rg;        // slot order; Xg unused when x_smem
  KrylovScalars *S;
  double absTol, relTol;
  int mItr;
  GridRed red;
  int r_smem, x_smem, ownMax, ahead;
};

// The stream: a warp's steps in groups of G, per group and lane G window
// columns (16 bits) and G blocks (row-major) as NV 16-byte vectors; vector q
// of the 32 lanes side by side.  Groups cross the ends of slices; the last
// group of a warp is padded with zero blocks.
template <int D, class VT>
struct Rec {
  static constexpr int DD = D * D;
  static constexpr int G = sizeof(VT) == 4 ? (D == 1 ? 8 : D == 4 ? 2 : 4) : D == 1 ? 4 : D == 4 ? 1 : 2;
  static constexpr int N16 = 16 / (int)sizeof(VT);  // values per vector
  static constexpr int NV = G * DD / N16;
  // groups in flight behind the current one
  static constexpr int PD = D == 1 ? (sizeof(VT) == 4 ? 4 : 2) : 1;
  static constexpr int SB = 64 + DD * 32 * (int)sizeof(VT);  // bytes per step
  static_assert(G * DD % N16 == 0, "whole vectors");
  // first byte of the stream of warp bw (of all blocks), whose partition
  // steps start at `first`: every warp's stream is padded by up to G - 1 steps
  static __host__ __device__ __forceinline__ size_t at(long long first, int bw) {
    return (size_t)(first + (long long)bw * (G - 1)) * SB;
  }
};
template <int D, class VT>
struct Group {
  using R = Rec<D, VT>;
  VT a[R::G * R::DD];
  unsigned short c[R::G];
  __device__ __forceinline__ void load(const unsigned char *g, int lane) {
    if constexpr (R::G == 8) {
      *reinterpret_cast<uint4 *>(c) = __ldg(reinterpret_cast<const uint4 *>(g) + lane);
    } else if constexpr (R::G == 4) {
      *reinterpret_cast<uint2 *>(c) = __ldg(reinterpret_cast<const uint2 *>(g) + lane);
    } else if constexpr (R::G == 2) {
      *reinterpret_cast<unsigned *>(c) = __ldg(reinterpret_cast<const unsigned *>(g) + lane);
    } else {
      c[0] = __ldg(reinterpret_cast<const unsigned short *>(g) + lane);
    }
#pragma unroll
    for (int q = 0; q < R::NV; q++) {
      const uint4 v = __ldg(reinterpret_cast<const uint4 *>(g + 64 * R::G + q * 512) + lane);
      *reinterpret_cast<uint4 *>(a + q * R::N16) = v;
    }
  }
};

// stream of every warp from the CSR; a warp packs up to 8 consecutive steps,
// so that the blocks a lane reads one after the other are neighbours
template <int D, class VT>
__global__ void __launch_bounds__(256) k_wcg_pack(PartArgs P, const VT *__restrict__ Val,
                                                  unsigned char *__restrict__ stream, int per) {
  using R = Rec<D, VT>;
  constexpr int NG = 8 / R::G;  // groups a turn
  const int lane = threadIdx.x & 31;
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long t = warp; t < (long long)P.nblk * kPartWarps * per; t += nw) {
    const int bw = (int)(t / per), t0 = (int)(t % per) * 8;
    const int first = __ldg(P.wbase + bw), n = __ldg(P.wbase + bw + 1) - first;
#pragma unroll
    for (int i = 0; i < NG; i++) {
      const int g0 = t0 + i * R::G;
      if (g0 >= n) break;
      unsigned char *g = stream + R::at(first, bw) + (size_t)g0 * R::SB;
      __align__(16) VT a[R::G * R::DD];
      __align__(16) unsigned short c[R::G];
#pragma unroll
      for (int u = 0; u < R::G; u++) {
        const size_t e = (size_t)(first + g0 + u) * 32 + lane;
        const int j = g0 + u < n ? __ldg(P.src + e) : -1;
        c[u] = g0 + u < n ? __ldg(P.lcol + e) : 0;
#pragma unroll
        for (int k = 0; k < R::DD; k++)
          a[u * R::DD + k] = j >= 0 ? __ldg(Val + (size_t)j * R::DD + k) : VT(0);
      }
#pragma unroll
      for (int u = 0; u < R::G; u++)
        reinterpret_cast<unsigned short *>(g)[lane * R::G + u] = c[u];
#pragma unroll
      for (int q = 0; q < R::NV; q++)
        reinterpret_cast<uint4 *>(g + 64 * R::G + q * 512)[lane] =
            *reinterpret_cast<const uint4 *>(a + q * R::N16);
    }
  }
}

// what warp 0 shares after a grid sum
template <class XT>
struct WcgScal {
  double err, errO, alpha, beta, eps;
  XT a;  // alpha or beta in the vector type
  int done, suc, itr, ok;
};

__device__ __forceinline__ void prefetch_l2(const unsigned char *p, unsigned bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// One pass of a warp over its stream, in direction REV: KP of its rows from
// the window, and the sum of P.KP.
template <bool REV, int W, int D, class VT, class XT, class AT>
__device__ __noinline__ AT wcg_pass(const unsigned char *__restrict__ stream, int ng,
                                       int nst, int nq, int w, int lane, int L, int ahead,
                                       const int *slen, const XT *win, XT *KP) {
  using R = Rec<D, VT>;
  const int RW = 32 / L;
  int q = REV ? nq - 1 : 0, s = w + q * W;
  // steps until the slice's end; a pass from the end starts with the padding
  int left = slen[s] + (REV ? ng * R::G - nst : 0);
  AT acc[D], dot = AT(0);
#pragma unroll
  for (int d = 0; d < D; d++) acc[d] = AT(0);
  const auto group = [&](int i) {
    return stream + (size_t)(REV ? ng - 1 - i : i) * (R::G * R::SB);
  };
  Group<D, VT> grp[R::PD + 1];
#pragma unroll
  for (int k = 0; k < R::PD; k++)
    if (k < ng) grp[k].load(group(k), lane);
#pragma unroll 1
  for (int i = 0; i < ng; i++) {
    if (i + R::PD < ng) grp[R::PD].load(group(i + R::PD), lane);
    const Group<D, VT> &cur = grp[0];
    if (ahead && i + ahead < ng && lane == 0)
      prefetch_l2(group(i + ahead), R::G * R::SB);
    // every step's entries before the first sum: the branch at the end of a
    // slice would otherwise expose the latency of each
    XT x[R::G][D];
#pragma unroll
    for (int u = 0; u < R::G; u++)
#pragma unroll
      for (int d = 0; d < D; d++) x[u][d] = win[cur.c[u] * D + d];
    if (left > R::G) {
      // no slice ends in this group
      left -= R::G;
#pragma unroll
      for (int v = 0; v < R::G; v++) {
        const int u = REV ? R::G - 1 - v : v;
#pragma unroll
        for (int d = 0; d < D; d++)
#pragma unroll
          for (int r = 0; r < D; r++)
            acc[r] = fma(AT(cur.a[u * R::DD + r * D + d]), AT(x[u][d]), acc[r]);
      }
    } else {
#pragma unroll
      for (int v = 0; v < R::G; v++) {
        const int u = REV ? R::G - 1 - v : v;
#pragma unroll
        for (int d = 0; d < D; d++)
#pragma unroll
          for (int r = 0; r < D; r++)
            acc[r] = fma(AT(cur.a[u * R::DD + r * D + d]), AT(x[u][d]), acc[r]);
        if (--left == 0) {
          // end of a slice: add the lanes of a row, store, next slice (none:
          // the padding at the end of the stream has no end of its own)
#pragma unroll 1
          for (int o = 1; o < L; o <<= 1)
#pragma unroll
            for (int d = 0; d < D; d++) acc[d] += __shfl_xor_sync(0xffffffffu, acc[d], o);
          if ((lane & (L - 1)) == 0) {
            const int k = (s * RW + lane / L) * D;
#pragma unroll
            for (int d = 0; d < D; d++) {
              KP[k + d] = XT(acc[d]);
              dot = fma(AT(win[k + d]), acc[d], dot);
            }
          }
#pragma unroll
          for (int d = 0; d < D; d++) acc[d] = AT(0);
          q += REV ? -1 : 1;
          s += REV ? -W : W;
          left = q >= 0 && q < nq ? slen[s] : 0x7fffffff;
        }
      }
    }
#pragma unroll
    for (int k = 0; k < R::PD; k++) grp[k] = grp[k + 1];
  }
  return dot;
}

template <int D, class VT, class XT>
__global__ void __launch_bounds__(kPartThreads, 1) k_wcg(WcgArgs<XT> A) {
  using AT = typename AccOf<VT>::T;
  using N = NodeL2<D, XT>;
  constexpr int VD = N::VD;
  extern __shared__ __align__(16) unsigned char smem[];
  const PartArgs &P = A.P;
  const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  constexpr int W = kPartWarps, NT = kPartThreads;
  const int L = P.L, RW = 32 / L;
  const int s0 = P.sbase[b], nsl = P.sbase[b + 1] - s0;
  const int own = nsl * RW, nhalo = P.hoff[b + 1] - P.hoff[b];
  const int *__restrict__ halo = P.halo + P.hoff[b];
  const size_t g0 = (size_t)s0 * RW;

  // shared memory: window | KP | slice lengths | (R, X)
  XT *win = reinterpret_cast<XT *>(smem);
  size_t off = ((size_t)P.winMax * D * sizeof(XT) + 15) & ~(size_t)15;
  XT *KP = reinterpret_cast<XT *>(smem + off);
  off += ((size_t)A.ownMax * D * sizeof(XT) + 15) & ~(size_t)15;
  int *slen = reinterpret_cast<int *>(smem + off);
  off += ((size_t)P.nslMax * sizeof(int) + 15) & ~(size_t)15;
  XT *Rs = reinterpret_cast<XT *>(smem + off), *Xs = Rs + (size_t)A.ownMax * D;
  XT *Xg = A.Xg + g0 * VD, *Rg = A.Rg + g0 * VD;
  __shared__ WcgScal<XT> sc;

  // this warp's stream: nst steps in ng groups, nq slices
  using Rc = Rec<D, VT>;
  const int first = P.wbase[b * W + w], nst = P.wbase[b * W + w + 1] - first;
  const int ng = (nst + Rc::G - 1) / Rc::G, nq = w < nsl ? (nsl - 1 - w) / W + 1 : 0;
  const unsigned char *__restrict__ stream = A.stream + Rc::at(first, b * W + w);

  // R_k = R, X = 0, |R|
  double acc0 = 0.0;
  for (int k = tid; k < own; k += NT) {
    const int row = __ldg(P.slotRow + g0 + k);
    XT rx[D], z[D];
#pragma unroll
    for (int d = 0; d < D; d++) {
      const double r = row >= 0 ? A.R[(size_t)row * D + d] : 0.0;
      acc0 += r * r;
      rx[d] = XT(r);
      z[d] = XT(0);
      win[k * D + d] = rx[d];
      if (A.r_smem) Rs[k * D + d] = rx[d];
      if (A.x_smem) Xs[k * D + d] = XT(0);
    }
    N::st(Rg + (size_t)k * VD, rx);
    if (!A.x_smem) N::st(Xg + (size_t)k * VD, z);
  }
  for (int k = tid; k < nsl; k += NT) slen[k] = P.slen[s0 + k];
  unsigned epoch = 1;
  bool ok = true;
  const auto share = [&](auto f) {  // f(total, sc) on lane 0 of warp 0, then all see sc
    if (w == 0) {
      const double tot = grid_red_total(A.red, epoch, &sc.ok);
      if (lane == 0) f(tot);
    }
    __syncthreads();
    epoch++;
    ok = sc.ok;
  };
  grid_red_arrive(acc0, A.red, epoch);
  share([&](double tot) {
    const double iNorm = sqrt(tot), e0 = fmax(A.absTol, A.relTol * iNorm);
    sc.err = sc.errO = iNorm * iNorm;
    sc.alpha = sc.beta = 0.0;
    sc.eps = e0 * e0;
    sc.done = sc.suc = sc.itr = 0;
    if (A.mItr < 1)
      sc.done = 2;
    else if (sc.err < sc.eps) {
      sc.done = 1;
      sc.suc = 1;
    }
    if (!isfinite(tot)) sc.done = 3;
    if (b == 0) {
      A.S->iNorm = iNorm;
      A.S->eps = sc.eps;
      A.S->mItr = A.mItr;
    }
  });
  if (ok && !sc.done) {
    for (int k = tid; k < nhalo; k += NT) {
      XT r[D];
      N::ld(A.Rg + (size_t)__ldg(halo + k) * VD, r);
#pragma unroll
      for (int d = 0; d < D; d++) win[(own + k) * D + d] = r[d];
    }
    __syncthreads();
  }

  bool rev = false;
  while (ok && !sc.done) {
    // 1. KP = K P, P.KP
    AT dot = AT(0);
    if (ng > 0)
      dot = rev ? wcg_pass<true, W, D, VT, XT, AT>(stream, ng, nst, nq, w, lane, L, A.ahead, slen, win, KP)
                : wcg_pass<false, W, D, VT, XT, AT>(stream, ng, nst, nq, w, lane, L, A.ahead, slen, win, KP);
    rev = !rev;
    grid_red_arrive(dot, A.red, epoch);
    share([&](double tot) {
      sc.errO = sc.err;
      sc.alpha = grid_div(sc.errO, tot);
      sc.a = XT(sc.alpha);
      if (!fix_finite(sc.alpha)) sc.done = 3;
    });
    if (!ok || sc.done) break;
    // 2. R and |R|^2; X while the sum is on its way
    const XT al = sc.a;
    XT acc = XT(0);
    if (A.r_smem) {
      for (int k = tid; k < own; k += NT) {
        XT r[D];
#pragma unroll
        for (int d = 0; d < D; d++) {
          r[d] = fma(-al, KP[k * D + d], Rs[k * D + d]);
          Rs[k * D + d] = r[d];
          acc = fma(r[d], r[d], acc);
        }
        N::st(Rg + (size_t)k * VD, r);
      }
    } else {
      for_nodes<kB<D, XT>, D, XT>(own, [&](int k, XT r[D]) { N::ld(Rg + (size_t)k * VD, r); },
                           [&](int k, XT r[D]) {
#pragma unroll
                             for (int d = 0; d < D; d++) {
                               r[d] = fma(-al, KP[k * D + d], r[d]);
                               acc = fma(r[d], r[d], acc);
                             }
                             N::st(Rg + (size_t)k * VD, r);
                           });
    }
    grid_red_arrive(acc, A.red, epoch);
    if (A.x_smem) {
      for (int k = tid; k < own * D; k += NT) Xs[k] = fma(al, win[k], Xs[k]);
    } else {
      for_nodes<kB<D, XT>, D, XT>(own, [&](int k, XT x[D]) { N::ld(Xg + (size_t)k * VD, x); },
                           [&](int k, XT x[D]) {
#pragma unroll
                             for (int d = 0; d < D; d++) x[d] = fma(al, win[k * D + d], x[d]);
                             N::st(Xg + (size_t)k * VD, x);
                           });
    }
    // 3. stopping tests in CGRAD's order, next direction
    share([&](double tot) {
      sc.err = tot;
      sc.beta = grid_div(tot, sc.errO);
      sc.a = XT(sc.beta);
      sc.itr++;
      if (!fix_finite(tot))
        sc.done = 3;
      else if (sc.itr >= A.mItr)
        sc.done = 2;
      else if (tot < sc.eps) {
        sc.done = 1;
        sc.suc = 1;
      }
    });
    if (!ok || sc.done) break;
    const XT be = sc.a;
    for_nodes<kB<D, XT>, D, XT>(nhalo,
                         [&](int k, XT r[D]) {
                           N::ld(A.Rg + (size_t)__ldg(halo + k) * VD, r);
                         },
                         [&](int k, XT r[D]) {
#pragma unroll
                           for (int d = 0; d < D; d++)
                             win[(own + k) * D + d] = fma(be, win[(own + k) * D + d], r[d]);
                         });
    if (A.r_smem) {
      for (int k = tid; k < own * D; k += NT) win[k] = fma(be, win[k], Rs[k]);
    } else {
      for_nodes<kB<D, XT>, D, XT>(own, [&](int k, XT r[D]) { N::ld(Rg + (size_t)k * VD, r); },
                           [&](int k, XT r[D]) {
#pragma unroll
                             for (int d = 0; d < D; d++)
                               win[k * D + d] = fma(be, win[k * D + d], r[d]);
                           });
    }
    __syncthreads();
  }
  __syncthreads();
  for (int k = tid; k < own; k += NT) {
    const int row = __ldg(P.slotRow + g0 + k);
    if (row < 0) continue;
    XT x[D];
    if (A.x_smem) {
#pragma unroll
      for (int d = 0; d < D; d++) x[d] = Xs[k * D + d];
    } else {
      N::ld(Xg + (size_t)k * VD, x);
    }
#pragma unroll
    for (int d = 0; d < D; d++) A.R[(size_t)row * D + d] = A.W[(size_t)row * D + d] * double(x[d]);
  }
  if (b == 0 && threadIdx.x == 0) {
    KrylovScalars *S = A.S;
    S->err = sc.err;
    S->errO = sc.errO;
    S->alpha = sc.alpha;
    S->beta = sc.beta;
    S->itr = sc.itr;
    S->suc = sc.suc;
    S->done = sc.done;
  }
  // any block that gave up a wait says so itself (block 0 may have finished)
  if (threadIdx.x == 0 && !ok) atomicExch(&A.red.buf->bar.err, 1);
}

// Most dynamic shared memory of a block of the kernel
template <int D, class VT, class XT>
static size_t wcg_cap() {
  static const size_t cap = [] { return smem_cap((const void *)k_wcg<D, VT, XT>); }();
  return cap;
}

// Shared memory of the kernel: the window and KP; R of the own rows, then X,
// where they fit too.  0: the window does not fit.
template <int D, class VT, class XT>
static size_t wcg_geometry(const PartArgs &P, WcgArgs<XT> &A) {
  const size_t cap = wcg_cap<D, VT, XT>();
  const auto up16 = [](size_t n) { return (n + 15) & ~(size_t)15; };
  A.ownMax = P.nslMax * (32 / P.L);
  const size_t own1 = (size_t)A.ownMax * D * sizeof(XT);
  size_t n =
      up16((size_t)P.winMax * D * sizeof(XT)) + up16(own1) + up16((size_t)P.nslMax * sizeof(int));
  if (n > cap) return 0;
  A.r_smem = n + own1 <= cap;
  if (A.r_smem) n += own1;
  A.x_smem = A.r_smem && n + own1 <= cap;
  if (A.x_smem) n += own1;
  return n;
}

template <int D, class VT, class XT>
static int wcg_t(gsls_lhs *lhs, gsls_sub_ls *ls, const VT *Val, double *R, const double *W,
                 bool keep, bool *ran) {
  *ran = false;
  cudaStream_t st = lhs->stream;
  Workspace &ws = lhs->ws;
  // window and KP of the own rows
  if (part_rows(lhs) * 2 * D * (long long)sizeof(XT) > (long long)wcg_cap<D, VT, XT>())
    return GSLS_OK;
  WcgArgs<XT> A{};
  size_t smem = 0;
  RowPart *part;
  GSLS_TRY(part_for(lhs, &part, [&](const RowPart &p) {
    smem = wcg_geometry<D, VT, XT>(part_args(p), A);
    return smem != 0;
  }));
  if (!part) return GSLS_OK;
  const PartArgs P = part_args(*part);
  const size_t vb = ((size_t)P.nslots * NodeL2<D, XT>::VD * sizeof(XT) + 127) & ~(size_t)127;
  const size_t sb = Rec<D, VT>::at(P.nsteps, P.nblk * kPartWarps);
  // no memory for a second copy of the matrix: the batched kernels take the
  // solve, and later ones of that size without another try
  if (sb >= ws.wcg_short) return GSLS_OK;
  if (!ws.wcg_stream.try_alloc(sb) || !ws.wcg_vec.try_alloc(2 * vb)) {
    ws.wcg_stream.release();
    ws.wcg_vec.release();
    ws.wcg_key = 0;
    ws.wcg_short = sb;
    return GSLS_OK;
  }
  *ran = true;
  const int key = D * 16 + (int)sizeof(VT);
  // keep: Val is the matrix that the last preconditioning on this lhs left
  // (no other call can have changed it), so its stream is packed already
  if (!(keep && ws.wcg_key == key && ws.wcg_val == Val && ws.wcg_serial == ws.pre_serial)) {
    k_wcg_pack<D, VT><<<8 * num_sms(), 256, 0, st>>>(P, Val, ws.wcg_stream.as<unsigned char>(),
                                                     (P.stMax + 7) / 8);
    GSLS_CHECK_LAUNCH();
    ws.wcg_key = key;
    ws.wcg_val = Val;
    ws.wcg_serial = ws.pre_serial;
  }
  unsigned char *sc = ws.scal.as<unsigned char>();
  GSLS_CUDA(cudaMemsetAsync(sc + kScalRed, 0, sizeof(GridBar), st));
  unsigned char *v = ws.wcg_vec.as<unsigned char>();
  A.P = P;
  A.stream = ws.wcg_stream.as<unsigned char>();
  A.R = R;
  A.W = W;
  A.Xg = reinterpret_cast<XT *>(v);
  A.Rg = reinterpret_cast<XT *>(v + vb);
  A.S = ws.scal.as<KrylovScalars>();
  A.absTol = ls->absTol;
  A.relTol = ls->relTol;
  A.mItr = ls->mItr;
  GridRedBuf *rb = reinterpret_cast<GridRedBuf *>(sc + kScalRed);
  A.red = GridRed{rb, (unsigned)P.nblk, wait_limit()};
  // a stream larger than L2 is prefetched into it three groups ahead (beam:
  // 54,700 -> 49,700 cycles a product; six ahead 52,300, twelve 67,700)
  A.ahead = (size_t)P.nsteps * Rec<D, VT>::SB > ((size_t)100 << 20) ? 3 : 0;
  void *args[] = {&A};
  const bool prof = prof_on();
  if (prof) cudaEventRecord(prof_event(0), st);
  GSLS_TRY(coop_launch((const void *)k_wcg<D, VT, XT>, wcg_cap<D, VT, XT>(), P.nblk, args, smem,
                       st));
  GSLS_CHECK_LAUNCH();
  if (prof) cudaEventRecord(prof_event(1), st);
  // the error word travels behind the scalars
  GSLS_CUDA(cudaMemcpyAsync(ws.h_scal, sc, kScalHost, cudaMemcpyDeviceToHost, st));
  GSLS_CUDA(cudaStreamSynchronize(st));
  const GridBar *hb = reinterpret_cast<const GridBar *>(
      reinterpret_cast<const unsigned char *>(ws.h_scal) + kScalRed);
  if (hb->err) ws.h_scal->done = 4;
  if (prof) {
    float ms = 0.f;
    cudaEventElapsedTime(&ms, prof_event(0), prof_event(1));
    prof_add("cg_persistent", ws.h_scal->itr, ms);
  }
  return GSLS_OK;
}

int wcg_run(gsls_lhs *lhs, gsls_sub_ls *ls, int D, bool mixed, const void *Val, double *R,
            const double *W, bool keep, bool *ran) {
#define GSLS_WCG_CASE(DV)                                                                    \
  case DV:                                                                                   \
    return mixed ? wcg_t<DV, float, float>(lhs, ls, (const float *)Val, R, W, keep, ran)     \
                 : wcg_t<DV, double, double>(lhs, ls, (const double *)Val, R, W, keep, ran);
  switch (D) {
    GSLS_WCG_CASE(1)
    GSLS_WCG_CASE(2)
    GSLS_WCG_CASE(3)
    GSLS_WCG_CASE(4)
    default:
      return GSLS_ERR_UNSUPPORTED;
  }
#undef GSLS_WCG_CASE
}

}  // namespace gsls
