// The Schur-complement CG of the NS solver (CGRAD_SCHUR,
// Code/Source/svFSILS/CGRAD.f:51-123) as one cooperative launch per call on
// the row partition of gsls_part.cuh.
//
// The operator S = mL - Gt mG is applied as two products.  Every block keeps
// its window of P and of GP = mG P in shared memory and reads the operands
// of its rows as two sequential streams per warp.  Iteration k:
//  1. GP of the own rows, published; grid barrier; GP of the halo;
//  2. SP = mL P - Gt GP and the partials of P.SP; grid sum: alpha;
//  3. X += alpha P, R -= alpha SP, R published, the partials of |R|^2; grid
//     sum: err, stopping tests; P = (err/errO) (P + (errO/err) R) for the own
//     rows and, from the published R, for the halo.
// A row reads ~15 entries of each vector: gathered from L2 (a 32-byte sector
// for every 4 or 16 bytes) they were 400 MB of the ~500 MB that an iteration
// moved on the cylinder of 216,318 nodes; the halos are 6 MB.
// Measured there (GB300, FP32): ~33 us per iteration against 45 us with the
// gathers (the operator, 96 MB with its columns, takes 8 us at the measured
// L2 read rate and 14 us at the HBM copy rate; two grid sums and a barrier
// ~9 us); the mixed step 453 -> 349 ms.
#include "gsls_wschur.cuh"

#include <cstring>

#include "gsls_gridbar.cuh"
#include "gsls_part.cuh"
#include "gsls_spmv.cuh"

namespace gsls {

// NB values per block in groups of G steps: per group and lane G window
// columns and G blocks as NV 16-byte vectors.  A group never crosses the end
// of a slice (with an end-of-slice branch after every step the two products
// took 57,000 instead of 33,000 cycles on the cylinder); the vectors of a
// last group's padding are not read.
template <int NB, class VT>
struct SRec {
  static constexpr int G = sizeof(VT) == 4 ? 4 : 2;
  static constexpr int N16 = 16 / (int)sizeof(VT);
  static constexpr int NV = G * NB / N16;
  static constexpr int PD = sizeof(VT) == 4 ? 3 : 2;  // groups in flight
  static constexpr int SB = 64 + NB * 32 * (int)sizeof(VT);
  static_assert(G * NB % N16 == 0, "whole vectors");
};
template <int NB, class VT>
struct SGroup {
  using R = SRec<NB, VT>;
  VT a[R::G * NB];
  unsigned short c[R::G];
  __device__ __forceinline__ void load(const unsigned char *g, int lane, int valid) {
    if constexpr (R::G == 4)
      *reinterpret_cast<uint2 *>(c) = __ldg(reinterpret_cast<const uint2 *>(g) + lane);
    else
      *reinterpret_cast<unsigned *>(c) = __ldg(reinterpret_cast<const unsigned *>(g) + lane);
#pragma unroll
    for (int q = 0; q < R::NV; q++)
      if (q * R::N16 < valid * NB)
        *reinterpret_cast<uint4 *>(a + q * R::N16) =
            __ldg(reinterpret_cast<const uint4 *>(g + 64 * R::G + q * 512) + lane);
  }
};

// one warp per slice; NB == 3: (mG), NB == 4: (Gt, mL)
template <int NB, class VT>
__global__ void __launch_bounds__(256) k_wschur_pack(PartArgs P, const VT *__restrict__ K3,
                                                     const VT *__restrict__ K1,
                                                     unsigned char *__restrict__ stream) {
  using R = SRec<NB, VT>;
  const int lane = threadIdx.x & 31;
  const int warp = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int nw = (int)(((long long)gridDim.x * blockDim.x) >> 5);
  for (int s = warp; s < P.nS; s += nw) {
    const int first = __ldg(P.sst + s), n = __ldg(P.slen + s), at = __ldg(P.soff + s);
#pragma unroll 2
    for (int g0 = 0; g0 < n; g0 += R::G) {
      unsigned char *g = stream + (size_t)(at + g0) * R::SB;
      __align__(16) VT a[R::G * NB];
#pragma unroll
      for (int u = 0; u < R::G; u++) {
        const size_t e = (size_t)(first + g0 + u) * 32 + lane;
        const int j = g0 + u < n ? __ldg(P.src + e) : -1;  // padding of the group
        reinterpret_cast<unsigned short *>(g)[lane * R::G + u] =
            g0 + u < n ? __ldg(P.lcol + e) : 0;
#pragma unroll
        for (int k = 0; k < 3; k++) a[u * NB + k] = j >= 0 ? __ldg(K3 + (size_t)j * 3 + k) : VT(0);
        if constexpr (NB == 4) a[u * NB + 3] = j >= 0 ? __ldg(K1 + j) : VT(0);
      }
#pragma unroll
      for (int q = 0; q < R::NV; q++)
        reinterpret_cast<uint4 *>(g + 64 * R::G + q * 512)[lane] =
            *reinterpret_cast<const uint4 *>(a + q * R::N16);
    }
  }
}

template <class XT>
struct WschurArgs {
  PartArgs P;
  const unsigned char *s1, *s2;
  XT *x;         // in: right-hand side, out: solution (row order)
  XT *Rg, *GPg;  // slot order; GPg 4 per node
  SchurScal *sc;
  double absTol, relTol;
  int mItr;
  GridRed red;
  int ownMax, tabMax;
};

// One pass of a warp over its groups (tab, ng of them), from the end if rev.
// NB 3: GP = mG P of its rows, into the window and out (4 per node); NB 4:
// SP = mL P - Gt GP into out, the sum of P.SP returned
template <int NB, class VT, class XT>
static __device__ __noinline__ typename AccOf<VT>::T wschur_pass(
    const unsigned char *__restrict__ stream, const int *tab, int ng, int w, int nq, int lane,
    int L, int rev, const XT *Pw, XT *GPw, XT *out) {
  using AT = typename AccOf<VT>::T;
  using R = SRec<NB, VT>;
  using N3 = NodeL2<3, XT>;
  const int RW = 32 / L, di = rev ? -1 : 1, fin = rev ? kGrpFirst : kGrpLast;
  int i0 = rev ? ng - 1 : 0, s = rev ? w + (nq - 1) * kPartWarps : w;
  AT acc[3] = {AT(0), AT(0), AT(0)}, dot = AT(0);
  // PD + 1 groups in registers take turns (see gsls_wcg.cu)
  SGroup<NB, VT> grp[R::PD + 1];
  int ent[R::PD + 1];
#pragma unroll
  for (int k = 0; k < R::PD; k++)
    if (k < ng) {
      ent[k] = tab[i0 + k * di];
      grp[k].load(stream + (size_t)(ent[k] & kGrpOff) * R::SB, lane, grp_valid(ent[k]));
    }
  const auto turn = [&](int i, int e, const SGroup<NB, VT> &cur, int &en, SGroup<NB, VT> &next) {
    if (i + R::PD < ng) {
      en = tab[i0 + (i + R::PD) * di];
      next.load(stream + (size_t)(en & kGrpOff) * R::SB, lane, grp_valid(en));
    }
    XT p[R::G], g[R::G][3];
#pragma unroll
    for (int u = 0; u < R::G; u++) {
      p[u] = Pw[cur.c[u]];
      if constexpr (NB == 4) {
#pragma unroll
        for (int m = 0; m < 3; m++) g[u][m] = GPw[cur.c[u] * 3 + m];
      }
    }
#pragma unroll
    for (int u = 0; u < R::G; u++) {
      if (u < grp_valid(e)) {
        if constexpr (NB == 3) {
#pragma unroll
          for (int m = 0; m < 3; m++) acc[m] = fma(AT(cur.a[u * 3 + m]), AT(p[u]), acc[m]);
        } else {
          acc[0] = fma(AT(cur.a[u * 4 + 3]), AT(p[u]), acc[0]);
#pragma unroll
          for (int m = 0; m < 3; m++) acc[1] = fma(AT(cur.a[u * 4 + m]), AT(g[u][m]), acc[1]);
        }
      }
    }
    if (e & fin) {
      // end of the slice
      constexpr int NA = NB == 3 ? 3 : 2;
#pragma unroll 1
      for (int o = 1; o < L; o <<= 1)
#pragma unroll
        for (int m = 0; m < NA; m++) acc[m] += __shfl_xor_sync(0xffffffffu, acc[m], o);
      if ((lane & (L - 1)) == 0) {
        const int k = s * RW + lane / L;
        if constexpr (NB == 3) {
          XT v[3];
#pragma unroll
          for (int m = 0; m < 3; m++) GPw[k * 3 + m] = v[m] = XT(acc[m]);
          N3::st(out + (size_t)k * 4, v);
        } else {
          const XT v = XT(acc[0] + AT(-1) * acc[1]);
          out[k] = v;
          dot = fma(AT(Pw[k]), AT(v), dot);
        }
      }
      acc[0] = acc[1] = acc[2] = AT(0);
      s += di * kPartWarps;
    }
  };
#pragma unroll 1
  for (int i = 0; i < ng; i += R::PD + 1) {
#pragma unroll
    for (int k = 0; k <= R::PD; k++)
      if (i + k < ng)
        turn(i + k, ent[k], grp[k], ent[(k + R::PD) % (R::PD + 1)],
             grp[(k + R::PD) % (R::PD + 1)]);
  }
  return dot;
}

template <class XT>
struct WschurShared {
  double err, errO, eps;
  XT alpha, malpha, c1, c2;
  int done, suc, itr, ok;
};

template <class VT, class XT>
__global__ void __launch_bounds__(kPartThreads, 1) k_wschur(WschurArgs<XT> A) {
  using AT = typename AccOf<VT>::T;
  using N1 = NodeL2<1, XT>;
  using N3 = NodeL2<3, XT>;
  using R1 = SRec<3, VT>;
  using R2 = SRec<4, VT>;
  constexpr int NT = kPartThreads;
  extern __shared__ __align__(16) unsigned char smem[];
  const PartArgs &P = A.P;
  const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int L = P.L, RW = 32 / L;
  const int s0 = P.sbase[b], nsl = P.sbase[b + 1] - s0;
  const int own = nsl * RW, nhalo = P.hoff[b + 1] - P.hoff[b];
  const int *__restrict__ halo = P.halo + P.hoff[b];
  const size_t g0 = (size_t)s0 * RW;
  // shared memory: P window | GP window | X | R | SP | groups of the warps
  XT *Pw = reinterpret_cast<XT *>(smem), *GPw = Pw + P.winMax, *X = GPw + 3 * (size_t)P.winMax;
  XT *R = X + A.ownMax, *SP = R + A.ownMax;
  int *tab = reinterpret_cast<int *>(SP + A.ownMax) + w * A.tabMax;
  XT *Rg = A.Rg + g0, *GPg = A.GPg + g0 * 4;
  __shared__ WschurShared<XT> sc;

  // this warp's groups (the same for both streams)
  static_assert(R1::G == R2::G, "one table");
  const int ng = part_groups<R1::G>(P.soff + s0, P.slen + s0, nsl, w, tab);
  const int nq = w < nsl ? (nsl - 1 - w) / kPartWarps + 1 : 0;
  const unsigned char *__restrict__ s1 = A.s1 + (size_t)P.soff[s0] * R1::SB;
  const unsigned char *__restrict__ s2 = A.s2 + (size_t)P.soff[s0] * R2::SB;

  // X = 0, R = P = right-hand side
  double acc = 0.0;
  for (int k = tid; k < own; k += NT) {
    const int row = __ldg(P.slotRow + g0 + k);
    const XT v = row >= 0 ? A.x[row] : XT(0);
    Pw[k] = v;
    R[k] = v;
    X[k] = XT(0);
    __stcg(Rg + k, v);
    acc += double(v) * double(v);
  }
  unsigned epoch = 1;
  bool ok = true;
  const auto share = [&](auto f) {  // f(total) on lane 0 of warp 0, then all see sc
    if (w == 0) {
      const double tot = grid_red_total(A.red, epoch, &sc.ok);
      if (lane == 0) f(tot);
    }
    __syncthreads();
    epoch++;
    ok = sc.ok;
  };
  grid_red_arrive(acc, A.red, epoch);
  share([&](double tot) {
    const double in = sqrt(tot), e = fmax(A.absTol, A.relTol * in);
    sc.err = sc.errO = in * in;
    sc.eps = e * e;
    sc.itr = 0;
    sc.suc = sc.err < sc.eps ? 1 : 0;
    sc.done = (sc.suc || A.mItr < 1) ? 1 : 0;
    if (!fix_finite(tot)) sc.done = 3;
    if (b == 0) A.sc->iNorm2 = tot;
  });
  if (ok && !sc.done) {
    for_nodes<kB<1, XT>, 1, XT>(
        nhalo, [&](int k, XT r[1]) { N1::ld(A.Rg + __ldg(halo + k), r); },
        [&](int k, XT r[1]) { Pw[own + k] = r[0]; });
    __syncthreads();
  }
  while (ok && !sc.done) {
    // 1. GP = mG P
    // odd iterations walk both streams from the end: what L2 still holds of
    // them is met first
    const int rev = sc.itr & 1;
    if (ng > 0) wschur_pass<3, VT, XT>(s1, tab, ng, w, nq, lane, L, rev, Pw, GPw, GPg);
    grid_bar_arrive(A.red);
    if (w == 0) grid_bar_wait(A.red, epoch, &sc.ok);
    __syncthreads();
    epoch++;
    if (!(ok = sc.ok)) break;
    for_nodes<kB<3, XT>, 3, XT>(
        nhalo, [&](int k, XT r[3]) { N3::ld(A.GPg + (size_t)__ldg(halo + k) * 4, r); },
        [&](int k, XT r[3]) {
#pragma unroll
          for (int m = 0; m < 3; m++) GPw[(own + k) * 3 + m] = r[m];
        });
    __syncthreads();
    // 2. SP = mL P - Gt GP, P.SP (added in FP64 beyond a thread)
    AT dot = AT(0);
    if (ng > 0)
      dot = wschur_pass<4, VT, XT>(s2, tab, ng, w, nq, lane, L, rev, Pw, GPw, SP);
    grid_red_arrive(double(dot), A.red, epoch);
    share([&](double tot) {
      sc.errO = sc.err;
      const double alpha = grid_div(sc.errO, tot);
      sc.alpha = XT(alpha);
      sc.malpha = XT(-alpha);
    });
    if (!ok) break;
    // 3. X, R and |R|^2
    const XT al = sc.alpha, mal = sc.malpha;
    acc = 0.0;
    for (int k = tid; k < own; k += NT) {
      const XT r = XT(R[k] + mal * SP[k]);
      R[k] = r;
      __stcg(Rg + k, r);
      acc += double(r) * double(r);
    }
    grid_red_arrive(acc, A.red, epoch);
    for (int k = tid; k < own; k += NT) X[k] = XT(X[k] + al * Pw[k]);
    share([&](double tot) {
      sc.err = tot;
      sc.c1 = XT(grid_div(sc.errO, tot));
      sc.c2 = XT(grid_div(tot, sc.errO));
      sc.itr++;
      if (!fix_finite(tot)) {
        sc.done = 3;
      } else if (sc.itr >= A.mItr) {
        sc.done = 2;  // no stop test after the last iteration
      } else if (tot < sc.eps) {
        sc.suc = 1;
        sc.done = 1;
      }
    });
    if (!ok || sc.done) break;
    // P = (err/errO) (P + (errO/err) R)
    const XT c1 = sc.c1, c2 = sc.c2;
    for_nodes<kB<1, XT>, 1, XT>(
        nhalo, [&](int k, XT r[1]) { N1::ld(A.Rg + __ldg(halo + k), r); },
        [&](int k, XT r[1]) { Pw[own + k] = XT(c2 * (Pw[own + k] + c1 * r[0])); });
    for (int k = tid; k < own; k += NT) Pw[k] = XT(c2 * (Pw[k] + c1 * R[k]));
    __syncthreads();
  }
  __syncthreads();
  for (int k = tid; k < own; k += NT) {
    const int row = __ldg(P.slotRow + g0 + k);
    if (row >= 0) A.x[row] = X[k];
  }
  if (b == 0 && tid == 0) {
    A.sc->err = sc.err;
    A.sc->errO = sc.errO;
    A.sc->eps = sc.eps;
    A.sc->itr = sc.itr;
    A.sc->mItr = A.mItr;
    A.sc->suc = sc.suc;
    A.sc->done = sc.done;
  }
  if (tid == 0 && !ok) atomicExch(&A.red.buf->bar.err, 1);
}

template <class XT>
static size_t wschur_smem(const RowPart &p) {
  return sizeof(XT) * (4 * (size_t)p.winMax + 3 * (size_t)p.nslMax * (32 / p.L)) +
         sizeof(int) * (size_t)kPartWarps * grp_cap(p.nslMax, p.grpMax, SRec<3, XT>::G);
}

template <class VT, class XT>
static size_t wschur_cap() {
  static const size_t cap = [] { return smem_cap((const void *)k_wschur<VT, XT>); }();
  return cap;
}

template <class VT>
int wschur_pack(gsls_lhs *lhs, const VT *mG, const VT *Gt, const VT *mL, bool *fits) {
  *fits = false;
  Workspace &ws = lhs->ws;
  // P and GP of the own rows, X, R and SP
  if (part_rows(lhs) * 7 * (long long)sizeof(VT) > (long long)wschur_cap<VT, VT>()) return GSLS_OK;
  GSLS_TRY(part_for(lhs, &ws.ns_part, [](const RowPart &p) {
    return wschur_smem<VT>(p) <= wschur_cap<VT, VT>();
  }));
  if (!ws.ns_part) return GSLS_OK;
  const PartArgs P = part_args(*ws.ns_part);
  const size_t n1 = (size_t)P.nsteps8 * SRec<3, VT>::SB, n2 = (size_t)P.nsteps8 * SRec<4, VT>::SB;
  const size_t vb = ((size_t)P.nslots * sizeof(VT) + 127) & ~(size_t)127;
  // no memory for the streams: the per-kernel Schur CG, without another try
  const size_t sb = n1 + n2 + 5 * vb + 512;
  if (sb >= ws.ns_short) return GSLS_OK;
  if (!ws.ns_stream.try_alloc(sb)) {
    ws.ns_short = sb;
    return GSLS_OK;
  }
  unsigned char *s1 = ws.ns_stream.as<unsigned char>(), *s2 = s1 + ((n1 + 127) & ~(size_t)127);
  k_wschur_pack<3, VT><<<8 * num_sms(), 256, 0, lhs->stream>>>(P, mG, nullptr, s1);
  GSLS_CHECK_LAUNCH();
  k_wschur_pack<4, VT><<<8 * num_sms(), 256, 0, lhs->stream>>>(P, Gt, mL, s2);
  GSLS_CHECK_LAUNCH();
  *fits = true;
  return GSLS_OK;
}

template <class VT, class XT>
int wschur_run(gsls_lhs *lhs, const gsls_sub_ls *ls, XT *x, SchurScal *out) {
  Workspace &ws = lhs->ws;
  cudaStream_t st = lhs->stream;
  const PartArgs P = part_args(*ws.ns_part);
  const size_t n1 = ((size_t)P.nsteps8 * SRec<3, VT>::SB + 127) & ~(size_t)127;
  const size_t n2 = ((size_t)P.nsteps8 * SRec<4, VT>::SB + 127) & ~(size_t)127;
  const size_t vb = ((size_t)P.nslots * sizeof(XT) + 127) & ~(size_t)127;
  unsigned char *s1 = ws.ns_stream.as<unsigned char>();
  unsigned char *sc = ws.scal.as<unsigned char>();
  const size_t smem = wschur_smem<XT>(*ws.ns_part);
  GSLS_CUDA(cudaMemsetAsync(sc + kScalRed, 0, sizeof(GridBar), st));
  WschurArgs<XT> A{};
  A.P = P;
  A.s1 = s1;
  A.s2 = s1 + n1;
  A.x = x;
  A.Rg = reinterpret_cast<XT *>(s1 + n1 + n2);
  A.GPg = reinterpret_cast<XT *>(s1 + n1 + n2 + vb);
  A.sc = reinterpret_cast<SchurScal *>(sc);
  A.absTol = ls->absTol;
  A.relTol = ls->relTol;
  A.mItr = ls->mItr;
  A.red = GridRed{reinterpret_cast<GridRedBuf *>(sc + kScalRed), (unsigned)P.nblk, wait_limit()};
  A.ownMax = P.nslMax * (32 / P.L);
  A.tabMax = grp_cap(P.nslMax, P.grpMax, SRec<3, VT>::G);
  void *args[] = {&A};
  const bool prof = prof_on();
  if (prof) cudaEventRecord(prof_event(0), st);
  GSLS_TRY(coop_launch((const void *)k_wschur<VT, XT>, wschur_cap<VT, XT>(), P.nblk, args, smem,
                       st));
  GSLS_CHECK_LAUNCH();
  if (prof) cudaEventRecord(prof_event(1), st);
  // the error word travels behind the scalars
  GSLS_CUDA(cudaMemcpyAsync(ws.h_scal, sc, kScalHost, cudaMemcpyDeviceToHost, st));
  GSLS_CUDA(cudaStreamSynchronize(st));
  const unsigned char *h = reinterpret_cast<const unsigned char *>(ws.h_scal);
  memcpy(out, h, sizeof(SchurScal));
  if (reinterpret_cast<const GridBar *>(h + kScalRed)->err) out->done = 4;
  if (prof) {
    // per CG iteration: count = iterations of this call
    float ms = 0.f;
    cudaEventElapsedTime(&ms, prof_event(0), prof_event(1));
    prof_add("schur", out->itr, ms);
    prof_add("schur_calls", 1, ms);
  }
  return GSLS_OK;
}

template int wschur_pack<float>(gsls_lhs *, const float *, const float *, const float *, bool *);
template int wschur_pack<double>(gsls_lhs *, const double *, const double *, const double *,
                                 bool *);
template int wschur_run<float, float>(gsls_lhs *, const gsls_sub_ls *, float *, SchurScal *);
template int wschur_run<double, double>(gsls_lhs *, const gsls_sub_ls *, double *, SchurScal *);

}  // namespace gsls
