// Construction of the row partition (gsls_part.cuh): the rows of each block on
// the host, the halos and columns on the device.
//
// It is paid once per lhs, by the first solve.  All on the host it took 1.6 ms
// for the 9,261 rows of the 20^3 cube and 42 ms for the 517,888 of the CEP slab,
// mostly the columns of every step and their upload (48 MB).
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <new>
#include <thread>

#include "gsls_part.cuh"

namespace gsls {

// f(b) for every block b, on up to 16 host threads; the result of a block depends
// on b only.  False when host memory could not be had.
template <class F>
static bool for_blocks(int nblk, long long work, const F &f) {
  const unsigned hw = std::thread::hardware_concurrency();
  const int T = (int)std::min<long long>(std::min({nblk, 16, hw ? (int)hw : 1}), 1 + work / 40000);
  std::atomic<int> next{0};
  std::atomic<bool> ok{true};
  const auto run = [&] {
    try {
      for (int b; (b = next.fetch_add(1)) < nblk;) f(b);
    } catch (...) {
      ok = false;
    }
  };
  std::vector<std::thread> th;
  try {
    for (int t = 1; t < T; t++) th.emplace_back(run);
  } catch (...) {
    // no more threads: the ones that started and this one do the work
  }
  run();
  for (auto &x : th) x.join();
  return ok;
}

// The rows of each block in slot order, their slices and steps
struct PartHost {
  int nblk = 0, L = 1, nslMax = 0, stMax = 0, grpMax = 0;
  long long steps8 = 0;
  bool ok = false;
  std::vector<int> wbase, sst, soff, sbase, slen, slotRow;
};

static void part_host(int nNo, const std::vector<int> &rp, const std::vector<int> &cp, int sms,
                      PartHost &H) {
  // blocks of at least 32 rows
  const int nblk = H.nblk = std::max(1, std::min({sms, kPartMaxBlocks, (nNo + 31) / 32}));
  constexpr int W = kPartWarps;
  const double rows = (double)nNo / nblk, len = nNo ? (double)rp[nNo] / nNo : 1.0;
  // Lanes per row: the least FP64 issue slots of a scheduler (its slices,
  // each with its steps and, per doubling of L, one more add), 1.5 times that
  // where no scheduler has more than one warp at work (one warp alone issues
  // every ~105 cycles instead of 64).  From four slices per warp on, L = 1.
  int &L = H.L;
  double best = 1e300;
  for (int l = 1, lg = 0; l <= 8; l *= 2, lg++) {
    const double nsl = ceil(rows * l / 32);
    const double cost = ceil(nsl / 4) * (3.0 * ceil(len / l) + lg) * (nsl <= 4 ? 1.5 : 1.0);
    if (cost < best) {
      best = cost;
      L = l;
    }
    if (nsl >= 4 * W) break;
  }
  const int RW = 32 / L;
  // Row order and the blocks' shares of it.  A few slices per warp: equal
  // numbers of rows, so that no block has a slice more than the others;
  // otherwise equal numbers of matrix blocks + 4 per row.
  std::vector<int> order((size_t)nNo), row0((size_t)nblk + 1, nNo);
  for (int i = 0; i < nNo; i++) order[i] = i;
  const bool by_rows = rows < 4.0 * W * RW;
  const auto wt = [&](int i) { return by_rows ? 1LL : 4LL + rp[i + 1] - rp[i]; };
  // cuts order[i0, i1) into blocks b0 .. b1-1
  const auto cut = [&](int i0, int i1, int b0, int b1) {
    long long tot = 0, run = 0;
    for (int k = i0; k < i1; k++) tot += wt(order[k]);
    int k = i0;
    for (int b = b0; b < b1; b++) {
      const long long lim = tot * (b - b0) / (b1 - b0);
      while (k < i1 && run < lim) run += wt(order[k++]);
      row0[b] = k;
    }
  };
  cut(0, nNo, 0, nblk);
  // Rows numbered plane by plane: a block of about one plane has a halo of
  // two.  A slab of q blocks cut into q strips across the numbering has less:
  // with planes of s x s rows, 2 rows q / s + 2 s^2 / q per block, least at
  // q = sqrt(s^3 / rows) (beam of 176 x 44 x 44 hexes: q = 6, window 7,890 ->
  // 4,100 entries).  The strips are the order of a breadth-first search of
  // the slab from its far end.
  int q = 1;
  if (nblk > 8 && rows >= 512) {
    const int b = nblk / 2, r0 = row0[b], r1 = row0[b + 1];
    std::vector<int> h;
    for (int i = r0; i < r1; i++)
      for (int j = rp[i]; j < rp[i + 1]; j++)
        if (cp[j] < r0 || cp[j] >= r1) h.push_back(cp[j]);
    std::sort(h.begin(), h.end());
    const double plane = 0.5 * (std::unique(h.begin(), h.end()) - h.begin());
    if (2.0 * plane > rows)
      q = std::max(1, std::min((int)lround(sqrt(plane * sqrt(plane) / rows)), nblk / 4));
  }
  bool ran = true;
  if (q > 1) {
    const int S = (nblk + q - 1) / q;
    std::vector<int> sb((size_t)S + 1), sr((size_t)S + 1);
    for (int k = 0; k <= S; k++) {
      sb[k] = (int)((long long)nblk * k / S);
      sr[k] = k < S ? row0[sb[k]] : nNo;
    }
    ran = for_blocks(S, rp[nNo], [&](int k) {
      const int r0 = sr[k], r1 = sr[k + 1];
      std::vector<signed char> mark((size_t)(r1 - r0), -1);  // last pass that saw a row
      const auto seen = [&](int i) -> signed char & { return mark[i - r0]; };
      int *const o = order.data() + r0;
      int start = r0;
      for (int pass = 0; pass < 2; pass++) {
        // pass 0 finds the far end, pass 1 orders the rows from there
        int n = 0, next = r0;
        while (n < r1 - r0) {
          int at = n;
          if (n == 0 && start < r1) {
            o[n++] = start;
            seen(start) = (signed char)pass;
          } else {
            while (seen(next) == pass) next++;
            o[n++] = next;
            seen(next) = (signed char)pass;
          }
          for (; at < n; at++)
            for (int j = rp[o[at]]; j < rp[o[at] + 1]; j++) {
              const int c = cp[j];
              if (c >= r0 && c < r1 && seen(c) != pass) {
                seen(c) = (signed char)pass;
                o[n++] = c;
              }
            }
        }
        if (n > 0) start = o[n - 1];
      }
      cut(r0, r1, sb[k], sb[k + 1]);
      // the rows of each block by number; at most nblk / S + 1 < 128 blocks
      std::vector<int> at(row0.begin() + sb[k], row0.begin() + sb[k + 1]);
      for (int b = sb[k]; b < sb[k + 1]; b++)
        for (int i = row0[b]; i < (b + 1 < sb[k + 1] ? row0[b + 1] : r1); i++)
          seen(order[i]) = (signed char)(b - sb[k]);
      for (int i = r0; i < r1; i++) order[at[seen(i)]++] = i;
    });
    if (!ran) throw std::bad_alloc();
  }
  // rows of each block by decreasing length, then number: slices and their steps
  std::vector<int> &sbase = H.sbase, &slotRow = H.slotRow, &slen = H.slen;
  sbase.assign((size_t)nblk + 1, 0);
  for (int b = 0; b < nblk; b++) {
    sbase[b + 1] = sbase[b] + (row0[b + 1] - row0[b] + RW - 1) / RW;
    H.nslMax = std::max(H.nslMax, sbase[b + 1] - sbase[b]);
  }
  const int nS = sbase[nblk];
  slotRow.assign((size_t)nS * RW, -1);
  slen.assign(nS, 1);
  std::vector<int> wst((size_t)nblk * W, 0);
  ran = for_blocks(nblk, nNo, [&](int b) {
    const int r0 = row0[b], r1 = row0[b + 1];
    int *const o = order.data() + r0;
    int longest = 0;
    for (int k = 0; k < r1 - r0; k++) longest = std::max(longest, rp[o[k] + 1] - rp[o[k]]);
    std::vector<int> at((size_t)longest + 2, 0);  // first place of each length, longest first
    for (int k = 0; k < r1 - r0; k++) at[longest - (rp[o[k] + 1] - rp[o[k]]) + 1]++;
    for (int l = 0; l < longest; l++) at[l + 1] += at[l];
    for (int k = 0; k < r1 - r0; k++)
      slotRow[(size_t)sbase[b] * RW + at[longest - (rp[o[k] + 1] - rp[o[k]])]++] = o[k];
    for (int s = sbase[b]; s < sbase[b + 1]; s++) {
      const int i = slotRow[(size_t)s * RW];  // the slice's longest row
      slen[s] = std::max(1, (rp[i + 1] - rp[i] + L - 1) / L);
      wst[(size_t)b * W + (s - sbase[b]) % W] += slen[s];
    }
  });
  if (!ran) throw std::bad_alloc();
  std::vector<int> &wbase = H.wbase;
  wbase.assign((size_t)nblk * W + 1, 0);
  long long steps = 0;
  for (size_t k = 0; k < wst.size(); k++) {
    wbase[k] = (int)steps;
    steps += wst[k];
    H.stMax = std::max(H.stMax, wst[k]);
    if (steps > (1LL << 31) / 32 - 1) return;
  }
  wbase[wst.size()] = (int)steps;
  // slices: their first steps in their warp's order, and in steps of their own
  // from multiples of 8
  H.sst.assign(nS, 0);
  H.soff.assign((size_t)nS + 1, 0);
  long long steps8 = 0;
  std::vector<int> wgr((size_t)nblk * W, 0);
  for (int b = 0; b < nblk; b++) {
    int next[W];
    for (int w = 0; w < W; w++) next[w] = wbase[(size_t)b * W + w];
    for (int s = sbase[b]; s < sbase[b + 1]; s++) {
      const int w = (s - sbase[b]) % W, g = (slen[s] + 7) / 8;
      H.sst[s] = next[w];
      next[w] += slen[s];
      H.soff[s] = (int)steps8;
      steps8 += 8 * g;
      wgr[(size_t)b * W + w] += g;
      if (steps8 > (1LL << 31) / 32 - 1 || steps8 - H.soff[sbase[b]] > kGrpOff) return;
    }
  }
  H.soff[nS] = (int)steps8;
  H.steps8 = steps8;
  for (int g : wgr) H.grpMax = std::max(H.grpMax, g);
  H.ok = true;
}

// The same on the graph's own numbering: breadth-first from a far end, which is
// where the search from row 0 ends.  A block of consecutive rows then lies
// together whatever numbering the mesh came with.
static void part_host_graph(int nNo, const std::vector<int> &rp, const std::vector<int> &cp,
                            int sms, PartHost &H) {
  std::vector<int> row((size_t)nNo), num((size_t)nNo, -1);  // row of a number, number of a row
  int start = 0;
  for (int pass = 0; pass < 2; pass++) {
    std::fill(num.begin(), num.end(), -1);
    int n = 0, next = 0;
    while (n < nNo) {
      int at = n;
      if (n > 0) {
        while (num[next] >= 0) next++;
        start = next;
      }
      num[start] = n;
      row[n++] = start;
      for (; at < n; at++)
        for (int j = rp[row[at]]; j < rp[row[at] + 1]; j++)
          if (num[cp[j]] < 0) {
            num[cp[j]] = n;
            row[n++] = cp[j];
          }
    }
    start = row[nNo - 1];
  }
  std::vector<int> rpn((size_t)nNo + 1), cpn((size_t)rp[nNo]);
  for (int i = 0; i < nNo; i++) rpn[i + 1] = rpn[i] + rp[row[i] + 1] - rp[row[i]];
  const int nb = 64;
  const bool ran = for_blocks(nb, rp[nNo], [&](int b) {
    for (int i = (int)((long long)nNo * b / nb); i < (int)((long long)nNo * (b + 1) / nb); i++)
      for (int j = rp[row[i]], k = rpn[i]; j < rp[row[i] + 1]; j++) cpn[k++] = num[cp[j]];
  });
  if (!ran) throw std::bad_alloc();
  part_host(nNo, rpn, cpn, sms, H);
  for (int &i : H.slotRow)
    if (i >= 0) i = row[i];
}

// ---- the halos and the steps' columns, on the device
struct PartBuild {
  const int *rowPtr, *colPtr, *sbase, *slen, *sst, *slotRow;
  int *rowSlot;  // slot of each row
  // per block and 32 slots: which of them are in its halo, and how many of
  // its halo's slots come before
  uint2 *words;
  int *count;  // halo entries of each block
  int nw, L;
  const int *hoff;
  int *halo, *src;
  unsigned short *lcol;
};
constexpr int kBuildThreads = 512;

__global__ void k_part_slots(long long n, const int *__restrict__ slotRow, int *rowSlot) {
  for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < n;
       k += (long long)gridDim.x * blockDim.x) {
    const int row = slotRow[k];
    if (row >= 0) rowSlot[row] = (int)k;
  }
}

// halo of block blockIdx.x: 8 lanes per row set the bits of its columns that
// are not the block's own
__global__ void __launch_bounds__(kBuildThreads) k_part_mark(PartBuild B) {
  __shared__ int sh[32];
  const int b = blockIdx.x, tid = threadIdx.x, RW = 32 / B.L;
  const int g0 = B.sbase[b] * RW, own = B.sbase[b + 1] * RW - g0;
  uint2 *w = B.words + (size_t)b * B.nw;
  for (int k = tid; k < B.nw; k += kBuildThreads) w[k] = make_uint2(0u, 0u);
  __syncthreads();
  for (int k = tid >> 3; k < own; k += kBuildThreads >> 3) {
    const int row = __ldg(B.slotRow + g0 + k);
    if (row < 0) continue;
    const int e = __ldg(B.rowPtr + row + 1);
    for (int j = __ldg(B.rowPtr + row) + (tid & 7); j < e; j += 8) {
      const int c = __ldg(B.rowSlot + __ldg(B.colPtr + j));
      if ((unsigned)(c - g0) < (unsigned)own) continue;
      const unsigned m = 1u << (c & 31);
      unsigned *x = &w[c >> 5].x;
      if (!(*(volatile unsigned *)x & m)) atomicOr(x, m);
    }
  }
  __syncthreads();
  int run = 0;
  for (int k0 = 0; k0 < B.nw; k0 += kBuildThreads) {
    const int k = k0 + tid;
    int tot;
    const int n = k < B.nw ? __popc(*(volatile unsigned *)&w[k].x) : 0;
    const int ex = block_scan_excl(n, sh, tot);
    if (k < B.nw) w[k].y = (unsigned)(run + ex);
    run += tot;
    __syncthreads();
  }
  if (tid == 0) B.count[b] = run;
}

// halo (by slot: neighbouring entries of it are neighbours in the vectors) and,
// a warp per slice, sources and window columns
__global__ void __launch_bounds__(kBuildThreads) k_part_fill(PartBuild B) {
  const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, RW = 32 / B.L;
  const int s0 = B.sbase[b], g0 = s0 * RW, own = B.sbase[b + 1] * RW - g0;
  const uint2 *__restrict__ w = B.words + (size_t)b * B.nw;
  for (int k = tid; k < B.nw; k += kBuildThreads) {
    const uint2 v = w[k];
    int *out = B.halo + B.hoff[b] + v.y;
    for (unsigned m = v.x; m; m &= m - 1) *out++ = 32 * k + __ffs(m) - 1;
  }
  const int g = lane / B.L, l = lane - g * B.L;
  for (int s = tid >> 5; s < own / RW; s += kBuildThreads >> 5) {
    const int me = s * RW + g, row = __ldg(B.slotRow + g0 + me), len = __ldg(B.slen + s0 + s);
    const int j0 = row >= 0 ? __ldg(B.rowPtr + row) : 0;
    const int n = row >= 0 ? __ldg(B.rowPtr + row + 1) - j0 : 0;
    const size_t P = (size_t)__ldg(B.sst + s0 + s) * 32 + lane;
#pragma unroll 4
    for (int t = 0; t < len; t++) {
      int src = -1, c = me;  // padding: zero block on the row's own entry
      if (t * B.L + l < n) {
        src = j0 + t * B.L + l;
        const int slot = __ldg(B.rowSlot + __ldg(B.colPtr + src));
        c = slot - g0;
        if ((unsigned)c >= (unsigned)own) {
          const uint2 v = w[slot >> 5];
          c = own + (int)v.y + __popc(v.x & ((1u << (slot & 31)) - 1u));
        }
      }
      B.src[P + (size_t)t * 32] = src;
      B.lcol[P + (size_t)t * 32] = (unsigned short)c;
    }
  }
}

// v appended to the image of the device buffer at a 16-byte boundary; its offset
template <class T>
static size_t append(std::vector<unsigned char> &img, const std::vector<T> &v) {
  const size_t at = (img.size() + 15) & ~(size_t)15;
  img.resize(at + sizeof(T) * v.size());
  if (!v.empty()) memcpy(img.data() + at, v.data(), sizeof(T) * v.size());
  return at;
}

static PartBuild part_build(const gsls_lhs *lhs, const RowPart &p) {
  const PartArgs a = part_args(p);
  PartBuild B{};
  B.rowPtr = lhs->d_rowPtr.as<int>();
  B.colPtr = lhs->d_colPtr.as<int>();
  B.sbase = a.sbase;
  B.slen = a.slen;
  B.sst = a.sst;
  B.slotRow = a.slotRow;
  B.nw = (int)((p.slots + 31) / 32);
  B.L = p.L;
  B.words = p.tmp.as<uint2>();
  B.rowSlot = reinterpret_cast<int *>(B.words + (size_t)B.nw * p.nblk);
  B.count = B.rowSlot + lhs->nNo;
  return B;
}

// the halos as bits in p.tmp; *ok false when there is no memory for them
static int part_mark(gsls_lhs *lhs, RowPart &p, bool *ok) {
  const size_t nw = ((size_t)p.slots + 31) / 32;
  *ok = p.tmp.try_alloc(nw * p.nblk * sizeof(uint2) + sizeof(int) * ((size_t)lhs->nNo + p.nblk));
  if (!*ok) return GSLS_OK;
  const PartBuild B = part_build(lhs, p);
  k_part_slots<<<4 * num_sms(), 256, 0, lhs->stream>>>(p.slots, B.slotRow, B.rowSlot);
  GSLS_CHECK_LAUNCH();
  k_part_mark<<<p.nblk, kBuildThreads, 0, lhs->stream>>>(B);
  GSLS_CHECK_LAUNCH();
  return GSLS_OK;
}

int part_setup(gsls_lhs *lhs, bool graph) {
  RowPart &p = lhs->ws.part[graph];
  if (p.built) return GSLS_OK;
  p.built = true;
  cudaStream_t st = lhs->stream;
  PartHost H;
  std::vector<unsigned char> img;
  try {
    (graph ? part_host_graph : part_host)(lhs->nNo, lhs->h_rowPtr, lhs->h_colPtr, num_sms(), H);
    if (!H.ok) return GSLS_OK;
    p.hoff.assign((size_t)H.nblk + 1, 0);
    img.reserve(sizeof(int) * (H.wbase.size() + 2 * H.soff.size() + 2 * H.sbase.size() +
                               H.slen.size() + H.slotRow.size()) + 256);
    p.off[0] = append(img, H.wbase);
    p.off[1] = append(img, H.sbase);
    p.off[2] = append(img, H.slen);
    p.off[3] = append(img, p.hoff);
    p.off[4] = append(img, H.slotRow);
    p.off[5] = append(img, H.sst);
    p.off[6] = append(img, H.soff);
  } catch (const std::bad_alloc &) {
    return GSLS_OK;
  }
  if (!p.buf.try_alloc(img.size() + 16)) return GSLS_OK;
  GSLS_CUDA(cudaMemcpyAsync(p.buf.p, img.data(), img.size(), cudaMemcpyHostToDevice, st));
  p.L = H.L;
  p.nslMax = H.nslMax;
  p.stMax = H.stMax;
  p.grpMax = H.grpMax;
  p.nS = (int)H.slen.size();
  p.steps8 = H.steps8;
  p.slots = (long long)H.slotRow.size();
  p.steps = (long long)H.wbase.back();
  p.nblk = H.nblk;
  bool ok;
  GSLS_TRY(part_mark(lhs, p, &ok));
  if (ok)
    GSLS_CUDA(cudaMemcpyAsync(p.hoff.data() + 1, part_build(lhs, p).count,
                              sizeof(int) * (size_t)p.nblk, cudaMemcpyDeviceToHost, st));
  GSLS_CUDA(cudaStreamSynchronize(st));  // also: img goes out of scope
  if (ok) {
    // a compact block of r rows has about (r^1/3 + 2)^3 - r neighbours; meshes
    // numbered plane by plane have up to 3.3 times as many in all (the CEP
    // slab), the same meshes numbered at random 5 to 13 times
    double halos = 0.0;
    const double r = (double)lhs->nNo / p.nblk;
    for (int b = 0; b < p.nblk; b++) halos += p.hoff[b + 1];
    p.scattered = halos > 4.0 * p.nblk * (pow(cbrt(r) + 2.0, 3.0) - r);
  }
  for (int b = 0; ok && b < p.nblk; b++) {
    const long long win = (long long)(H.sbase[b + 1] - H.sbase[b]) * (32 / p.L) + p.hoff[b + 1];
    ok = win <= 65535;  // 16-bit columns; bounds the sum of the halos too
    if (!ok) break;
    p.winMax = std::max(p.winMax, (int)win);
    p.hoff[b + 1] += p.hoff[b];
  }
  if (!ok) {
    p.buf.release();
    p.tmp.release();
    return GSLS_OK;
  }
  GSLS_CUDA(cudaMemcpyAsync(p.buf.as<unsigned char>() + p.off[3], p.hoff.data(),
                            sizeof(int) * p.hoff.size(), cudaMemcpyHostToDevice, st));
  p.ok = true;
  return GSLS_OK;
}

int part_fill(gsls_lhs *lhs, RowPart &p) {
  if (p.tab.p) return GSLS_OK;
  const size_t nh = (size_t)p.hoff[p.nblk], n = (size_t)p.steps * 32;
  bool ok = p.tab.try_alloc(sizeof(int) * (nh + n) + sizeof(short) * n + 16);
  if (ok && !p.tmp.p) GSLS_TRY(part_mark(lhs, p, &ok));
  if (!ok) {
    p.ok = false;
    p.tab.release();
    p.buf.release();
    p.tmp.release();
    return GSLS_OK;
  }
  const PartArgs a = part_args(p);
  PartBuild B = part_build(lhs, p);
  B.hoff = a.hoff;
  B.halo = const_cast<int *>(a.halo);
  B.src = const_cast<int *>(a.src);
  B.lcol = const_cast<unsigned short *>(a.lcol);
  k_part_fill<<<p.nblk, kBuildThreads, 0, lhs->stream>>>(B);
  GSLS_CHECK_LAUNCH();
  GSLS_CUDA(cudaStreamSynchronize(lhs->stream));
  p.tmp.release();
  return GSLS_OK;
}

PartArgs part_args(const RowPart &p) {
  PartArgs a{};
  const unsigned char *d = p.buf.as<unsigned char>();
  const auto ints = [&](int k) { return reinterpret_cast<const int *>(d + p.off[k]); };
  a.wbase = ints(0);
  a.sbase = ints(1);
  a.slen = ints(2);
  a.hoff = ints(3);
  a.slotRow = ints(4);
  a.sst = ints(5);
  a.soff = ints(6);
  a.halo = p.tab.as<int>();
  if (a.halo) {
    a.src = a.halo + p.hoff[p.nblk];
    a.lcol = reinterpret_cast<const unsigned short *>(a.src + (size_t)p.steps * 32);
  }
  a.nblk = p.nblk;
  a.L = p.L;
  a.winMax = p.winMax;
  a.nslMax = p.nslMax;
  a.stMax = p.stMax;
  a.grpMax = p.grpMax;
  a.nS = p.nS;
  a.nsteps8 = p.steps8;
  a.nslots = p.slots;
  a.nsteps = p.steps;
  return a;
}

}  // namespace gsls
