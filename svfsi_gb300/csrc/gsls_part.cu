// Host construction of the row partition (gsls_part.cuh).
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <new>
#include <thread>

#include "gsls_part.cuh"

namespace gsls {

// f(b, scratch) for every block b, on up to 8 host threads; the result of a
// block depends on b only, and it leaves the n scratch entries at -1.  False
// when host memory could not be had.
template <class F>
static bool for_blocks(int nblk, long long work, size_t n, const F &f) {
  const unsigned hw = std::thread::hardware_concurrency();
  const int T = (int)std::min<long long>(std::min({nblk, 8, hw ? (int)hw : 1}), 1 + work / 40000);
  std::atomic<int> next{0};
  std::atomic<bool> ok{true};
  const auto run = [&] {
    try {
      std::vector<int> scratch(n, -1);
      for (int b; (b = next.fetch_add(1)) < nblk;) f(b, scratch);
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

struct PartHost {
  int nblk = 0, L = 1, winMax = 0, nslMax = 0, stMax = 0, grpMax = 0;
  long long steps8 = 0;
  bool ok = false;
  std::vector<int> wbase, sst, soff, sbase, slen, hoff, halo, slotRow, src;
  std::vector<unsigned short> lcol;
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
    ran = for_blocks(S, rp[nNo], (size_t)nNo, [&](int k, std::vector<int> &seen) {
      const int r0 = sr[k], r1 = sr[k + 1];
      int *const o = order.data() + r0;
      int start = r0;
      for (int pass = 0; pass < 2; pass++) {
        // pass 0 finds the far end, pass 1 orders the rows from there
        int n = 0, next = r0;
        while (n < r1 - r0) {
          int at = n;
          if (n == 0 && start < r1) {
            o[n++] = start;
            seen[start] = pass;
          } else {
            while (seen[next] == pass) next++;
            o[n++] = next;
            seen[next] = pass;
          }
          for (; at < n; at++)
            for (int j = rp[o[at]]; j < rp[o[at] + 1]; j++) {
              const int c = cp[j];
              if (c >= r0 && c < r1 && seen[c] != pass) {
                seen[c] = pass;
                o[n++] = c;
              }
            }
        }
        if (n > 0) start = o[n - 1];
      }
      for (int i = r0; i < r1; i++) seen[i] = -1;
      cut(r0, r1, sb[k], sb[k + 1]);
    });
    if (!ran) throw std::bad_alloc();
  }
  // pass 1: rows of each block by decreasing length, slices and their steps
  std::vector<int> &sbase = H.sbase, &slotRow = H.slotRow, &slen = H.slen;
  sbase.assign((size_t)nblk + 1, 0);
  for (int b = 0; b < nblk; b++) sbase[b + 1] = sbase[b] + (row0[b + 1] - row0[b] + RW - 1) / RW;
  const int nS = sbase[nblk];
  slotRow.assign((size_t)nS * RW, -1);
  slen.assign(nS, 1);
  std::vector<int> rowSlot(nNo), blk(nNo);
  std::vector<int> wst((size_t)nblk * W, 0);
  ran = for_blocks(nblk, rp[nNo], 0, [&](int b, std::vector<int> &) {
    const int r0 = row0[b], r1 = row0[b + 1];
    std::vector<int> idx(order.begin() + r0, order.begin() + r1);
    std::sort(idx.begin(), idx.end());
    std::stable_sort(idx.begin(), idx.end(),
                     [&](int x, int y) { return rp[x + 1] - rp[x] > rp[y + 1] - rp[y]; });
    for (int k = 0; k < r1 - r0; k++) {
      slotRow[(size_t)sbase[b] * RW + k] = idx[k];
      rowSlot[idx[k]] = sbase[b] * RW + k;
      blk[idx[k]] = b;
    }
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
  // slices in steps of their own, from multiples of 8
  H.sst.assign(nS, 0);
  H.soff.assign((size_t)nS + 1, 0);
  long long steps8 = 0;
  std::vector<int> wgr((size_t)nblk * W, 0);
  for (int b = 0; b < nblk; b++)
    for (int s = sbase[b]; s < sbase[b + 1]; s++) {
      const int g = (slen[s] + 7) / 8;
      H.soff[s] = (int)steps8;
      steps8 += 8 * g;
      wgr[(size_t)b * W + (s - sbase[b]) % W] += g;
      if (steps8 > (1LL << 31) / 32 - 1 || steps8 - H.soff[sbase[b]] > kGrpOff) return;
    }
  H.soff[nS] = (int)steps8;
  H.steps8 = steps8;
  for (int g : wgr) H.grpMax = std::max(H.grpMax, g);
  // pass 2: halo of each block, sources and window columns of its steps
  std::vector<std::vector<int>> hl(nblk);
  std::vector<int> &src = H.src;
  std::vector<unsigned short> &lcol = H.lcol;
  src.assign((size_t)steps * 32, -1);
  lcol.assign((size_t)steps * 32, 0);
  std::vector<char> fit(nblk, 1);
  ran = for_blocks(nblk, rp[nNo], (size_t)nNo, [&](int b, std::vector<int> &loc) {
    const int r0 = row0[b], r1 = row0[b + 1], own = (sbase[b + 1] - sbase[b]) * RW;
    std::vector<int> &h = hl[b];
    for (int k = r0; k < r1; k++)
      for (int j = rp[order[k]]; j < rp[order[k] + 1]; j++)
        if (blk[cp[j]] != b && loc[cp[j]] < 0) {
          loc[cp[j]] = 0;
          h.push_back(cp[j]);
        }
    std::sort(h.begin(), h.end());
    if ((long long)own + (long long)h.size() > 65535) {
      fit[b] = 0;
      for (int c : h) loc[c] = -1;
      return;
    }
    for (size_t k = 0; k < h.size(); k++) loc[h[k]] = own + (int)k;
    std::vector<int> at(W);
    for (int w = 0; w < W; w++) at[w] = wbase[(size_t)b * W + w];
    for (int s = sbase[b]; s < sbase[b + 1]; s++) {
      const int w = (s - sbase[b]) % W, st0 = at[w];
      at[w] += slen[s];
      H.sst[s] = st0;
      for (int g = 0; g < RW; g++) {
        const int i = slotRow[(size_t)s * RW + g];
        const unsigned short me = (unsigned short)((s - sbase[b]) * RW + g);
        const int j0 = i >= 0 ? rp[i] : 0, len = i >= 0 ? rp[i + 1] - j0 : 0;
        for (int t = 0; t < slen[s] * L; t++) {
          const size_t P = (size_t)(st0 + t / L) * 32 + g * L + t % L;
          if (t >= len) {
            lcol[P] = me;  // padding: zero block on the row's own entry
            continue;
          }
          const int c = cp[j0 + t];
          src[P] = j0 + t;
          if (blk[c] == b)
            lcol[P] = (unsigned short)(rowSlot[c] - sbase[b] * RW);
          else
            lcol[P] = (unsigned short)loc[c];
        }
      }
    }
    for (int &c : h) {
      loc[c] = -1;
      c = rowSlot[c];
    }
  });
  if (!ran) throw std::bad_alloc();
  H.ok = true;
  H.hoff.assign((size_t)nblk + 1, 0);
  for (int b = 0; b < nblk; b++) {
    H.ok = H.ok && fit[b];
    H.hoff[b + 1] = H.hoff[b] + (int)hl[b].size();
    H.winMax = std::max(H.winMax, (sbase[b + 1] - sbase[b]) * RW + (int)hl[b].size());
    H.nslMax = std::max(H.nslMax, sbase[b + 1] - sbase[b]);
  }
  if (!H.ok) return;
  H.halo.reserve((size_t)H.hoff[nblk]);
  for (int b = 0; b < nblk; b++) H.halo.insert(H.halo.end(), hl[b].begin(), hl[b].end());
}

// v appended to the image of the device buffer at a 16-byte boundary; its offset
template <class T>
static size_t append(std::vector<unsigned char> &img, const std::vector<T> &v) {
  const size_t at = (img.size() + 15) & ~(size_t)15;
  img.resize(at + sizeof(T) * v.size());
  if (!v.empty()) memcpy(img.data() + at, v.data(), sizeof(T) * v.size());
  return at;
}

static int part_build(gsls_lhs *lhs, RowPart &p) {
  PartHost H;
  part_host(lhs->nNo, lhs->h_rowPtr, lhs->h_colPtr, num_sms(), H);
  p.ok = H.ok;
  if (H.ok) {
    std::vector<unsigned char> img;
    img.reserve(sizeof(int) * (H.wbase.size() + 2 * H.soff.size() + H.sbase.size() + H.slen.size() + H.hoff.size() +
                               H.halo.size() + H.slotRow.size() + H.src.size()) +
                2 * H.lcol.size() + 256);
    p.off[0] = append(img, H.wbase);
    p.off[1] = append(img, H.sbase);
    p.off[2] = append(img, H.slen);
    p.off[3] = append(img, H.hoff);
    p.off[4] = append(img, H.halo);
    p.off[5] = append(img, H.slotRow);
    p.off[6] = append(img, H.src);
    p.off[7] = append(img, H.lcol);
    p.off[8] = append(img, H.sst);
    p.off[9] = append(img, H.soff);
    if (!p.buf.try_alloc(img.size() + 16)) {
      p.ok = false;
      p.built = true;
      return GSLS_OK;
    }
    GSLS_CUDA(cudaMemcpyAsync(p.buf.p, img.data(), img.size(), cudaMemcpyHostToDevice,
                              lhs->stream));
    GSLS_CUDA(cudaStreamSynchronize(lhs->stream));  // img goes out of scope
    p.L = H.L;
    p.winMax = H.winMax;
    p.nslMax = H.nslMax;
    p.stMax = H.stMax;
    p.grpMax = H.grpMax;
    p.nS = (int)H.slen.size();
    p.steps8 = H.steps8;
    p.slots = (long long)H.slotRow.size();
    p.steps = (long long)H.wbase.back();
  }
  p.nblk = H.nblk;
  p.built = true;
  return GSLS_OK;
}

int part_setup(gsls_lhs *lhs) {
  RowPart &p = lhs->ws.part;
  if (p.built) return GSLS_OK;
  try {
    return part_build(lhs, p);
  } catch (const std::bad_alloc &) {
    p.ok = false;
    p.built = true;
    return GSLS_OK;
  }
}

PartArgs part_args(const RowPart &p) {
  PartArgs a;
  const unsigned char *d = p.buf.as<unsigned char>();
  const auto ints = [&](int k) { return reinterpret_cast<const int *>(d + p.off[k]); };
  a.wbase = ints(0);
  a.sbase = ints(1);
  a.slen = ints(2);
  a.hoff = ints(3);
  a.halo = ints(4);
  a.slotRow = ints(5);
  a.src = ints(6);
  a.sst = ints(8);
  a.soff = ints(9);
  a.lcol = reinterpret_cast<const unsigned short *>(d + p.off[7]);
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
