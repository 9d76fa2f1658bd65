// Grid-wide barrier and reductions of the persistent (cooperative) Krylov
// kernels.  Every wait is bounded: after `limit` polls (kBarSpinDefault
// unless set, each a 20 ns sleep plus an L2 round trip: seconds at most; the
// host can lower it with gsls_set_wait_limit) the waiting block sets the
// error word and returns false, and every other block leaves at its next
// poll or at its own limit, so a launch that lost a block ends with an
// error status instead of hanging.
#pragma once

#include "gsls_fixsum.cuh"
#include "gsls_internal.cuh"

namespace gsls {

struct GridBar {
  unsigned count;  // arrivals, monotonic within one launch (zeroed before it)
  unsigned pad;
  int err, pad2;
};

// Barrier number `epoch` (1, 2, ...) of the launch: every block adds one
// arrival (release at GPU scope), and the count is polled with acquire loads
// until all nblk * epoch arrivals are in; no reset, so the last arriver has
// nothing more to publish.  The error word is polled every 32 iterations.
__device__ __forceinline__ unsigned ld_acquire_gpu(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
// Grid-wide sum that is also a grid barrier, split into arrive and wait so
// that a block can work between the two.  Thread 0 writes the block's partial
// and then adds one to a counter (release); lane 0 of warp 0 polls the counter
// (acquire), and warp 0 adds the partials.  Two sets of partials take turns:
// a block that writes set e & 1 has passed round e - 1, so every block has
// read round e - 2.  Before a launch the counter is zero (one memset of the
// GridBar).  The counter alone takes 1.2 us a round on 152 blocks; one slot
// per block polled by every block took 4.1 us with its sum, a master block
// that adds and publishes 3.3 us.
//
// Sums are in integer arithmetic (gsls_fixsum.cuh): with FP64 adds a block
// sum of 16 warps took 1.3 us and the last one over 152 partials 0.9 us.
// What every warp would repeat in FP64 (quotients, conversions) belongs on
// lane 0 of warp 0, which shares it.
struct GridRedBuf {
  GridBar bar;
  int4 part[2 * 256];  // (exponent, limbs) of each block
};
struct GridRed {
  GridRedBuf *buf;
  unsigned nblk, limit;  // nblk <= 256
};

__device__ __forceinline__ void grid_red_publish(const GridRed &g, unsigned epoch, int e,
                                                 const int S[3]) {
  __stcg(g.buf->part + (epoch & 1u) * 256 + blockIdx.x, make_int4(e, S[0], S[1], S[2]));
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&g.buf->bar.count) : "memory");
}

// The functions below stay out of line: a persistent kernel that inlines them
// at every use grows past the instruction cache, and each of its phases then
// waits for instruction fetches (the windowed CG at 85 KB of code: 14,000
// cycles for a wait of 4,000).  They take and return values only: an argument
// by reference lives in local memory, which the matrix stream keeps evicting
// from L1.

// FP32: sum of the block in FP32 (at most 32 warps)
static __device__ __noinline__ void grid_red_arrive(float v, GridRed g, unsigned epoch) {
  __shared__ float s_w[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll 1
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (lane == 0) s_w[wid] = v;
  __syncthreads();
  if (wid == 0) {
    float b = lane < nw ? s_w[lane] : 0.f;
#pragma unroll 1
    for (int o = 16; o > 0; o >>= 1) b += __shfl_xor_sync(0xffffffffu, b, o);
    if (lane == 0) {
      const unsigned long long u = (unsigned long long)__double_as_longlong(double(b));
      const int e = max(fix_exp(u), 1);
      int S[3];
      fix_limbs(u, e, S);
      grid_red_publish(g, epoch, e, S);
    }
  }
}

// FP64: at most 256 threads with a value other than zero (limb sums stay
// below 2^31)
static __device__ __noinline__ void grid_red_arrive(double v, GridRed g, unsigned epoch) {
  __shared__ int s_e[32], s_l[32][3];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const unsigned long long u = (unsigned long long)__double_as_longlong(v);
  const int we = __reduce_max_sync(0xffffffffu, fix_exp(u));
  if (lane == 0) s_e[wid] = we;
  __syncthreads();
  const int e = max(1, __reduce_max_sync(0xffffffffu, lane < nw ? s_e[lane] : 0));
  int S[3];
  fix_limbs(u, e, S);
#pragma unroll
  for (int k = 0; k < 3; k++) S[k] = __reduce_add_sync(0xffffffffu, S[k]);
  if (lane < 3) s_l[wid][lane] = lane == 0 ? S[0] : lane == 1 ? S[1] : S[2];
  __syncthreads();
  if (wid == 0) {
#pragma unroll
    for (int k = 0; k < 3; k++) S[k] = __reduce_add_sync(0xffffffffu, lane < nw ? s_l[lane][k] : 0);
    if (lane == 0) grid_red_publish(g, epoch, e, S);
  }
}

// a round without a value
__device__ __forceinline__ void grid_bar_arrive(GridRed g) {
  __syncthreads();
  if (threadIdx.x == 0)
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&g.buf->bar.count) : "memory");
}

// Called by warp 0: waits until all blocks have arrived at round `epoch`;
// *okp (shared memory) is 0 when a wait ran out, here or in another block.
static __device__ __noinline__ void grid_bar_wait(GridRed g, unsigned epoch, int *okp) {
  if ((threadIdx.x & 31) == 0) {
    int ok = 1;
    const unsigned target = epoch * g.nblk;
    unsigned it = 0;
    while (ld_acquire_gpu(&g.buf->bar.count) < target) {
      ++it;
      if ((it & 31u) == 0u && *(volatile int *)&g.buf->bar.err) {
        ok = 0;
        break;
      }
      if (it >= g.limit) {
        atomicExch(&g.buf->bar.err, 1);
        ok = 0;
        break;
      }
      if (it > 64u) __nanosleep(20);
    }
    *okp = ok;
  }
  __syncwarp();
}

// Called by warp 0: grid_bar_wait, then the total of the round on every lane.
// A NaN or infinite addend gives a NaN total.
static __device__ __noinline__ double grid_red_total(GridRed g, unsigned epoch, int *okp) {
  const int lane = threadIdx.x & 31;
  grid_bar_wait(g, epoch, okp);
  const int4 *part = g.buf->part + (epoch & 1u) * 256;
  constexpr int kPer = 5;  // 160 blocks a turn
  int E = 1;
  long long H = 0;
  unsigned Lo = 0;
  for (unsigned k0 = 0; k0 < g.nblk; k0 += 32 * kPer) {
    int4 q[kPer];
#pragma unroll
    for (int k = 0; k < kPer; k++)
      q[k] = k0 + lane + 32u * k < g.nblk ? __ldcg(part + k0 + lane + 32 * k)
                                          : make_int4(0, 0, 0, 0);
    int e = E;
#pragma unroll
    for (int k = 0; k < kPer; k++) e = max(e, q[k].x);
    e = __reduce_max_sync(0xffffffffu, e);
    if (k0 > 0 && e > E) {
      // the sum of the earlier turns, relative to the larger exponent
      int lo = (int)Lo;
      fix_down(H, lo, e - E);
      Lo = (unsigned)lo;
    }
    E = e;
#pragma unroll 1
    for (int k = 0; k < kPer; k++) {
      const int4 p = k == 0 ? q[0] : k == 1 ? q[1] : k == 2 ? q[2] : k == 3 ? q[3] : q[4];
      const int S[3] = {p.y, p.z, p.w};
      long long h;
      int l;
      fix_align(p.x, S, E, h, l);
      H += h;
      Lo += (unsigned)l;
    }
    H += Lo >> 23;
    Lo &= kFixMask;
  }
  // |H| < 2^58: 26 + 26 bits and the signed rest
  const unsigned a = __reduce_add_sync(0xffffffffu, (unsigned)(H & 0x3ffffff));
  const unsigned b = __reduce_add_sync(0xffffffffu, (unsigned)((H >> 26) & 0x3ffffff));
  const int c = __reduce_add_sync(0xffffffffu, (int)(H >> 52));
  Lo = __reduce_add_sync(0xffffffffu, Lo);
  const long long T = ((long long)c << 52) + ((long long)b << 26) + (long long)a;
  return E == 0x7ff ? __longlong_as_double(0x7ff8000000000000ll) : fix_double(T, Lo, E);
}

// a / b out of line (the Krylov scalars)
static __device__ __noinline__ double grid_div(double a, double b) { return fix_div(a, b); }

}  // namespace gsls
