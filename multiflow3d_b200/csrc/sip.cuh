// solver = 1: pressure_1sweep (press.for:274-420) with Stone's strongly
// implicit procedure, sipsol(44) (sipsol.for:2-206), on the device.
//
// The ILU factorisation and the two substitutions are recurrences over the
// previous cell along j, i and k (the reference's ijk-1, ijk-nj, ijk-nij).
// A cell depends only on cells of a smaller i+j+k, so every cell of one
// hyperplane i+j+k = h can be formed at once with exactly the reference's
// operands and operation order.  Where a block's rows fit one cluster's
// warps, both substitutions run in one launch in which every warp carries a
// row segment and waits for its neighbours alone (k_sip_subst).  Small planes
// that this suits less - narrow and tall ones, very many blocks - are walked
// by one CTA each, hyperplane by hyperplane (k_sip_subst_col, _block), and
// larger planes take a launch per hyperplane, the whole sweep captured once
// in a CUDA graph.  The factors and the residual live in per-block arrays,
// for k_sip_subst in the order in which its warps read them (SipBlk), else
// over the ghost-inclusive box, i fastest, zero outside the interior (the
// reference zeroes its arrays and only ever writes interior cells).
// The correction pp is the level-1 phi of the
// multigrid storage, so the pressure update, the halo refresh of pp
// (exchange(44): its face values are the multigrid halo's) and
// calvel/calmas are the multigrid path's own kernels.
//
// The sweep loop's stopping test runs on the device (SipCtl): the sweeps of
// a call are queued without a host round trip, those past the stop return at
// once.  The summed |residual| of a sweep, which only steers that test, is
// reduced in a fixed order (deterministic, but not the reference's serial
// order: the test can differ only when a ratio lies within rounding of
// 0.001 or 1e-5).
#pragma once

namespace mf3d {

constexpr double kSipAlfa = 0.92;  // sipsol.for:31
constexpr double kSipSmall = 1e-20;

struct SipBlk {
  double *lb, *lw, *ls, *lpr, *un, *ue, *ut, *res;
  int nx, ny, nz;
  // segments of 32 columns per row of j, 0: plain layout.  With segments,
  // lane l of row j's segment q holds column i = 32q + l + 1, whose cell k it
  // forms at step t = k - 1 + l: element (((j-1)*nseg + q)*T + t)*32 + l with
  // T = sip_steps(nz), so that a warp reads a step's operands as one line and
  // successive steps as successive lines.  Slots without a cell hold 0.
  int nseg;
};
// steps of a row segment: nz + 31, in whole pairs of chunks (k_sip_subst)
constexpr int SIP_K = 4;  // steps per chunk
__host__ __device__ inline int sip_steps(int nz) { return (nz + 31 + 2 * SIP_K - 1) / (2 * SIP_K) * (2 * SIP_K); }
__device__ __forceinline__ long long sip_plain(const SipBlk &S, int i, int j, int k) {
  return ((long long)k * (S.ny + 2) + j) * (S.nx + 2) + i;
}
__device__ __forceinline__ long long sip_idx(const SipBlk &S, int i, int j, int k) {
  if (!S.nseg) return sip_plain(S, i, j, k);
  const int l = (i - 1) & 31;
  return (((long long)(j - 1) * S.nseg + ((i - 1) >> 5)) * sip_steps(S.nz) + (k - 1 + l)) * 32 + l;
}
// a's value at (i, j, k), 0 outside the interior
__device__ __forceinline__ double sip_at(const SipBlk &S, const double *a, int i, int j, int k) {
  return i < 1 || j < 1 || k < 1 || i > S.nx || j > S.ny || k > S.nz ? 0.0 : a[sip_idx(S, i, j, k)];
}

// The sweep loop of one call (sipsol.for:172-190's test), on the device.
// k_sip_sum moves `next` to `run`: the sweep's residual reads next, its
// substitutions and halo refresh read run.
struct SipCtl {
  double res1, relast;
  int run, next;
  int sweeps;       // of this call
  int pad;
  long long total;  // of the solve
};
__global__ void k_sip_begin(SipCtl *c, int first_call) {
  pdl_wait();
  c->res1 = 0.0;
  c->relast = 0.0;
  c->run = 0;
  c->next = 1;
  c->sweeps = 0;
  if (first_call) c->total = 0;
}

// One hyperplane i+j+k = h of the ILU factors (sipsol.for:79-101).
// Thread per (i, j) of every block.
__global__ void k_sip_factor(const SipBlk *__restrict__ sb, const BlkLev *__restrict__ bl,
                             const Tile *__restrict__ tiles, int h) {
  pdl_wait();
  const Tile t = tiles[blockIdx.x];
  const SipBlk S = sb[t.blk];
  const int q = t.i0 + threadIdx.x;
  if (q >= S.nx * S.ny) return;
  const int i = q % S.nx + 1, j = q / S.nx + 1, k = h - i - j;
  if (k < 1 || k > S.nz) return;
  const BlkLev &B = bl[t.blk];
  const Coef<double> cf(B);
  const double aw = cf.aw[i], ae = cf.ae[i], as = cf.as[j], an = cf.an[j], ab = cf.ab[k], at = cf.at[k];
  const double ap = -1.0 * (aw + ae + as + an + ab + at);
  const long long c = sip_idx(S, i, j, k);
  const double unb = sip_at(S, S.un, i, j, k - 1), ueb = sip_at(S, S.ue, i, j, k - 1), utb = sip_at(S, S.ut, i, j, k - 1);
  const double unw = sip_at(S, S.un, i - 1, j, k), uew = sip_at(S, S.ue, i - 1, j, k), utw = sip_at(S, S.ut, i - 1, j, k);
  const double uns = sip_at(S, S.un, i, j - 1, k), ues = sip_at(S, S.ue, i, j - 1, k), uts = sip_at(S, S.ut, i, j - 1, k);
  const double lb = ab / (1. + kSipAlfa * (unb + ueb));
  const double lw = aw / (1. + kSipAlfa * (unw + utw));
  const double ls = as / (1. + kSipAlfa * (ues + uts));
  const double p1 = kSipAlfa * (lb * unb + lw * unw);
  const double p2 = kSipAlfa * (lb * ueb + ls * ues);
  const double p3 = kSipAlfa * (lw * utw + ls * uts);
  const double lpr = 1. / (ap + p1 + p2 + p3 - lb * utb - lw * uew - ls * uns + kSipSmall);
  S.lb[c] = lb; S.lw[c] = lw; S.ls[c] = ls; S.lpr[c] = lpr;
  S.un[c] = (an - p1) * lpr;
  S.ue[c] = (ae - p2) * lpr;
  S.ut[c] = (at - p3) * lpr;
}

// The residual of pp (sipsol.for:137-147) over every interior cell, and
// each CTA's sum of |res| (a fixed tree) into part[blockIdx.x].
__global__ void __launch_bounds__(RW_TX *RW_RJ) k_sip_residual(const SipBlk *__restrict__ sb,
                                                               const BlkLev *__restrict__ bl,
                                                               const Tile *__restrict__ tiles,
                                                               double *__restrict__ part,
                                                               const SipCtl *__restrict__ ctl) {
  pdl_wait();
  if (!ctl->next) return;
  __shared__ double red[RW_RJ];
  const Tile t = tiles[blockIdx.x];
  const SipBlk S = sb[t.blk];
  const BlkLev &B = bl[t.blk];
  const Coef<double> cf(B);
  const double *__restrict__ fi = phi_of<double>(B);
  const double *__restrict__ su = rhs_of<double>(B);
  const int i = t.i0 + threadIdx.x, j = t.j0 + threadIdx.y;
  double acc = 0.0;
  if (i <= S.nx && j <= S.ny) {
    const int k1 = min(t.k0 + RW_KCH - 1, S.nz);
#pragma unroll 4
    for (int k = t.k0; k <= k1; ++k) {
      const double aw = cf.aw[i], ae = cf.ae[i], as = cf.as[j], an = cf.an[j], ab = cf.ab[k], at = cf.at[k];
      const double ap = -1.0 * (aw + ae + as + an + ab + at);
      const double r = (su[cell_off(B, i, j, k)] - ap * fi[cell_off(B, i, j, k)] - an * fi[cell_off(B, i, j + 1, k)] -
                        as * fi[cell_off(B, i, j - 1, k)] - ae * fi[cell_off(B, i + 1, j, k)] -
                        aw * fi[cell_off(B, i - 1, j, k)] - ab * fi[cell_off(B, i, j, k - 1)] -
                        at * fi[cell_off(B, i, j, k + 1)]);
      S.res[sip_idx(S, i, j, k)] = r;
      acc = acc + fabs(r);
    }
  }
  for (int o = 16; o > 0; o >>= 1) acc = acc + __shfl_xor_sync(0xffffffffu, acc, o);
  if (threadIdx.x == 0) red[threadIdx.y] = acc;
  __syncthreads();
  if (threadIdx.x == 0 && threadIdx.y == 0) {
    double v = 0.0;
    for (int r = 0; r < RW_RJ; ++r) v = v + red[r];
    part[blockIdx.x] = v;
  }
}

// The per-CTA sums added in index order by one CTA (a fixed tree), then
// the stopping test of sipsol.for on the sum.  After a wait of the
// substitutions gave up nothing runs any more: the call has failed.
__global__ void k_sip_sum(const double *__restrict__ part, int n, SipCtl *__restrict__ ctl, const int *err) {
  pdl_wait();
  __shared__ double s[1024];
  const int go = *(volatile const int *)err == ERR_SIP_WAIT ? 0 : ctl->next;
  double v = 0.0;
  if (go)
    for (int q = threadIdx.x; q < n; q += blockDim.x) v = v + part[q];
  s[threadIdx.x] = v;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) s[threadIdx.x] = s[threadIdx.x] + s[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x != 0) return;
  ctl->run = go;
  if (!go) {
    ctl->next = 0;
    return;
  }
  const double resab = s[0];
  if (ctl->sweeps == 0) ctl->res1 = resab;
  const double rsm = resab / (ctl->res1 + kSipSmall);
  const double reldif = fabs(rsm - ctl->relast);
  ctl->relast = rsm;
  ++ctl->sweeps;
  ++ctl->total;
  ctl->next = (rsm <= 0.001 || reldif <= 0.00001) ? 0 : 1;
}

// Forward substitution on hyperplane h (sipsol.for:149-157).  `run` is loaded
// beside the operands and looked at before the store: a launch is a chain of
// loads, and one more ahead of them cost 0.6 us of 2.9 (96x96x64, 3 calls of 4
// sweeps: 17.9 ms with it, 13.9 without).
__global__ void k_sip_forward(const SipBlk *__restrict__ sb, const Tile *__restrict__ tiles, int h,
                              const SipCtl *__restrict__ ctl) {
  pdl_wait();
  const int run = ctl->run;
  const Tile t = tiles[blockIdx.x];
  const SipBlk S = sb[t.blk];
  const int q = t.i0 + threadIdx.x;
  if (q >= S.nx * S.ny) return;
  const int i = q % S.nx + 1, j = q / S.nx + 1, k = h - i - j;
  if (k < 1 || k > S.nz) return;
  const long long c = sip_plain(S, i, j, k);
  const double r = (S.res[c] - S.lb[c] * S.res[sip_plain(S, i, j, k - 1)] - S.lw[c] * S.res[sip_plain(S, i - 1, j, k)] -
                    S.ls[c] * S.res[sip_plain(S, i, j - 1, k)]) *
                   S.lpr[c];
  if (run) S.res[c] = r;
}

// Backward substitution on hyperplane h and the correction of pp
// (sipsol.for:159-170).
__global__ void k_sip_backward(const SipBlk *__restrict__ sb, const BlkLev *__restrict__ bl,
                               const Tile *__restrict__ tiles, int h, const SipCtl *__restrict__ ctl) {
  pdl_wait();
  const int run = ctl->run;
  const Tile t = tiles[blockIdx.x];
  const SipBlk S = sb[t.blk];
  const int q = t.i0 + threadIdx.x;
  if (q >= S.nx * S.ny) return;
  const int i = q % S.nx + 1, j = q / S.nx + 1, k = h - i - j;
  if (k < 1 || k > S.nz) return;
  const long long c = sip_plain(S, i, j, k);
  const double r = S.res[c] - S.un[c] * S.res[sip_plain(S, i, j + 1, k)] - S.ue[c] * S.res[sip_plain(S, i + 1, j, k)] -
                   S.ut[c] * S.res[sip_plain(S, i, j, k + 1)];
  double *fi = phi_of<double>(bl[t.blk]);
  const long long e = cell_off(bl[t.blk], i, j, k);
  const double f = fi[e] + r;
  if (run) {
    S.res[c] = r;
    fi[e] = f;
  }
}

// Both substitutions of every block in one launch.  A block is a cluster of
// `cl` CTAs (cl = 1: a plain CTA), CTA r owning `rows` = ceil(ny/cl) rows of
// j, one warp per row segment of 32 columns (SipBlk).  Forward, a warp goes
// through its steps t = 0..T-1; at step t lane l forms cell k = t-l+1 from
// its own previous value (k-1), the lane to the left's (west: the same k one
// step earlier, by shuffle; lane 0 from the segment to the west) and the row
// to the south at the same step.  Backward it goes from T-1 down with the
// lane to the right and the row to the north.
// There is no barrier per step.  Warps work in chunks of SIP_K steps: a warp
// takes the chunk's values of its neighbours out of its own shared memory,
// runs the steps and leaves its values in its neighbours' (in the next CTA's
// across a slab's edge).  An empty slot holds kSipEmpty, a signalling NaN no
// arithmetic gives, so the value itself says that it is there: no fence lies
// on the way, which would wait for the operands in flight.  Where shared
// memory holds a slot for every step (RING false) that is all.  For longer
// lines (RING) the slots are rings: the reader empties them again, every D
// steps a warp publishes how far it is, and a writer waits until its readers
// are past the slots.  All warps of a cluster are resident and values only
// flow from lower to higher rows and segments (backward: the reverse), each
// step of a segment after the step 31 later of the one before, with more
// than 2D slots to spare, so every wait ends; each is bounded all the same.
// A lane's five operands of a step are loaded D steps ahead.  W, the warps a
// CTA can hold, is the smallest of 8, 16 and 32 with which a cluster holds the
// block: at 32 a thread has 64 registers.
// What bounds it is the chain: T/4 + ny chunks one after the other each way,
// each four steps of a shuffle and four dependent FP64 operations; DRAM and
// issue slots are nearly idle.  Eight blocks of 32^3: 70 us a sweep (cold),
// against 312 us for one CTA per block with two barriers per hyperplane and
// the operands one step ahead; the solve of 50 calls of 4 sweeps 65.2 -> 17.2
// ms.  A barrier per hyperplane over a cluster with operands by cp.async four
// steps ahead took 180 us; the rings' fences (RING) cost 8 % of the solve.
constexpr long long kSipEmpty = 0x7ff45a5a5a5a5a5aLL;
__host__ __device__ constexpr int sip_ring(int W) { return W == 32 ? 16 : 32; }  // ring slots
struct SipShared {
  int done[32];         // steps this CTA's warps have done (RING)
  int lo[32], hi[32];   // the same of the slab below's last row, the slab above's first
  // then per warp R slots of 32 values of the neighbouring row, by step, then
  // per warp R of the neighbouring segment's edge lane, by cell k; R = T or
  // sip_ring(W)
  __device__ __forceinline__ double *across(int w, int R) { return (double *)(this + 1) + (long long)w * R * 32; }
  __device__ __forceinline__ double *along(int w, int W, int R) {
    return (double *)(this + 1) + (long long)W * R * 32 + (long long)w * R;
  }
};
static inline size_t sip_smem(int warps, int R) { return sizeof(SipShared) + (size_t)warps * R * 33 * sizeof(double); }

// A waiting lane's look at the clock.  t0: when it began to wait (0: now),
// which it returns; 0 (and *err set) after kMaxWaitNs.
__device__ __noinline__ unsigned long long sip_patience(unsigned long long t0, int *err) {
  const unsigned long long t = global_ns();
  if (t0 == 0) return t;
  if (t - t0 <= kMaxWaitNs) return t0;
  atomicExch(err, ERR_SIP_WAIT);
  return 0;
}
// Whether the warp waits on.  Its lanes vote and shuffle together, so all of
// them give up when one does, whatever times they read.
__device__ __forceinline__ bool sip_wait_on(unsigned long long &t0, int *err) {
  t0 = sip_patience(t0, err);
  return __all_sync(0xffffffffu, t0 != 0);
}
// until every lane has read *p >= need (seen: the least of the last values
// read), the same for all lanes
__device__ __forceinline__ bool sip_credit(const int *p, int need, int &seen, bool cluster, int *err) {
  unsigned long long t0 = 0;
  while (seen < need) {
    int v;
    if (cluster) asm volatile("ld.acquire.cluster.shared::cta.s32 %0, [%1];" : "=r"(v) : "r"(smem_u32(p)) : "memory");
    else asm volatile("ld.acquire.cta.shared::cta.s32 %0, [%1];" : "=r"(v) : "r"(smem_u32(p)) : "memory");
    seen = __reduce_min_sync(0xffffffffu, v);
    if (seen < need && !sip_wait_on(t0, err)) return false;
  }
  return true;
}

// One direction of the warp `warp` (row j, segment q).  ring: the
// neighbouring row's `across` (null: none), far: it lies in another CTA;
// remote_done: where the row this warp reads from, in another CTA, looks for
// its progress (null: that row is this CTA's).  False when a wait gave up.
template <bool FWD, int W, int D, bool RING>
__device__ __forceinline__ bool sip_pass(const SipBlk &S, SipShared &sh, int warp, int nw, int q, int lane, int j,
                                         double *ring, bool far, const int *ring_done, int *remote_done, int *err) {
  constexpr int K = SIP_K;
  const int nz = S.nz, nseg = S.nseg, T = sip_steps(nz);
  const int R = RING ? sip_ring(W) : T, mask = RING ? R - 1 : -1;
  const bool row_in = FWD ? j > 1 : j < S.ny;
  const bool seg_in = FWD ? q > 0 : q < nseg - 1, seg_out = FWD ? q < nseg - 1 : q > 0;
  const bool takes = seg_in && lane == (FWD ? 0 : 31), gives = seg_out && lane == (FWD ? 31 : 0);
  const long long base = ((long long)(j - 1) * nseg + q) * T * 32 + lane + (FWD ? 0 : (long long)(T - 1) * 32);
  constexpr int dir = FWD ? 32 : -32;  // elements from step to step
  const double *a0 = S.res + base, *a1 = (FWD ? S.lb : S.un) + base, *a2 = (FWD ? S.lw : S.ue) + base,
               *a3 = (FWD ? S.ls : S.ut) + base, *a4 = S.lpr + base;
  double *out = S.res + base;
  volatile long long *mine = (volatile long long *)(sh.across(warp, R) + lane);
  volatile long long *edge = (volatile long long *)sh.along(warp, nw, R);
  volatile double *give = (volatile double *)sh.along(seg_out ? warp + (FWD ? 1 : -1) : warp, nw, R);
  const int *give_done = &sh.done[seg_out ? warp + (FWD ? 1 : -1) : warp];
  volatile double *to = ring + lane;
  // kz - 1 of step n = 0; columns past nx have no cell
  int kz = 32 * q + lane + 1 <= S.nx ? (FWD ? 0 : T - 1) - lane : FWD ? -(1 << 29) : (1 << 29);
  int seen = 0, seen_give = 0;
  unsigned long long t0 = 0;
  double x0[D], x1[D], x2[D], x3[D], x4[D];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    x0[d] = a0[d * dir]; x1[d] = a1[d * dir]; x2[d] = a2[d * dir]; x3[d] = a3[d * dir];
    if (FWD) x4[d] = a4[d * dir];
  }
  double prev = 0.0;
  for (int n0 = 0; n0 < T; n0 += D) {
#pragma unroll
    for (int c = 0; c < D; c += K) {
      const int slot0 = (n0 + c) & mask;
      // the neighbours' values of the chunk
      double nb[K], sd[K];
#pragma unroll
      for (int d = 0; d < K; ++d) nb[d] = sd[d] = 0.0;
      if (row_in) {
        for (;;) {
          bool there = true;
#pragma unroll
          for (int d = 0; d < K; ++d) {
            const long long v = mine[(slot0 + d) * 32];
            there = there && v != kSipEmpty;
            nb[d] = __longlong_as_double(v);
          }
          if (__all_sync(0xffffffffu, there)) break;
          if (!sip_wait_on(t0, err)) return false;
        }
        t0 = 0;
        if (RING)
#pragma unroll
          for (int d = 0; d < K; ++d) mine[(slot0 + d) * 32] = kSipEmpty;
      }
      if (seg_in) {
        for (;;) {
          bool there = true;
          if (takes)
#pragma unroll
            for (int d = 0; d < K; ++d) {
              const int k1 = kz + (FWD ? d : -d);
              if ((unsigned)k1 < (unsigned)nz) {
                const long long v = edge[k1 & mask];
                there = there && v != kSipEmpty;
                sd[d] = __longlong_as_double(v);
              }
            }
          if (__all_sync(0xffffffffu, there)) break;
          if (!sip_wait_on(t0, err)) return false;
        }
        t0 = 0;
        if (RING && takes)
#pragma unroll
          for (int d = 0; d < K; ++d) {
            const int k1 = kz + (FWD ? d : -d);
            if ((unsigned)k1 < (unsigned)nz) edge[k1 & mask] = kSipEmpty;
          }
      }
      double v[K];
#pragma unroll
      for (int d = 0; d < K; ++d) {
        double side = FWD ? __shfl_up_sync(0xffffffffu, prev, 1) : __shfl_down_sync(0xffffffffu, prev, 1);
        if (lane == (FWD ? 0 : 31)) side = sd[d];
        const bool cell = (unsigned)(kz + (FWD ? d : -d)) < (unsigned)nz;
        const int x = c + d;
        v[d] = FWD ? (x0[x] - x1[x] * prev - x2[x] * side - x3[x] * nb[d]) * x4[x]
                   : x0[x] - x1[x] * nb[d] - x2[x] * side - x3[x] * prev;
        if (!cell) v[d] = 0.0;
        prev = v[d];
      }
      if (ring) {
        if (RING && !sip_credit(ring_done, n0 + c + K - R, seen, far, err)) return false;
#pragma unroll
        for (int d = 0; d < K; ++d) to[(slot0 + d) * 32] = v[d];
      }
      if (seg_out) {
        // the edge lane's m-th cell is the reader's step m (backward: m + T-nz-31);
        // the reader is past cell m - R before cell m is written
        const int first = n0 + c - (FWD ? 31 : T - nz);  // m of the chunk's first step
        if (RING && !sip_credit(give_done, min(first + K, nz) - R + (FWD ? 0 : T - nz - 31), seen_give, false, err))
          return false;
        if (gives)
#pragma unroll
          for (int d = 0; d < K; ++d) {
            const int k1 = kz + (FWD ? d : -d);
            if ((unsigned)k1 < (unsigned)nz) give[k1 & mask] = v[d];
          }
      }
      // D steps on, their slots are read and emptied: publish it, before the
      // chunk's own global stores and the next loads
      if (RING && c == D - K) {
        __syncwarp();
        if (lane == 0) {
          if (remote_done) {
            asm volatile("fence.acq_rel.cluster;" ::: "memory");
            asm volatile("st.relaxed.cluster.s32 [%0], %1;" ::"l"(remote_done), "r"(n0 + D) : "memory");
          }
          asm volatile("st.release.cta.shared::cta.s32 [%0], %1;" ::"r"(smem_u32(&sh.done[warp])), "r"(n0 + D) : "memory");
        }
      }
#pragma unroll
      for (int d = 0; d < K; ++d)
        if ((unsigned)(kz + (FWD ? d : -d)) < (unsigned)nz) out[d * dir] = v[d];
      // the operands of the chunk D steps on (past the last: none)
      if (n0 + c + D < T) {
#pragma unroll
        for (int d = 0; d < K; ++d) {
          const int x = c + d, e = (D + d) * dir;
          x0[x] = a0[e]; x1[x] = a1[e]; x2[x] = a2[e]; x3[x] = a3[e];
          if (FWD) x4[x] = a4[e];
        }
      }
      a0 += K * dir; a1 += K * dir; a2 += K * dir; a3 += K * dir; a4 += K * dir; out += K * dir;
      kz += FWD ? K : -K;
    }
  }
  return true;
}

template <int W, int D, bool RING>
__global__ void __launch_bounds__(32 * W) k_sip_subst(const SipBlk *__restrict__ sb,
                                                      const SipCtl *__restrict__ ctl, int cl, int *err) {
  // testing aid: the first warp of the first block may be told to withhold its values
  const bool first = blockIdx.x == 0 && threadIdx.x < 32;
  const int hold = first && threadIdx.x == 0 ? *(volatile int *)&g_test_extra_tx : 0;
  pdl_wait();
  if (!ctl->run) return;
  extern __shared__ __align__(16) unsigned char sip_dyn[];
  SipShared &sh = *(SipShared *)sip_dyn;
  const SipBlk S = sb[blockIdx.x / cl];
  const int rank = blockIdx.x % cl, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int nseg = S.nseg, R = RING ? sip_ring(W) : sip_steps(S.nz);
  const int rows = (S.ny + cl - 1) / cl, j0 = rank * rows, nr = min(rows, S.ny - j0);  // nr <= 0: no row
  const int jr = warp / nseg, q = warp - jr * nseg, j = j0 + jr + 1;
  const bool mine = nr > 0 && jr < nr;
  SipShared *above = nullptr, *below = nullptr;  // the slabs of higher and of lower rows
  if (cl > 1) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    if (mine && jr == nr - 1 && j < S.ny) above = cluster.map_shared_rank(&sh, rank + 1);
    if (mine && jr == 0 && rank > 0) below = cluster.map_shared_rank(&sh, rank - 1);
  }
  auto sync = [&] {
    __syncthreads();
    if (cl > 1) cluster_sync_all();
  };
  auto clear = [&] {
    for (int e = threadIdx.x; e < nw * R * 33; e += blockDim.x) ((long long *)(&sh + 1))[e] = kSipEmpty;
    if (threadIdx.x < 32) sh.done[threadIdx.x] = sh.lo[threadIdx.x] = sh.hi[threadIdx.x] = 0;
    sync();
  };
  clear();
  bool ok = true;
  if (first) ok = __shfl_sync(0xffffffffu, hold ? atomicExch(&g_test_extra_tx, 0) : 0, 0) == 0;
  if (mine && ok) {
    const bool up = jr < nr - 1;  // the row above is this CTA's
    ok = sip_pass<true, W, D, RING>(S, sh, warp, nw, q, lane, j,
                                    above ? above->across(q, R) : up ? sh.across(warp + nseg, R) : nullptr,
                                    above != nullptr, above ? &sh.hi[q] : &sh.done[up ? warp + nseg : 0],
                                    below ? &below->hi[q] : nullptr, err);
  }
  sync();
  clear();
  if (mine && ok)
    sip_pass<false, W, D, RING>(S, sh, warp, nw, q, lane, j,
                                below ? below->across((rows - 1) * nseg + q, R)  // the slab below is full
                                : jr > 0 ? sh.across(warp - nseg, R) : nullptr,
                                below != nullptr, below ? &sh.lo[q] : &sh.done[jr > 0 ? warp - nseg : 0],
                                above ? &above->lo[q] : nullptr, err);
  sync();  // no CTA leaves while another may still write its shared memory
}

// pp += the backward substitution's result (sipsol.for:159-170), of every
// interior cell: apart from the substitutions, whose few CTAs the scattered
// accesses of the colour-split layout would bind.
__global__ void __launch_bounds__(RW_TX *RW_RJ) k_sip_add(const SipBlk *__restrict__ sb, const BlkLev *__restrict__ bl,
                                                          const Tile *__restrict__ tiles,
                                                          const SipCtl *__restrict__ ctl) {
  pdl_wait();
  if (!ctl->run) return;
  const Tile t = tiles[blockIdx.x];
  const SipBlk S = sb[t.blk];
  const BlkLev &B = bl[t.blk];
  double *__restrict__ fi = phi_of<double>(B);
  const double *__restrict__ r = S.res;
  const int i = t.i0 + threadIdx.x, j = t.j0 + threadIdx.y;
  if (i > S.nx || j > S.ny) return;
  const int k1 = min(t.k0 + RW_KCH - 1, S.nz);
#pragma unroll 4
  for (int k = t.k0; k <= k1; ++k) {
    const long long e = cell_off(B, i, j, k);
    fi[e] = fi[e] + r[sip_idx(S, i, j, k)];
  }
}

// Both substitutions of a block in one CTA: its hyperplanes one after
// another, a CTA barrier between them (a block's recurrences never reach
// into another block).  For small blocks, where a hyperplane holds a few
// thousand cells at most, this replaces 2*(nx+ny+nz-2) launches per sweep
// by one; the per-cell arithmetic is k_sip_forward's and k_sip_backward's.
__global__ void __launch_bounds__(1024) k_sip_subst_block(const SipBlk *__restrict__ sb,
                                                          const BlkLev *__restrict__ bl,
                                                          const SipCtl *__restrict__ ctl) {
  pdl_wait();
  if (!ctl->run) return;
  const SipBlk S = sb[blockIdx.x];
  const BlkLev &B = bl[blockIdx.x];
  double *fi = phi_of<double>(B);
  const int hmax = S.nx + S.ny + S.nz, pairs = S.nx * S.ny;
  for (int h = 3; h <= hmax; ++h) {
    for (int q = threadIdx.x; q < pairs; q += blockDim.x) {
      const int i = q % S.nx + 1, j = q / S.nx + 1, k = h - i - j;
      if (k < 1 || k > S.nz) continue;
      const long long c = sip_plain(S, i, j, k);
      S.res[c] = (S.res[c] - S.lb[c] * S.res[sip_plain(S, i, j, k - 1)] - S.lw[c] * S.res[sip_plain(S, i - 1, j, k)] -
                  S.ls[c] * S.res[sip_plain(S, i, j - 1, k)]) *
                 S.lpr[c];
    }
    __syncthreads();
  }
  for (int h = hmax; h >= 3; --h) {
    for (int q = threadIdx.x; q < pairs; q += blockDim.x) {
      const int i = q % S.nx + 1, j = q / S.nx + 1, k = h - i - j;
      if (k < 1 || k > S.nz) continue;
      const long long c = sip_plain(S, i, j, k);
      const double r = S.res[c] - S.un[c] * S.res[sip_plain(S, i, j + 1, k)] -
                       S.ue[c] * S.res[sip_plain(S, i + 1, j, k)] - S.ut[c] * S.res[sip_plain(S, i, j, k + 1)];
      S.res[c] = r;
      const long long e = cell_off(B, i, j, k);
      fi[e] = fi[e] + r;
    }
    __syncthreads();
  }
}

// The same two substitutions with one thread per (i, j) column, for blocks
// of at most 1024 columns.  At hyperplane h column (i, j) holds cell
// k = h-i-j: the cell below is its own previous value (a register), and
// the cells west and south (forward) or east and north (backward) at the
// same k were formed by those columns one hyperplane earlier and wait in a
// shared-memory plane.  Each hyperplane is then two CTA barriers and no
// dependent global load; the operands of the next cell are loaded one step
// ahead.  The arithmetic is the reference's, operand for operand.
__global__ void __launch_bounds__(1024) k_sip_subst_col(const SipBlk *__restrict__ sb,
                                                        const BlkLev *__restrict__ bl,
                                                        const SipCtl *__restrict__ ctl) {
  pdl_wait();
  if (!ctl->run) return;
  extern __shared__ double plane[];  // (ny+2) x (nx+2), zero border
  const SipBlk S = sb[blockIdx.x];
  const BlkLev &B = bl[blockIdx.x];
  double *fi = phi_of<double>(B);
  const int nx = S.nx, ny = S.ny, nz = S.nz, px = nx + 2;
  const int tid = threadIdx.x;
  for (int q = tid; q < (ny + 2) * px; q += blockDim.x) plane[q] = 0.0;
  const bool col = tid < nx * ny;
  const int i = tid % nx + 1, j = tid / nx + 1;
  const int hmax = nx + ny + nz;
  __syncthreads();
  // forward: res = (res - lb*res(k-1) - lw*res(i-1) - ls*res(j-1)) * lpr
  double below = 0.0;
  int kn = 3 - i - j;  // k at the next step
  double nres = 0.0, nlb = 0.0, nlw = 0.0, nls = 0.0, nlpr = 0.0;
  auto fetch_f = [&](int k) {
    if (col && k >= 1 && k <= nz) {
      const long long c = sip_plain(S, i, j, k);
      nres = S.res[c]; nlb = S.lb[c]; nlw = S.lw[c]; nls = S.ls[c]; nlpr = S.lpr[c];
    }
  };
  fetch_f(kn);
  for (int h = 3; h <= hmax; ++h) {
    const int k = h - i - j;
    const bool act = col && k >= 1 && k <= nz;
    double v = 0.0;
    if (act) {
      const double w = plane[j * px + i - 1], so = plane[(j - 1) * px + i];
      v = (nres - nlb * below - nlw * w - nls * so) * nlpr;
    }
    fetch_f(k + 1);
    __syncthreads();
    if (act) {
      plane[j * px + i] = v;
      S.res[sip_plain(S, i, j, k)] = v;
      below = v;
    }
    __syncthreads();
  }
  // backward: res = res - un*res(j+1) - ue*res(i+1) - ut*res(k+1); fi += res
  for (int q = tid; q < (ny + 2) * px; q += blockDim.x) plane[q] = 0.0;
  __syncthreads();
  double above = 0.0;
  double bres = 0.0, bun = 0.0, bue = 0.0, but = 0.0;
  auto fetch_b = [&](int k) {
    if (col && k >= 1 && k <= nz) {
      const long long c = sip_plain(S, i, j, k);
      bres = S.res[c]; bun = S.un[c]; bue = S.ue[c]; but = S.ut[c];
    }
  };
  fetch_b(hmax - i - j);
  for (int h = hmax; h >= 3; --h) {
    const int k = h - i - j;
    const bool act = col && k >= 1 && k <= nz;
    double r = 0.0;
    if (act) {
      const double no = plane[(j + 1) * px + i], ea = plane[j * px + i + 1];
      r = bres - bun * no - bue * ea - but * above;
    }
    fetch_b(k - 1);
    __syncthreads();
    if (act) {
      plane[j * px + i] = r;
      S.res[sip_plain(S, i, j, k)] = r;
      const long long e = cell_off(B, i, j, k);
      fi[e] = fi[e] + r;
      above = r;
    }
    __syncthreads();
  }
}

constexpr size_t kSipSmem = 220 * 1024;
constexpr int kSipSlabs = 8;  // CTAs per block of k_sip_subst at most (portable cluster size)
// CTAs per block of k_sip_subst with at most W warps each: as many as leave
// each about 4 warps while every cluster is resident at once (the operands
// stream over more SMs), at least what the warps need; 0 where 8 CTAs do not
// hold a block's warps.  warps: per CTA.
static int sip_slabs(const std::vector<SipBlk> &hb, int nsm, int W, int &warps) {
  long long need = 1, want = 1;
  for (const auto &b : hb) {
    const long long nseg = (b.nx + 31) / 32, fit = W / nseg;
    if (!fit) return 0;
    need = std::max(need, (b.ny + fit - 1) / fit);
    want = std::max(want, (b.ny * nseg + 3) / 4);
  }
  if (need > kSipSlabs) return 0;
  const int cl = (int)std::max(need, std::min<long long>(std::min<long long>(kSipSlabs, want), nsm / (long long)hb.size()));
  warps = 1;
  for (const auto &b : hb) warps = std::max(warps, (b.ny + cl - 1) / cl * ((b.nx + 31) / 32));
  return cl;
}

constexpr int kSipBlockCells = 4096;  // columns of a plane that one CTA walks at most

// Which way for a view.  k_sip_subst's time is its chain, the rows, row
// segments and chunks of steps one after the other, times the waves its
// clusters need; a CTA's is its hyperplanes, at a price that grows with the
// columns at work, times the waves of blocks; the launches' is theirs, growing
// with their CTAs.  k_sip_subst falls behind on narrow tall planes (one or two
// lanes of 32 at work, 17 and more warps a CTA) and on more clusters than the
// device holds.  The estimates are microseconds a sweep, fitted to all three on
// shapes that k_sip_subst takes (1..400 x 4..256 columns, 3..200 planes, 1..216
// blocks; 9 to 12 % rms).  Over 479 random ones of them the choice takes 0.6 %
// longer than the better way on average and 26 % at worst, always k_sip_subst
// up to 8.4 times longer, never up to 12 times.  4x130x8 in 200 blocks, 2 calls
// of 4 sweeps: 37 ms and 8.4; 32x32x32 in 64 blocks: 3.1 and 4.8 ms.
static double sip_rows_us(const std::vector<SipBlk> &hb, int warps, bool ring, int clusters) {
  double chain = 0.0, slots = 0.0;
  int chunks = 0;  // of a row segment: the warps at work at once at most
  for (const auto &b : hb) {
    const int nseg = (b.nx + 31) / 32, c = sip_steps(b.nz) / SIP_K;
    chain = std::max(chain, b.ny + 17.0 * (nseg - 1) + c);
    chunks = std::max(chunks, c);
    slots += 32.0 * b.ny * nseg * sip_steps(b.nz);
  }
  const int nb = (int)hb.size(), waves = (nb + clusters - 1) / clusters;
  const double price = warps > 16 ? 0.21 + 0.03 * std::min(warps, chunks) + 0.025 * warps : ring ? 0.73 : 0.38;
  return 43.0 + waves * 2.0 * chain * price + 1.2 * nb + 3.7e-5 * slots;
}
static double sip_cta_us(const std::vector<SipBlk> &hb, int nsm) {
  double planes = 0.0, price = 0.0, cells = 0.0;
  for (const auto &b : hb) {
    const double cols = (double)b.nx * b.ny, h = b.nx + b.ny + b.nz, at_work = cols * b.nz / h;
    planes = std::max(planes, h - 2.0);
    price = std::max(price, cols <= 1024 ? 0.58 + 1.9e-3 * at_work
                                         : 0.74 + 3.1e-3 * at_work + 1.5e-4 * cols + 8.2e-4 * b.nx);
    cells += cols * b.nz;
  }
  const int nb = (int)hb.size(), waves = (nb + nsm - 1) / nsm;
  return 27.0 + waves * 2.0 * planes * price * (1.0 + 0.48 * std::min(nb, nsm) / nsm) + 1.4 * nb + 7.8e-5 * cells;
}
static double sip_launch_us(const std::vector<SipBlk> &hb) {
  double planes = 0.0, cols = 0.0, at_work = 0.0;
  for (const auto &b : hb) {
    const double c = (double)b.nx * b.ny, h = b.nx + b.ny + b.nz;
    planes = std::max(planes, h - 2.0);
    cols += c;
    at_work += c * b.nz / h;
  }
  return 20.0 + 2.0 * planes * (1.9 + 1.8e-6 * cols + 9.4e-5 * at_work) + 1.5 * (double)hb.size();
}

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------
struct SipState {
  std::vector<DevBuf<double>> arrays;  // per block: 8 arrays
  DevBuf<SipBlk> sb;
  DevBuf<Tile> t_ij;                   // (i, j) pairs of every block
  int n_ij = 0, hmax = 0;
  DevBuf<double> part;
  DevBuf<SipCtl> ctl;
  int cl = 0, warps = 0;               // k_sip_subst: CTAs per block (0: another way), warps per CTA,
  size_t smem = 0;                     // its shared memory and variant
  void (*subst)(const SipBlk *, const SipCtl *, int, int *) = nullptr;
  void (*cta)(const SipBlk *, const BlkLev *, const SipCtl *) = nullptr;  // one CTA per block, or null
  size_t cta_smem = 0;
  cudaGraphExec_t sweep = nullptr;     // hyperplane launches: forward + backward substitutions,
  int *next = nullptr;                 // the stopping test's answer on the host (pinned),
  cudaEvent_t tested = nullptr;        // there once this is recorded
  ~SipState() {
    if (sweep) cudaGraphExecDestroy(sweep);
    if (tested) cudaEventDestroy(tested);
    if (next) cudaFreeHost(next);
  }
};

static int sip_prepare(mf3d_ctx *C, View &V) {
  if (C->sip) return MF3D_OK;
  cudaStream_t s = C->stream;
  auto S = std::make_unique<SipState>();
  const int nb = (int)V.blk.size();
  std::vector<SipBlk> hb(nb);
  std::vector<long long> items;
  int st;
  S->arrays.resize((size_t)8 * nb);
  for (int b = 0; b < nb; ++b) {
    const mf3d_block_desc &d = V.blk[b]->d;
    hb[b].nx = d.nx; hb[b].ny = d.ny; hb[b].nz = d.nz;
    items.push_back((long long)d.nx * d.ny);
    S->hmax = std::max(S->hmax, d.nx + d.ny + d.nz);
  }
  // one launch for the substitutions: k_sip_subst where the rows fit a cluster
  // and the arrays in its order (sip_steps of 32 columns a row segment) leave
  // half of the free memory, or a CTA per block, whichever is estimated the
  // fastest, these two or the launches
  auto elems = [](const SipBlk &b, int nseg) {
    return nseg ? (size_t)b.ny * nseg * sip_steps(b.nz) * 32 : (size_t)(b.nx + 2) * (b.ny + 2) * (b.nz + 2);
  };
  for (int W : {8, 16, 32}) {
    S->cl = sip_slabs(hb, C->nsm, W, S->warps);
    if (S->cl) break;
  }
  size_t need = 0, room = 0, all = 0;
  for (const auto &b : hb) need += 8 * sizeof(double) * elems(b, (b.nx + 31) / 32);
  if (S->cl && (cudaMemGetInfo(&room, &all) != cudaSuccess || need > room / 2)) S->cl = 0;
  int clusters = 0;  // resident at once
  bool ring = false;
  if (S->cl) {
    int T = 1;
    for (const auto &b : hb) T = std::max(T, sip_steps(b.nz));
    ring = S->warps > 16 || sip_smem(S->warps, T) > kSipSmem;
    S->subst = S->warps <= 8    ? (ring ? k_sip_subst<8, 8, true> : k_sip_subst<8, 8, false>)
               : S->warps <= 16 ? (ring ? k_sip_subst<16, 8, true> : k_sip_subst<16, 8, false>)
                                : k_sip_subst<32, 4, true>;
    S->smem = sip_smem(S->warps, ring ? sip_ring(S->warps <= 8 ? 8 : S->warps <= 16 ? 16 : 32) : T);
    CK(cudaFuncSetAttribute(S->subst, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSipSmem));
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)S->cl;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(nb * S->cl));
    cfg.blockDim = dim3(32 * S->warps);
    cfg.dynamicSmemBytes = S->smem;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&clusters, S->subst, &cfg) != cudaSuccess || clusters < 1) {
      cudaGetLastError();
      S->cl = 0;
    }
  }
  int cols = 1, px = 1;  // columns of the largest plane; its size with a border
  for (const auto &b : hb) {
    cols = std::max(cols, b.nx * b.ny);
    px = std::max(px, (b.nx + 2) * (b.ny + 2));
  }
  const double by_launch = sip_launch_us(hb), by_cta = cols <= kSipBlockCells ? sip_cta_us(hb, C->nsm) : 1e300;
  if (S->cl && sip_rows_us(hb, S->warps, ring, clusters) > 0.95 * (0.75 * by_cta <= by_launch ? by_cta : by_launch)) S->cl = 0;
  if (!S->cl && 0.75 * by_cta <= by_launch) {  // the launches only where they are clearly faster
    S->cta = cols <= 1024 ? k_sip_subst_col : k_sip_subst_block;
    S->cta_smem = cols <= 1024 ? (size_t)px * sizeof(double) : 0;
  }
  for (int b = 0; b < nb; ++b) {
    const int nseg = S->cl ? (hb[b].nx + 31) / 32 : 0;
    const size_t n = elems(hb[b], nseg);
    double *p[8];
    for (int a = 0; a < 8; ++a) {
      DevBuf<double> &A = S->arrays[(size_t)8 * b + a];
      if ((st = A.alloc(n))) return st;
      CK(cudaMemsetAsync(A.p, 0, n * sizeof(double), s));
      p[a] = A.p;
    }
    hb[b] = SipBlk{p[0], p[1], p[2], p[3], p[4], p[5], p[6], p[7], hb[b].nx, hb[b].ny, hb[b].nz, nseg};
  }
  if ((st = S->sb.upload(hb, s))) return st;
  auto t = make_tiles(items);
  S->n_ij = (int)t.size();
  if ((st = S->t_ij.upload(t, s))) return st;
  if ((st = S->part.alloc(std::max(V.n_int, 1)))) return st;
  if ((st = S->ctl.alloc(1))) return st;
  // the factors, hyperplane by hyperplane (the coefficients never change)
  const BlkLev *L1 = V.lv[1].tab.p;
  for (int h = 3; h <= S->hmax; ++h)
    launch(k_sip_factor, S->n_ij, kTile, 0, s, S->sb.p, L1, S->t_ij.p, h);
  if (!S->cl && !S->cta) {
    CK(cudaMallocHost(&S->next, sizeof(int)));
    CK(cudaEventCreateWithFlags(&S->tested, cudaEventDisableTiming));
    cudaGraph_t g = nullptr;
    CK(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    for (int h = 3; h <= S->hmax; ++h)
      launch(k_sip_forward, S->n_ij, kTile, 0, s, S->sb.p, S->t_ij.p, h, (const SipCtl *)S->ctl.p);
    for (int h = S->hmax; h >= 3; --h)
      launch(k_sip_backward, S->n_ij, kTile, 0, s, S->sb.p, L1, S->t_ij.p, h, (const SipCtl *)S->ctl.p);
    CK(cudaStreamEndCapture(s, &g));
    const cudaError_t e = cudaGraphInstantiate(&S->sweep, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) { set_error(std::string("SIP graph: ") + cudaGetErrorString(e)); return MF3D_E_CUDA; }
  }
  CK(cudaStreamSynchronize(s));
  C->launches += S->hmax - 2;
  C->sip = std::move(S);
  return MF3D_OK;
}

// sipsol(44): pp := 0, then up to nswp sweeps, the stopping test on the
// device (SipCtl).  The host queues them without waiting, but looks at the
// test every kSipAhead sweeps so that a long budget is not queued in vain.
// A sweep of hyperplane launches, hundreds of them, costs nearly as much when
// it has nothing to do: there the host reads each test's answer while the
// substitutions it precedes are running, and queues no sweep past the stop.
constexpr int kSipAhead = 8;
static int sip_solve(mf3d_ctx *C, View &V, bool first_call) {
  cudaStream_t s = C->stream;
  SipState &S = *C->sip;
  const ViewLevel &L1 = V.lv[1];
  for (size_t b = 0; b < V.blk.size(); ++b) {
    const BlkLev &B = V.blk[b]->lv[1].desc;
    CK(cudaMemsetAsync(B.phi, 0, (size_t)2 * B.cstr * sizeof(double), s));
  }
  SipCtl *ctl = S.ctl.p;
  launch(k_sip_begin, 1, 1, 0, s, ctl, first_call ? 1 : 0);
  ++C->launches;
  for (int sweep = 1; sweep <= C->prm.nswp; ++sweep) {
    launch(k_sip_residual, V.n_int, dim3(RW_TX, RW_RJ), 0, s, S.sb.p, L1.tab.p, V.t_int.p, S.part.p,
           (const SipCtl *)ctl);
    launch(k_sip_sum, 1, 1024, 0, s, (const double *)S.part.p, V.n_int, ctl, (const int *)V.err.p);
    if (S.cl) {
      launch_cl(S.subst, (int)V.blk.size() * S.cl, 32 * S.warps, S.smem, s, S.cl, S.sb.p, (const SipCtl *)ctl, S.cl,
                V.err.p);
      launch(k_sip_add, V.n_int, dim3(RW_TX, RW_RJ), 0, s, S.sb.p, L1.tab.p, V.t_int.p, (const SipCtl *)ctl);
    } else if (S.cta) {
      launch(S.cta, (int)V.blk.size(), 1024, S.cta_smem, s, S.sb.p, L1.tab.p, (const SipCtl *)ctl);
    } else {
      CK(cudaMemcpyAsync(S.next, &ctl->next, sizeof(int), cudaMemcpyDeviceToHost, s));
      CK(cudaEventRecord(S.tested, s));
      CK(cudaGraphLaunch(S.sweep, s));
    }
    halo<double>(C, V, 1, SUB_A, &ctl->run);
    C->launches += 2 + (S.cl ? 2 : S.cta ? 1 : 2 * (S.hmax - 2));
    if (S.sweep) {
      CK(cudaEventSynchronize(S.tested));
      if (!*S.next) break;
    } else if (sweep % kSipAhead == 0 && sweep < C->prm.nswp) {
      int next = 0;
      CK(cudaMemcpyAsync(&next, &ctl->next, sizeof next, cudaMemcpyDeviceToHost, s));
      CK(cudaStreamSynchronize(s));
      if (!next) break;
    }
  }
  return MF3D_OK;
}

// pressure_1sweep: the outer loop on the host, one domain.
static int solve_view_sip(mf3d_ctx *C, View &V, const double *dt, const double *alfapr, mf3d_solve_info *infos,
                          double *hist, int hcap) {
  cudaStream_t s = C->stream;
  C->launches = 0;
  CK(cudaEventRecord(C->ev0, s));
  int st = solve_begin<double>(C, V, dt, alfapr);
  if (st) return st;
  if ((st = sip_prepare(C, V))) return st;
  DomState D;
  CK(cudaMemcpyAsync(&D, V.ds.p, sizeof D, cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  const int maxcy = std::min(std::max(C->prm.maxcy, 0), V.hcap);
  double rmax = D.rmax0;
  int calls = 0, done = D.done == 2 ? 2 : 0;
  std::vector<double> hh;
  using Clock = std::chrono::steady_clock;
  Clock::time_point began = Clock::now();
  for (int iter = 1; iter <= maxcy && done == 0; ++iter) {
    if (iter > 1 && rmax < D.eps) { done = 1; break; }
    if ((st = sip_solve(C, V, calls == 0))) return st;
    ++calls;
    launch(k_add_correction<double>, V.n_pairs, kTile, 0, s, V.df.p, V.t_pairs.p, V.act.p, V.pairs_kch);
    p_exchange(C, V, V.act.p);
    CK(cudaMemsetAsync(V.rmax.p, 0, sizeof(unsigned long long), s));
    calvel_calmas<double>(C, V, V.act.p, V.rmax.p, 0);
    field_evolve(C, V, V.act.p);
    C->launches += 2;
    if (iter == maxcy) break;  // the reference runs no calmas after its last round
    unsigned long long bits = 0;
    CK(cudaMemcpyAsync(&bits, V.rmax.p, sizeof bits, cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    // a wait that gave up took kMaxWaitNs: only after such a round is its code
    // read, and collect() then reports it
    const Clock::time_point now = Clock::now();
    if (now - began > std::chrono::nanoseconds(kMaxWaitNs / 2)) {
      int e = 0;
      CK(cudaMemcpyAsync(&e, V.err.p, sizeof e, cudaMemcpyDeviceToHost, s));
      CK(cudaStreamSynchronize(s));
      if (e == ERR_SIP_WAIT) break;
    }
    began = now;
    std::memcpy(&rmax, &bits, sizeof rmax);
    hh.push_back(rmax);
    if (!(rmax <= 1.7976931348623157e308)) done = 2;
  }
  D.rmax = rmax;
  D.iter = calls;
  D.done = done == 0 ? 3 : done;
  C->sip_sweeps = 0;
  if (calls)
    CK(cudaMemcpyAsync(&C->sip_sweeps, &C->sip->ctl.p->total, sizeof(long long), cudaMemcpyDeviceToHost, s));
  CK(cudaMemcpyAsync(V.ds.p, &D, sizeof D, cudaMemcpyHostToDevice, s));
  if (!hh.empty()) CK(cudaMemcpyAsync(V.hist.p, hh.data(), std::min<size_t>(hh.size(), V.hcap) * sizeof(double),
                                      cudaMemcpyHostToDevice, s));
  CK(cudaStreamSynchronize(s));
  if ((st = solve_end<double>(C, V))) return st;
  CK(cudaEventRecord(C->ev1, s));
  CK(cudaStreamSynchronize(s));
  CK(cudaGetLastError());
  float ms = 0.f;
  cudaEventElapsedTime(&ms, C->ev0, C->ev1);
  // collect() reports D.iter entries of the history; ours holds one per
  // completed round that was followed by a calmas
  const int res = collect(C, V, infos, nullptr, 0, ms);
  if (hist && hcap > 0)
    for (int q = 0; q < (int)hh.size() && q < hcap; ++q) hist[q] = hh[q];
  return res;
}

}  // namespace mf3d
