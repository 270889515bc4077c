// PCG of one body inside one thread-block cluster of 16 blocks.
//
// A solve of a small or medium body is bound by latency: on the whole GPU an
// iteration costs two grid barriers, or one and a matvec whose inputs come
// through L2 (7-9 us an iteration whatever the body's size).  Here the body's
// rows are spread over the blocks of one cluster; each block keeps its rows'
// vectors in registers, the matvec input of its rows and of the foreign rows
// they read in shared memory, and its matrix in registers and shared memory,
// as far as that goes.  The two exchanges of an iteration (the input's foreign
// entries, the sums) are asynchronous stores into the other blocks' shared
// memory that count down a barrier there: one trip each, where a store and a
// cluster barrier cost three (16 blocks exchanging 16 bytes each: 0.2 against
// 0.55 us).  What bounds it: those two trips and the chains of FP64 operations
// and shuffles between them, up to 4 slices a block (2.0-2.4 us an iteration
// where kPcg1 took 6.6-8.4); above, the workers' reads of shared memory (4.9 us
// at 3,840 rows against 8.9, 7.0 at 4,624 against 9.0).
//
// The arrangement is that of Chronopoulos and Gear ("s-step iterative methods
// for symmetric linear systems", 1989), as in kPcg1: u = P r, w = A u, and
// with gamma = r.u, delta = w.u: beta = gamma / gamma_prev, p.A p = delta -
// beta gamma / alpha_prev, alpha = gamma / p.A p, p = u + beta p, s = w + beta
// s, x += alpha p, r -= alpha s; x, r, p and s are FP64 in both precisions and
// u is rounded to S, on both sides, as it is published.
#pragma once

#include "tl_cluster_build.h"
#include "tl_sell.cuh"

namespace tl {

constexpr uint32_t CLUSTER_T = 512;     // threads of a block
constexpr uint32_t CLUSTER_W = CLUSTER_T / 32;
constexpr uint32_t CLUSTER_MAX = 16;    // blocks of a cluster (above 8 needs the non-portable size)
constexpr uint32_t CLUSTER_OWNERS = 8;  // most warps of a block that own rows
constexpr uint32_t CLUSTER_REG = 4;     // column slots a worker keeps in registers
constexpr uint32_t CLUSTER_PARTS = 4;   // most workers that share a slice (15 slots on a Kuhn lattice)

struct ClusterDev {
  uint32_t slices;            // most slices of one block
  uint32_t owners;            // warps of a block that own rows; the others work on the matvec
  uint32_t parts;             // workers that share a slice's column slots
  uint32_t entries;           // vector entries reserved per block
  uint32_t positions;         // column slots reserved per block
  uint32_t cached;            // column slots of a worker's slice kept in shared memory, beyond its registers'
  uint32_t far;               // whether some slots are left in L2
  const uint32_t* foreign;    // [blocks] foreign entries of each block's vector
  const uint16_t* local;      // [block positions]
  const uint4* push;          // [rows]
  const uint32_t* over_start; // [rows + 1]
  const uint32_t* over;
};

// Shared-memory layout of a block, in bytes.  The matrix and the vector are
// FP64 in both precisions: a conversion to FP64 costs as much as four FP64
// fused multiply-adds (15 against 62 lanes a clock per SM measured), so a
// block's entries are converted once per solve and a published value once per
// iteration, not at each of its 15 uses.
struct ClusterLayout {
  size_t bars, scalars, sums, red, share, vec, local, val, total;
};
__host__ __device__ inline ClusterLayout clusterLayout(const ClusterDev& c, uint32_t cached) {
  ClusterLayout l;
  size_t at = 0;
  const auto take = [&](size_t bytes) {
    const size_t here = at;
    at += (bytes + 15) / 16 * 16;
    return here;
  };
  l.bars = take(3 * sizeof(uint64_t));
  l.scalars = take(4 * sizeof(double));
  l.sums = take(2 * 3 * CLUSTER_MAX * sizeof(double));
  l.red = take(3 * CLUSTER_OWNERS * sizeof(double));
  l.share = take(size_t(c.parts) * c.slices * 32 * 3 * sizeof(double));
  l.vec = take(size_t(c.entries) * 24);
  l.local = take(size_t(c.positions) * sizeof(uint16_t));
  l.val = take(size_t(c.slices) * c.parts * cached * 9 * SELL_ROWS * sizeof(double));
  l.total = at;
  return l;
}

__device__ __forceinline__ void clusterBarrier() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t clusterRank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t clusterSize() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t smemAddress(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }
// The shared::cluster address of the same place in block `rank`.
__device__ __forceinline__ uint32_t inBlock(uint32_t address, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(address), "r"(rank));
  return r;
}
// Asynchronous stores into a block of the cluster; each counts its bytes at
// that block's barrier `bar`.
__device__ __forceinline__ void sendTo(uint32_t a, uint32_t bar, double x, double y) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(a),
               "l"(__double_as_longlong(x)), "l"(__double_as_longlong(y)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void sendTo(uint32_t a, uint32_t bar, double x) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(a),
               "l"(__double_as_longlong(x)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void barInit(uint32_t bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
// The block's one arrival of a phase, with the bytes the phase waits for.
__device__ __forceinline__ void barExpect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Waits for the phase of the given parity; bounded like the grid barriers.
__device__ __forceinline__ bool barWait(uint32_t bar, uint32_t parity, GridSyncDev* sync) {
  unsigned long long t0 = 0;
  for (uint32_t tries = 0;; ++tries) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
    if ((tries & 63u) == 63u) {
      if (t0 == 0) t0 = globalTimer();
      else if (globalTimer() - t0 > TL_BARRIER_LIMIT_NS) {
        atomicExch(&sync->error, 5);  // TL_ERR_TIMEOUT
        return false;
      }
    }
  }
}

// Sum over the warp, in every lane.
__device__ __forceinline__ double warpSum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// acc += block x.
__device__ __forceinline__ void clusterFma(const double (&b)[9], V3<double> x, V3<double>& acc) {
  acc.x = fma(b[0], x.x, fma(b[1], x.y, fma(b[2], x.z, acc.x)));
  acc.y = fma(b[3], x.x, fma(b[4], x.y, fma(b[5], x.z, acc.y)));
  acc.z = fma(b[6], x.x, fma(b[7], x.y, fma(b[8], x.z, acc.z)));
}

// The first c.owners warps of a block own its rows, K slices each, and do
// all of the solve but the matvec, which the other warps, the workers, do: a
// worker's registers hold its matrix entries, an owner's the iteration's
// vectors.  Three block barriers an iteration hand over: the published vector,
// the products, the scalars.
template <class S, int K>
__global__ void __launch_bounds__(CLUSTER_T, 1)
    kPcgCluster(Sys<S> s, SellDev<S> g, ClusterDev c, Vec4<S>* X, uint32_t x0zero, uint32_t tangent) {
  constexpr uint32_t NONE = CLUSTER_NO_PUSH;
  constexpr int R = int(CLUSTER_REG);
  extern __shared__ __align__(16) unsigned char tlCluster[];
  // a wait of an earlier solve ran out: this solve leaves too (nothing changes the word before it runs)
  if (*(volatile int*)&s.sync->error != 0) return;
  const ClusterLayout lay = clusterLayout(c, c.cached);
  double* const scalars = reinterpret_cast<double*>(tlCluster + lay.scalars);
  double* const share = reinterpret_cast<double*>(tlCluster + lay.share);
  double2* const vecXY = reinterpret_cast<double2*>(tlCluster + lay.vec);  // (x, y) of each entry, then z
  double* const vecZ = reinterpret_cast<double*>(vecXY + c.entries);
  uint16_t* const local = reinterpret_cast<uint16_t*>(tlCluster + lay.local);
  double* const val = reinterpret_cast<double*>(tlCluster + lay.val);
  const uint32_t haloBar = smemAddress(tlCluster + lay.bars), sumsBar = haloBar + 8, vecAt = smemAddress(vecXY);
  const uint32_t rank = clusterRank(), C = clusterSize();
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const bool owner = warp < c.owners;
  const uint32_t stride = c.slices * 32u;  // of the products' components
  uint32_t haloUse = 0, sumsUse = 0;       // phases of the barriers used so far
  if (tid == 0) {
    for (uint32_t k = 0; k < 3; ++k) barInit(haloBar + 8 * k);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  clusterBarrier();  // every block of the cluster runs, its barriers ready, before its shared memory is written
  const uint32_t sA = clusterSlice(g.slices, C, rank), sB = clusterSlice(g.slices, C, rank + 1);
  const uint32_t mine = sB - sA;
  bool good = true;
  if (!owner) {
    // ------------------------------------------------------------ workers
    const uint32_t pA = __ldg(&g.slice_start[sA]), pB = __ldg(&g.slice_start[sB]);
    const uint32_t worker = warp - c.owners, workers = CLUSTER_W - c.owners;
    const uint32_t part = worker / c.slices < c.parts ? worker / c.slices : 0u;
    const uint32_t step = c.parts > 1u ? c.slices : workers;  // a worker's slices (one, where slices are shared)
    const uint32_t slice0 = worker / c.slices < c.parts ? worker - part * c.slices : c.slices;
    for (uint32_t i = tid - 32u * c.owners; i < (pB - pA) / 8u; i += 32u * workers)
      cpAsync<16>(local + 8 * i, c.local + pA + 8 * i);
    cpAsyncCommit();
    // the column slots of slice ls that are this worker's: block position of the first, and their number
    const auto slotsOf = [&](uint32_t ls, uint32_t& count) {
      const uint32_t p0 = __ldg(&g.slice_start[sA + ls]), width = (__ldg(&g.slice_start[sA + ls + 1]) - p0) >> 5;
      const uint32_t k0 = width * part / c.parts;
      count = width * (part + 1u) / c.parts - k0;
      return p0 + 32u * k0 + lane;
    };
    double reg[R][9];  // the first slots of the first slice
    uint32_t regAt[R], first0 = 0, count0 = 0;
#pragma unroll
    for (int k = 0; k < R; ++k) {
      regAt[k] = 0u;
#pragma unroll
      for (int m = 0; m < 9; ++m) reg[k][m] = 0.0;
    }
    for (uint32_t ls = slice0; ls < mine; ls += step) {
      uint32_t count;
      const uint32_t first = slotsOf(ls, count);
      const uint32_t inReg = ls == slice0 ? uint32_t(R) : 0u;
      const S* const from = g.val + size_t(first >> 5) * 9 * SELL_ROWS + lane;
      double* const to = val + size_t(ls * c.parts + part) * c.cached * 9 * SELL_ROWS + lane;
      for (uint32_t k = inReg; k < min(count, inReg + c.cached); ++k)
#pragma unroll
        for (int m = 0; m < 9; ++m)
          to[(size_t(k - inReg) * 9 + m) * SELL_ROWS] = double(from[(size_t(k) * 9 + m) * SELL_ROWS]);
      if (inReg) {
        first0 = first;
        count0 = count;
#pragma unroll
        for (int k = 0; k < R; ++k)
          if (uint32_t(k) < count) {
#pragma unroll
            for (int m = 0; m < 9; ++m) reg[k][m] = double(from[(size_t(k) * 9 + m) * SELL_ROWS]);
            regAt[k] = __ldg(&c.local[first + 32u * k]);
          }
      }
    }
    cpAsyncWaitAll();
    const auto entryOf = [&](uint32_t i) -> V3<double> {
      const double2 a = vecXY[i];
      return {a.x, a.y, vecZ[i]};
    };
    static_assert(R == 4, "the sum of the register slots is written out");
    const bool allInReg = c.parts > 1u && c.cached == 0u && !c.far;
    // the worker's products of the published vector; their owners sum the parts
    const auto multiply = [&]() {
      if (allInReg) {
        if (slice0 >= mine) return;
        V3<double> e[R], sum[R];
#pragma unroll
        for (int q = 0; q < R; ++q) e[q] = entryOf(regAt[q]);
#pragma unroll
        for (int q = 0; q < R; ++q) {
          sum[q] = {0, 0, 0};
          clusterFma(reg[q], e[q], sum[q]);
        }
        const V3<double> all = (sum[0] + sum[1]) + (sum[2] + sum[3]);
        double* const t = share + part * 3u * stride + slice0 * 32u + lane;
        t[0] = all.x;
        t[stride] = all.y;
        t[2 * stride] = all.z;
        return;
      }
      for (uint32_t ls = slice0; ls < mine; ls += step) {
        V3<double> even = {0, 0, 0}, odd = {0, 0, 0};
        uint32_t first = first0, count = count0, k = 0;
        if (ls == slice0) {
          V3<double> e[R];
#pragma unroll
          for (int q = 0; q < R; ++q) e[q] = entryOf(regAt[q]);
#pragma unroll
          for (int q = 0; q < R; ++q) clusterFma(reg[q], e[q], q & 1 ? odd : even);
          k = min(count, uint32_t(R));
        } else {
          first = slotsOf(ls, count);
        }
        const uint16_t* const at = local + (first - pA);
        const double* near = val + size_t(ls * c.parts + part) * c.cached * 9 * SELL_ROWS + lane;
        for (const uint32_t end = min(count, k + c.cached); k < end; ++k, near += 9 * SELL_ROWS) {
          double blk[9];
#pragma unroll
          for (int m = 0; m < 9; ++m) blk[m] = near[m * SELL_ROWS];
          clusterFma(blk, entryOf(at[k * 32]), k & 1u ? odd : even);
        }
        const S* far = g.val + (size_t(first >> 5) + k) * 9 * SELL_ROWS + lane;
        for (; k < count; ++k, far += 9 * SELL_ROWS) {  // what is left in L2
          double blk[9];
#pragma unroll
          for (int m = 0; m < 9; ++m) blk[m] = double(__ldg(far + m * SELL_ROWS));
          clusterFma(blk, entryOf(at[k * 32]), k & 1u ? odd : even);
        }
        double* const t = share + part * 3u * stride + ls * 32u + lane;
        t[0] = even.x + odd.x;
        t[stride] = even.y + odd.y;
        t[2 * stride] = even.z + odd.z;
      }
    };
    const uint32_t rounds = x0zero ? 0u : 1u;  // A x first, where the solve starts from x
    for (uint32_t round = 0;; ++round) {
      if (round >= rounds) {
        __syncthreads();  // the scalars
        const double state = scalars[2];
        if (state != 0.0) {
          good = state < 2.0;
          break;
        }
      }
      __syncthreads();  // the published vector: the block's own rows
      const bool in = barWait(haloBar, haloUse & 1u, s.sync);  // and the foreign ones
      ++haloUse;
      if (!in) scalars[3] = 1.0;
      multiply();
      __syncthreads();  // the products
    }
  } else {
    // ------------------------------------------------------------- owners
    const BodyStepDev st = s.step[0];
    const uint32_t haloBytes = 24u * __ldg(&c.foreign[rank]);
    bool own[K], freeRow[K];
    uint32_t row[K], to[K][CLUSTER_INLINE], over0[K], over1[K];
    Sym<S> P[K];
    V3<double> x[K], r[K], p[K], sv[K], u[K], w[K];
    double rhsSquared = 0.0;
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const uint32_t ls = uint32_t(j) * c.owners + warp;
      own[j] = ls < mine;
      row[j] = (sA + ls) * SELL_ROWS + lane;
      const bool live = own[j] && row[j] < g.rows;
      freeRow[j] = live && !s.anch[row[j]];
      P[j] = {1, 1, 1, 0, 0, 0};
      x[j] = r[j] = p[j] = sv[j] = {0, 0, 0};
      over0[j] = over1[j] = 0;
#pragma unroll
      for (int d = 0; d < int(CLUSTER_INLINE); ++d) to[j][d] = NONE;
      if (live) {
        const Vec4<S> q0 = s.pre0[row[j]], q1 = s.pre1[row[j]];
        P[j] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y};
        const V3<double> rhs = cvt<double>(xyz(s.right[row[j]]));
        rhsSquared += dot(rhs, rhs);
        if (freeRow[j]) r[j] = rhs;
        if (!x0zero) x[j] = cvt<double>(xyz(X[row[j]]));
        const uint4 code = __ldg(&c.push[row[j]]);
        to[j][0] = code.x;
        to[j][1] = code.y;
        to[j][2] = code.z;
        to[j][3] = code.w;
        over0[j] = __ldg(&c.over_start[row[j]]);
        over1[j] = __ldg(&c.over_start[row[j] + 1]);
      }
    }
    // value of row j for the matvec: to the blocks that read it, and the block's own entry
    const auto send = [&](uint32_t code, V3<double> a) {
      // the places of one block lie as far apart in the cluster's window as in the block's
      const uint32_t entry = code & 0xffffu, bar = inBlock(haloBar, code >> 16);
      const uint32_t at = bar + (vecAt - haloBar) + 16u * entry;
      sendTo(at, bar, a.x, a.y);
      sendTo(at + 16u * c.entries - 8u * entry, bar, a.z);
    };
    const auto publish = [&](const V3<double> (&a)[K]) {
      if (tid == 0) barExpect(haloBar, haloBytes);
#pragma unroll
      for (int j = 0; j < K; ++j) {
        if (!own[j]) continue;
#pragma unroll
        for (int d = 0; d < int(CLUSTER_INLINE); ++d)
          if (to[j][d] != NONE) send(to[j][d], a[j]);
        for (uint32_t o = over0[j]; o < over1[j]; ++o) send(__ldg(&c.over[o]), a[j]);
        const uint32_t i = (uint32_t(j) * c.owners + warp) * SELL_ROWS + lane;
        vecXY[i] = make_double2(a[j].x, a[j].y);
        vecZ[i] = a[j].z;
      }
      __syncthreads();  // the published vector
    };
    const auto products = [&]() {
      __syncthreads();
#pragma unroll
      for (int j = 0; j < K; ++j) {
        w[j] = {0, 0, 0};
        if (!own[j]) continue;
        const double* t = share + (uint32_t(j) * c.owners + warp) * SELL_ROWS + lane;
        for (uint32_t q = 0; q < c.parts; ++q, t += 3u * stride)
          w[j] = w[j] + V3<double>{t[0], t[stride], t[2 * stride]};
      }
    };
    double gamma = 0.0, inverse = 0.0, ratio = 0.0;  // of the last update: gamma, 1 / gamma, p.A p / gamma (warp 0)
    // The block's sums leave in two packets a block pair, (a, b) and then d, from warp 0: the stores cost by
    // their number.
    double* const red = reinterpret_cast<double*>(tlCluster + lay.red);
    bool timely = true;  // no wait of warp 0 ran out
    const auto ownersMeet = [&]() {  // lane 0's entries of red are then visible to every owner's lanes
      if (c.owners > 1u) asm volatile("bar.sync 1, %0;" ::"r"(32u * c.owners) : "memory");
      else __syncwarp();
    };
    const auto sendPair = [&](double a, double bb) {
      if (lane == 0) {
        red[warp] = a;
        red[CLUSTER_OWNERS + warp] = bb;
      }
      ownersMeet();
      if (warp != 0) return;
      a = bb = 0.0;
      for (uint32_t o = 0; o < c.owners; ++o) {
        a += red[o];
        bb += red[CLUSTER_OWNERS + o];
      }
      const uint32_t half = sumsUse & 1u, bar = sumsBar + 8u * half;
      if (lane == 0) barExpect(bar, 24u * C);
      if (lane < C) {
        const uint32_t rb = inBlock(bar, lane);
        sendTo(rb + uint32_t(lay.sums - lay.bars) + half * (24u * CLUSTER_MAX) - 8u * (1u + half) + 16u * rank, rb, a, bb);
      }
    };
    // warp 0 returns with the cluster's sums, false if the wait ran out
    const auto total = [&](double& a, double& bb, double d) -> double {
      if (lane == 0) red[2 * CLUSTER_OWNERS + warp] = d;
      ownersMeet();
      const uint32_t half = sumsUse & 1u, bar = sumsBar + 8u * half, parity = (sumsUse >> 1) & 1u;
      ++sumsUse;
      if (warp != 0) return 0.0;
      d = 0.0;
      for (uint32_t o = 0; o < c.owners; ++o) d += red[2 * CLUSTER_OWNERS + o];
      if (lane < C) {
        const uint32_t rb = inBlock(bar, lane);
        sendTo(rb + uint32_t(lay.sums - lay.bars) + half * (24u * CLUSTER_MAX) - 8u * (1u + half) + 16u * CLUSTER_MAX + 8u * rank,
               rb, d);
      }
      const bool in = barWait(bar, parity, s.sync);
      const double* const rec = reinterpret_cast<const double*>(tlCluster + lay.sums) + half * (3u * CLUSTER_MAX);
      const uint32_t q = lane & 15u;
      double v = 0.0;
      d = 0.0;
      if (q < C) {
        v = rec[2 * q + (lane >> 4)];  // a in the lower lanes, b in the upper ones
        d = rec[2 * CLUSTER_MAX + q];
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        const double v2 = __shfl_xor_sync(0xffffffffu, v, o), d2 = __shfl_xor_sync(0xffffffffu, d, o);
        v += v2;
        d += d2;
      }
      a = __shfl_sync(0xffffffffu, v, 0);
      bb = __shfl_sync(0xffffffffu, v, 16);
      timely = in;
      return d;
    };
    const auto precondition = [&](int j, V3<double> a) {
      const Sym<double> q = {double(P[j].xx), double(P[j].yy), double(P[j].zz),
                             double(P[j].xy), double(P[j].xz), double(P[j].yz)};
      return roundTo<S>(symMul(q, a));
    };
    if (tid == 0) scalars[3] = 0.0;
    if (!x0zero) {  // r = right - A x
      publish(x);
      products();
#pragma unroll
      for (int j = 0; j < K; ++j)
        if (freeRow[j]) r[j] = r[j] - w[j];
    }
    // |right|; every block has read x once its sums are here
    double length = 0.0, floor = 0.0, target = 0.0, startRes = 0.0;
    {
      double sq = warpSum(rhsSquared), none = 0.0;
      sendPair(sq, none);
      total(sq, none, 0.0);
      if (warp == 0) {
        floor = fmax(sqrt(sq), 1.1754943508222875e-38);  // std::numeric_limits<float>::min()
        target = st.tolerance * floor;
        if (lane == 0) scalars[2] = timely && scalars[3] == 0.0 ? 0.0 : 2.0;
      }
    }
#pragma unroll
    for (int j = 0; j < K; ++j) u[j] = precondition(j, r[j]);
    uint32_t taken = 0;
    for (bool started = false;; started = true) {
      __syncthreads();  // the scalars
      const double alpha = scalars[0], beta = scalars[1], state = scalars[2];
      if (state != 0.0) {
        good = state < 2.0;
        break;
      }
      if (started) {
#pragma unroll
        for (int j = 0; j < K; ++j) {
          p[j] = u[j] + beta * p[j];
          sv[j] = w[j] + beta * sv[j];
          x[j] = x[j] + alpha * p[j];
          r[j] = r[j] - alpha * sv[j];
          u[j] = precondition(j, r[j]);
        }
        ++taken;
      }
      publish(u);
      // while the workers multiply
      double ru = 0.0, rr = 0.0, wu = 0.0;
#pragma unroll
      for (int j = 0; j < K; ++j) {
        ru += dot(r[j], u[j]);
        rr += dot(r[j], r[j]);
      }
      ru = warpSum(ru);
      rr = warpSum(rr);
      sendPair(ru, rr);
      if (warp == 0 && taken) {
        inverse = 1.0 / gamma;
        ratio *= inverse;
      }
      products();
#pragma unroll
      for (int j = 0; j < K; ++j) wu += dot(w[j], u[j]);
      wu = warpSum(wu);
      wu = total(ru, rr, wu);
      if (warp == 0) {
        length = rr;
        if (taken == 0u) startRes = sqrt(length) / floor;
        // the reference's loop-top test and breakdown test
        double a = 0.0, bl = 0.0, next2 = 1.0;
        if (!timely || scalars[3] != 0.0) {
          next2 = 2.0;
        } else if (taken < st.limit && !(length <= target * target)) {
          bl = taken ? ru * inverse : 0.0;
          const double pAp = taken ? wu - bl * ru * ratio : wu;
          if (pAp > 0.0 && ru > 0.0) {
            a = ru / pAp;
            ratio = pAp;
            gamma = ru;
            next2 = 0.0;
          }
        }
        if (lane == 0) {
          scalars[0] = a;
          scalars[1] = bl;
          scalars[2] = next2;
        }
      }
    }
    if (good) {
#pragma unroll
      for (int j = 0; j < K; ++j)
        if (own[j] && row[j] < g.rows) X[row[j]] = pack(cvt<S>(x[j]));
      if (rank == 0 && tid == 0) {
        const double residual = sqrt(length);
        CgBodyDev o;
        o.squared = gamma;
        o.target = target;
        o.floor = floor;
        o.length = length;
        o.stride = scalars[0];
        o.blend = scalars[1];
        o.start_res = startRes;
        o.rel_res = residual / floor;
        o.taken = taken;
        o.done = 1u;
        o.pad0 = o.pad1 = 0;
        s.cg[0] = o;
        CgReportDev rep = s.cgrep[0];
        rep.iterations += taken;
        rep.capped += (taken == st.limit && residual > target) ? 1u : 0u;
        rep.applications += taken + (x0zero ? 1u : 2u);  // A x, and A u of the start and of each update
        rep.solves += 1u;
        rep.tangent_iterations += tangent ? taken : 0u;
        rep.worst_rel = fmax(rep.worst_rel, o.rel_res);
        if (rep.pass_solves == 0u) rep.pass_start = o.start_res;
        rep.pass_end = o.rel_res;
        rep.pass_iterations += taken;
        rep.pass_solves += 1u;
        s.cgrep[0] = rep;
      }
    }
  }
  clusterBarrier();  // no block leaves while another may still write to it
}

}  // namespace tl
