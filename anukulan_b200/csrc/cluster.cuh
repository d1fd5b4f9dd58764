// cluster_chunk_kernel: up to a check period of iterations of one small LP, or
// of a few cases of a stack over a small matrix, in one launch.
//
// A small matrix does not fill the device, and two product launches per
// iteration cost two launch latencies and two rounds of loading the same
// schedule, matrix and step vectors, however little work they hold. Here each
// case runs on one thread-block cluster whose CTAs stay resident for the
// launch's iterations. Cases never exchange anything, so clusters are
// independent of each other. Each CTA owns a contiguous range of the rows of
// K~' (the primal side) and of K~ (the dual side) and holds those slices in
// shared memory. A thread owns one of the columns and one of the rows and
// keeps their step vectors in registers. Every CTA holds full copies of the
// gathered vectors, x_bar and y, in shared memory. An iteration is two phases:
//
//   primal: (K~'y)_j for its columns from its copy of y, then the primal step;
//           the new x_bar_j goes to every CTA's copy of x_bar;
//   dual:   (K~ x_bar)_i for its rows from its copy of x_bar, then the dual
//           step; the new y_i goes to every CTA's copy of y.
//
// A phase ends with the exchange: each CTA's entries, contiguous in the copies
// (a copy is laid out by owner: entry `place` = owner * stride + thread), go
// to each peer as one bulk copy through distributed shared memory that signals
// the peer's mbarrier as its bytes land, and the next phase starts when all
// the peers' entries have landed. No barrier is needed beside that: a CTA
// sends its part of a vector only after its sums against the previous one, and
// nobody can compute the next version without it, so no copy is overwritten
// while it is read.
//
// What bounds a phase is that chain of latencies. Measured between 16 CTAs:
// 0.4 us for an exchange of 240 entries per CTA, against 1.2 us through global
// memory (the store's release, the cluster barrier and the reload) and 1.1 us
// for storing every entry into every peer. Rows are dealt to threads by
// length, so a warp's rows end together, and the CTA has no more threads than
// its rows need, because idle warps still issue the phase's instructions.
//
// Waits are bounded: a wait longer than kClusterPatience sets the launch's
// status, which the host reads; its CTA then goes straight to the
// cluster barrier at the end, as its peers do when their own waits run out.
//
// Per iteration, against two launches per iteration: a 1,000 x 1,500 LP 2.35 us
// (3.7) in FP32 and 3.8 (4.0) in FP64; a refinery plan of 24 periods 3.3 (4.35)
// in FP32; 12 cases of it as a stack 3.9 (8.2) in FP32, 7 in FP64 5.4 (13.0).
//
// The sums are the ones the two-launch path takes, in its order, so iterates
// are the same bit for bit:
//  - a single LP (rows_kernel): a row of at most kSerialRow nonzeros left to
//    right from zero, products and sums rounded separately; a longer row (up
//    to kLongRow) by one warp, lane-strided partial sums, then the shuffle
//    tree;
//  - a stack (seg_kernel): rows cut into the segments of the case-stack
//    schedule, each summed in order from zero, segment sums added in order.
#pragma once

#include <cooperative_groups.h>

#include "kernels.cuh"

namespace anu {

// The longest launch: its Halpern weights sit in shared memory.
constexpr int kClusterMaxLen = 1024;
// The most threads, hence rows of either matrix, per CTA.
constexpr int kClusterThreadsMax = 1024;
// Clock cycles (about a second) before a wait gives up.
constexpr long long kClusterPatience = 1ll << 31;

// A row that is summed apart from its owner thread, into partial sum `slot`.
// Single LP: `count` nonzeros from entry `first` of the slice, by a warp.
// Stack: one segment, by a thread, its nonzeros kClusterStride entries apart.
struct ClusterPart {
  int32_t first, count, slot;
};
// A thread's row (an index into the matrix) and how it gets its sum: from its
// own `count` nonzeros, kClusterStride entries apart from `first`, or, when
// apart is set, from `count` partial sums at slot `first`. The lanes of a warp
// read neighbouring entries: no bank conflicts.
struct ClusterRow {
  int32_t row, first, count, apart;
};
constexpr int kClusterStride = 32;

// One matrix's share of the cluster, by CTA.
struct ClusterRows {
  const int32_t* __restrict__ bounds;      // CTAs + 1 row bounds
  const int32_t* __restrict__ part_start;  // CTAs + 1 offsets into part
  const ClusterRow* __restrict__ row;      // by CTA, then by thread
  const ClusterPart* __restrict__ part;
  // Per nonzero: its column's place in the copy it is gathered from, and its
  // entry in the CTA's slice.
  const int32_t* __restrict__ place;
  const int32_t* __restrict__ entry;
  int32_t max_rows, max_entries, max_parts;  // the most one CTA holds
  int32_t stride;  // this matrix's rows per owner in the copy its results go to
};

// A nonzero of a slice: its column's place and value, one shared-memory load.
template <class T>
struct alignas(2 * sizeof(T)) ClusterNz {
  int32_t place;
  T val;
};

// Byte offsets of a CTA's dynamic shared memory, each section 16-byte
// aligned: the copies of x_bar and y, the two slices, their sums taken apart
// (what and the results), the launch's Halpern weights and their complements,
// and the two mbarriers.
struct ClusterLayout {
  size_t xs, ys, nzt, nzk, partt, partk, part, wt, bars, total;
  template <class T>
  __host__ __device__ static ClusterLayout of(int32_t ctas, const ClusterRows& ktr,
                                              const ClusterRows& kr, int32_t len) {
    auto up = [](size_t b) { return (b + 15) & ~size_t(15); };
    auto most = [](int32_t a, int32_t b) { return a > b ? a : b; };
    ClusterLayout l{};
    l.xs = 0;
    l.ys = up(sizeof(T) * ctas * ktr.stride);
    l.nzt = up(l.ys + sizeof(T) * ctas * kr.stride);
    l.nzk = up(l.nzt + sizeof(ClusterNz<T>) * ktr.max_entries);
    l.partt = up(l.nzk + sizeof(ClusterNz<T>) * kr.max_entries);
    l.partk = up(l.partt + sizeof(ClusterPart) * ktr.max_parts);
    l.part = up(l.partk + sizeof(ClusterPart) * kr.max_parts);
    l.wt = up(l.part + sizeof(T) * most(ktr.max_parts, kr.max_parts));
    l.bars = up(l.wt + sizeof(T) * 2 * len);
    l.total = l.bars + 16;
    return l;
  }
};

// The step vectors (case-interleaved, K cases).
template <class T>
struct ClusterStep {
  int32_t K;
  int32_t it0;  // the launch's first iteration, within the chunk
  int32_t num_eq;
  const StepParams* __restrict__ p;
  const double* __restrict__ w_table;
  T* x;
  const T* __restrict__ c;
  const T* __restrict__ lo;
  const T* __restrict__ hi;
  T* anchor;
  T* dx;
  T* sum_x;
  T* y;
  const T* __restrict__ q;
  T* kx;
  T* anchor_y;
  T* anchor_kx;
  T* dy;
  T* sum_y;
  const T* __restrict__ ylo;  // may be null (zero)
  int32_t* status;  // set to kSyncTimedOut by a wait that gave up
};

// The cluster barrier in its two halves. Non-.aligned forms: correct whether
// or not the warp has reconverged.
__device__ __forceinline__ void cluster_arrive() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release;\n" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire;\n" ::: "memory");
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
// The address in CTA `rank` of this CTA's shared address a.
__device__ __forceinline__ uint32_t peer_addr(uint32_t a, int rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ bool bar_ready(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n.reg .pred p;\n"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// One exchanged vector: this CTA's copy of it, its own part (`bytes` at
// `mine`) and the mbarrier its peers' parts signal. The mbarrier's one arrival
// is the CTA's own, made with the byte count to expect; bytes that land before
// it are counted against it.
struct Exchange {
  uint32_t bar, mine, bytes;
  int rank, ctas;
  // Every thread, once its entry is in the copy. Returns whether any thread of
  // the CTA reports a wait that gave up (`bad`).
  __device__ __forceinline__ bool send(bool bad) const {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    bad = __syncthreads_or(bad) != 0;
    if (bad) return true;
    // One peer per warp at a time: a warp issues its copies one by one.
    if (threadIdx.x % 32 == 0)
      for (int q = static_cast<int>(threadIdx.x) / 32; q < ctas;
           q += static_cast<int>(blockDim.x) / 32)
        if (q != rank)
          asm volatile(
              "cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes "
              "[%0], [%1], %2, [%3];" ::"r"(peer_addr(mine, q)),
              "r"(mine), "r"(bytes), "r"(peer_addr(bar, q))
              : "memory");
    return false;
  }
  // False when the wait gave up.
  __device__ __forceinline__ bool receive(uint32_t parity) const {
    if (threadIdx.x == 0)
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                   "r"(bytes * static_cast<uint32_t>(ctas - 1))
                   : "memory");
    if (bar_ready(bar, parity)) return true;
    const long long start = clock64();
    while (!bar_ready(bar, parity))
      if (clock64() - start > kClusterPatience) return false;
    return true;
  }
};

// A CTA's share of one matrix, and this thread's row of it.
template <class T>
struct ClusterSlice {
  int32_t parts;
  ClusterRow mine;
  const ClusterNz<T>* nz;
  const ClusterPart* apart;
  bool has_row;
};

template <class T>
__device__ __forceinline__ ClusterSlice<T> load_slice(const CsrView<T>& a, const ClusterRows& cr,
                                                      int rank, ClusterNz<T>* nz,
                                                      ClusterPart* apart) {
  const int32_t t = threadIdx.x, threads = static_cast<int32_t>(blockDim.x);
  ClusterSlice<T> s;
  const int32_t rb = cr.bounds[rank], re = cr.bounds[rank + 1];
  const int32_t p0 = cr.part_start[rank];
  s.parts = cr.part_start[rank + 1] - p0;
  for (int32_t i = t; i < s.parts; i += threads) apart[i] = cr.part[p0 + i];
  s.apart = apart;
  s.has_row = t < re - rb;
  s.mine = s.has_row ? cr.row[rb + t] : ClusterRow{0, 0, 0, 0};
  const int32_t z0 = a.start[rb], nnz = a.start[re] - z0;
  for (int32_t k = t; k < nnz; k += threads) {
    ClusterNz<T> z;
    z.place = cr.place[z0 + k];
    z.val = a.value[z0 + k];
    nz[cr.entry[z0 + k]] = z;
  }
  s.nz = nz;
  return s;
}

// The sum of `count` nonzeros, kClusterStride entries apart from `first`,
// against `x`, in order; loads run a few nonzeros ahead of the adds.
template <bool kStack, class T>
__device__ __forceinline__ T serial_sum(const ClusterNz<T>* nz, const T* x, int32_t first,
                                        int32_t count) {
  constexpr int kAhead = 8;
  T s = 0;
  for (int32_t k = 0; k < count; k += kAhead) {
    // Past the end the last nonzero is read again and not added: no branches.
    ClusterNz<T> z[kAhead];
    T xv[kAhead];
#pragma unroll
    for (int i = 0; i < kAhead; ++i) z[i] = nz[first + kClusterStride * min(k + i, count - 1)];
#pragma unroll
    for (int i = 0; i < kAhead; ++i) xv[i] = x[z[i].place];
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      const T next = kStack ? madd(s, z[i].val, xv[i]) : strict_add(s, strict_mul(z[i].val, xv[i]));
      s = k + i < count ? next : s;
    }
  }
  return s;
}

// The sum of this thread's row against the CTA's copy `xs`.
template <bool kStack, class T>
__device__ __forceinline__ T cluster_sum(const ClusterSlice<T>& a, const T* xs, T* part) {
  const int32_t t = threadIdx.x, threads = static_cast<int32_t>(blockDim.x);
  // The sums apart go to the last threads, the rows are the first ones.
  if constexpr (kStack) {
    for (int32_t i = threads - 1 - t; i < a.parts; i += threads) {
      const ClusterPart d = a.apart[i];
      part[d.slot] = serial_sum<true>(a.nz, xs, d.first, d.count);
    }
  } else {
    const int warps = threads / 32, lane = t % 32;
    for (int32_t i = warps - 1 - t / 32; i < a.parts; i += warps) {
      const ClusterPart d = a.apart[i];
      constexpr int kAhead = 4;  // loads of up to 128 nonzeros before the first add
      T s = 0;
      for (int32_t k = lane; k < d.count; k += 32 * kAhead) {
        ClusterNz<T> z[kAhead];
        T x[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) z[u] = a.nz[d.first + min(k + 32 * u, d.count - 1)];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) x[u] = xs[z[u].place];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
          const T next = strict_add(s, strict_mul(z[u].val, x[u]));
          s = k + 32 * u < d.count ? next : s;
        }
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1)
        s = strict_add(s, __shfl_down_sync(0xffffffffu, s, off));
      if (lane == 0) part[d.slot] = s;
    }
  }
  T sum = 0;
  if (a.has_row && !a.mine.apart) {
    sum = serial_sum<kStack>(a.nz, xs, a.mine.first, a.mine.count);
    if (kStack) sum = add(static_cast<T>(0), sum);
  }
  if (a.parts > 0) {  // the same for every thread of the CTA
    __syncthreads();
    if (a.has_row && a.mine.apart) {
      if (kStack)
        for (int32_t g = 0; g < a.mine.count; ++g) sum = add(sum, part[a.mine.first + g]);
      else
        sum = part[a.mine.first];
    }
  }
  return sum;
}

// `len` iterations (at most kClusterMaxLen) from iteration s.it0 of a chunk:
// K~'y with the primal step, then K~ x_bar with the dual step; cluster k runs
// case k. `flags` is every iteration's epilogue flags, `last_flags` the last
// one's. Every CTA has at least as many threads as rows of either matrix.
// Dynamic shared memory: ClusterLayout.
//
// Launched with programmatic stream serialisation: the next launch's CTAs
// start where they fit and load what no launch of the chunk writes while this
// one still runs.
template <class T, bool kStack>
__global__ void __launch_bounds__(kClusterThreadsMax)
    cluster_chunk_kernel(CsrView<T> kt, ClusterRows ktr, CsrView<T> k, ClusterRows kr,
                         ClusterStep<T> s, int32_t len, uint32_t flags, uint32_t last_flags) {
  extern __shared__ __align__(16) unsigned char cluster_smem[];
  pdl_launch();
  const auto cluster = cooperative_groups::this_cluster();
  const int rank = static_cast<int>(cluster.block_rank());
  const int ctas = static_cast<int>(cluster.num_blocks());
  const int32_t kase = static_cast<int32_t>(blockIdx.x) / ctas;
  const int32_t K = s.K, t = threadIdx.x;
  const StepParams P = s.p[kase];
  if (!P.active) return;
  const bool accumulate = (flags & kAccumulate) != 0;
  const ClusterLayout lay = ClusterLayout::of<T>(ctas, ktr, kr, len);
  T* xs = reinterpret_cast<T*>(cluster_smem + lay.xs);
  T* ys = reinterpret_cast<T*>(cluster_smem + lay.ys);
  T* part = reinterpret_cast<T*>(cluster_smem + lay.part);
  T* wt = reinterpret_cast<T*>(cluster_smem + lay.wt);
  T* my_x = xs + rank * ktr.stride;
  T* my_y = ys + rank * kr.stride;
  const uint32_t bars = smem_addr(cluster_smem + lay.bars);
  const Exchange ex{bars, smem_addr(my_x), static_cast<uint32_t>(sizeof(T)) * ktr.stride, rank,
                    ctas};
  const Exchange ey{bars + 8, smem_addr(my_y), static_cast<uint32_t>(sizeof(T)) * kr.stride, rank,
                    ctas};
  if (t == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(ex.bar) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(ey.bar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  cluster_arrive();  // every CTA runs and its mbarriers are ready
  const ClusterSlice<T> st =
      load_slice(kt, ktr, rank, reinterpret_cast<ClusterNz<T>*>(cluster_smem + lay.nzt),
                 reinterpret_cast<ClusterPart*>(cluster_smem + lay.partt));
  const ClusterSlice<T> sk =
      load_slice(k, kr, rank, reinterpret_cast<ClusterNz<T>*>(cluster_smem + lay.nzk),
                 reinterpret_cast<ClusterPart*>(cluster_smem + lay.partk));
  const int32_t j = st.mine.row, i = sk.mine.row;
  const size_t ej = (size_t)j * K + kase, ei = (size_t)i * K + kase;
  const bool cone = i >= s.num_eq;
  T c = 0, lo = 0, hi = 0, q = 0, floor_v = 0;
  if (st.has_row) {
    c = s.c[ej];
    lo = s.lo[ej];
    hi = s.hi[ej];
  }
  if (sk.has_row) {
    q = s.q[ei];
    if (s.ylo) floor_v = s.ylo[ei];
  }
  const T tau = static_cast<T>(P.tau), sigma = static_cast<T>(P.sigma),
          gamma = static_cast<T>(P.gamma), eta = static_cast<T>(P.eta);
  const uint32_t mode0 = step_mode(P, s.it0), mode1 = step_mode(P, s.it0 + 1);
  for (int32_t it = t; it < len; it += static_cast<int32_t>(blockDim.x)) {
    const double w = s.w_table[(size_t)(s.it0 + it) * K + kase];
    wt[2 * it] = static_cast<T>(w);
    wt[2 * it + 1] = static_cast<T>(1.0 - w);
  }
  // ---- what the launch before writes
  pdl_wait();
  T x = 0, ax = 0, sx = 0, y = 0, kx = 0, ay = 0, ak = 0, sy = 0;
  if (st.has_row) {
    x = s.x[ej];
    ax = s.anchor[ej];
    if (accumulate) sx = s.sum_x[ej];
  }
  if (sk.has_row) {
    y = s.y[ei];
    kx = s.kx[ei];
    ay = s.anchor_y[ei];
    ak = s.anchor_kx[ei];
    if (accumulate) sy = s.sum_y[ei];
    my_y[t] = y;
  }
  cluster_wait();
  bool bad = ey.send(false);  // its __syncthreads also covers the slices and the weights
  for (int32_t it = 0; it < len; ++it) {
    const uint32_t mode = it == 0 ? mode0 : mode1;
    const T w = wt[2 * it], wc = wt[2 * it + 1];
    const uint32_t parity = static_cast<uint32_t>(it) & 1u;
    bad = !ey.receive(parity);
    const T kty = cluster_sum<kStack>(st, ys, part);
    T d = 0;
    if (st.has_row) {
      const PrimalMove<T> o = primal_move<T>(x, c, lo, hi, ax, kty, tau, gamma, w, wc, mode);
      my_x[t] = o.x_bar;
      x = o.next;
      d = o.d;
    }
    bad = ex.send(bad);
    if (bad) break;  // the same for every thread of the CTA
    if (st.has_row) {
      if (mode & kStepAnchor) ax = x;
      if (accumulate) sx = add(sx, mul(eta, x));
      if (it == len - 1 && (last_flags & kWriteDelta)) s.dx[ej] = d;
    }
    bad = !ex.receive(parity);
    const T bar = cluster_sum<kStack>(sk, xs, part);
    if (sk.has_row) {
      const DualMove<T> o =
          dual_move<T>(y, q, kx, cone, floor_v, ay, ak, bar, sigma, gamma, w, wc, mode);
      my_y[t] = o.next_y;
      y = o.next_y;
      kx = o.next_k;
      d = o.d;
    }
    if (it < len - 1) {
      bad = ey.send(bad);
      if (bad) break;
    }
    if (sk.has_row) {
      if (mode & kStepAnchor) {
        ay = y;
        ak = kx;
      }
      if (accumulate) sy = add(sy, mul(eta, y));
      if (it == len - 1 && (last_flags & kWriteDelta)) s.dy[ei] = d;
    }
  }
  if (bad) *s.status = kSyncTimedOut;
  if (st.has_row) {
    s.x[ej] = x;
    if (mode0 & kStepAnchor) s.anchor[ej] = ax;
    if (accumulate) s.sum_x[ej] = sx;
  }
  if (sk.has_row) {
    s.y[ei] = y;
    s.kx[ei] = kx;
    if (mode0 & kStepAnchor) {
      s.anchor_y[ei] = ay;
      s.anchor_kx[ei] = ak;
    }
    if (accumulate) s.sum_y[ei] = sy;
  }
  // No CTA leaves while a peer's copy may still read or write its memory.
  cluster_arrive();
  cluster_wait();
}

}  // namespace anu
