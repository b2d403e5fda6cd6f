// (P)CG for systems whose iterations are bound by launches and latency rather than by the
// matrix: one thread-block cluster runs them all in one kernel.  Same recurrences and stopping
// rule as the three-kernel loop in gf_solve.cu (SPRmatrix::CPU_CG,
// src/SPRmatrix/SPRmatrix.cc:405-480).
//
// A CTA holds its slices of the matrix (node-block slices, gf_sell.cu) in shared memory for the
// whole solve.  A slice's 32 nodes are a warp, each lane with its rows of r and p in registers;
// where slices are few, further warps take a share of the slice's neighbours in the product.
// Where a whole direction vector fits besides, every CTA keeps one and a node's owner stores its
// new values to the CTAs that read them (a mask per node, from the columns), so that the product
// gathers from its own shared memory; else the direction lives in the CTAs' shared memory, a
// range of nodes to a CTA, and is gathered from there.  An iteration exchanges three things: p.q,
// then (r.z, r.r), then the new p.  With copies they are asynchronous stores that complete on a
// barrier of the CTA they go to, which waits for their bytes alone; a buffer is written again only
// after an answer that its reader sends when it is done with it.  Waits are bounded; a CTA
// that gives up tells the others and leaves the iteration as a whole, the others follow when their
// own waits run out, and the host starts again with the three-kernel loop.  Without copies there
// is a cluster barrier after each.  Each CTA adds all parts of a sum in the same order, so a solve is
// reproducible.
//
// Microseconds per iteration (FP64 Jacobi-PCG; the same with cluster barriers; gathering from the
// other CTAs; the three-kernel loop): Q4 64 x 64 3.0 (3.4; 3.7; 9.8), Q8 20 x 20 3.1 (3.5; 4.0;
// 9.9), Brick8 6^3 4.0 (4.4; 5.8; 15.4), Brick20 4^3 5.2 (5.5; 8.1; 22.2); FP32 Brick8 11^3 5.1
// (5.3; 9.0).  What is left is latency: sums over a warp, a CTA and the cluster, twice.  The matrix
// has to fit the 16 CTAs' shared memory (3.4 MB with the vectors): read from L2 instead, 16 SMs
// took 22.6 us on Q8 64 x 64, where the loop takes 10.4 on all of them, and a grid-wide version
// (148 CTAs, sums through global memory) took 13.  Storing z with r.z, so that readers form p
// themselves, cost more in gathers from other CTAs than the barrier it saved (Q4 64 4.3 us).
#include <algorithm>

#include "gf_internal.cuh"

namespace {

constexpr int kCluster = 16;          // CTAs (a size beyond 8 is opt-in)
constexpr int kThreadsMax = 1024;
constexpr size_t kSmemMax = 220 * 1024;   // per CTA: one to an SM

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Address of this CTA's shared address `a` in CTA `rank`
__device__ __forceinline__ uint32_t map_rank(uint32_t a, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ double ld_cluster(uint32_t a, double) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float ld_cluster(uint32_t a, float) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void st_cluster(uint32_t a, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void st_cluster(uint32_t a, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
// The DIM values of a node: from the cluster, from this CTA's shared memory, and to the cluster
template <int DIM, typename V>
__device__ __forceinline__ void ld_node(uint32_t a, V (&v)[DIM]) {
  if constexpr (DIM == 2 && sizeof(V) == 8) {
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "r"(a) : "memory");
  } else if constexpr (DIM == 2) {
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v[0]), "=f"(v[1]) : "r"(a) : "memory");
  } else {
#pragma unroll
    for (int c = 0; c < DIM; ++c) v[c] = ld_cluster(a + c * (uint32_t)sizeof(V), V(0));
  }
}

template <int DIM, typename V>
__device__ __forceinline__ void ld_node(const unsigned char* a, V (&v)[DIM]) {
  if constexpr (DIM == 2 && sizeof(V) == 8) {
    const double2 q = *reinterpret_cast<const double2*>(a);
    v[0] = q.x;
    v[1] = q.y;
  } else if constexpr (DIM == 2) {
    const float2 q = *reinterpret_cast<const float2*>(a);
    v[0] = q.x;
    v[1] = q.y;
  } else {
#pragma unroll
    for (int c = 0; c < DIM; ++c) v[c] = reinterpret_cast<const V*>(a)[c];
  }
}
template <int DIM, typename V>
__device__ __forceinline__ void st_node(uint32_t a, const V (&v)[DIM]) {
  if constexpr (DIM == 2 && sizeof(V) == 8) {
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v[0]), "d"(v[1]) : "memory");
  } else if constexpr (DIM == 2) {
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v[0]), "f"(v[1]) : "memory");
  } else {
#pragma unroll
    for (int c = 0; c < DIM; ++c) st_cluster(a + c * (uint32_t)sizeof(V), v[c]);
  }
}

// Stores that complete on a barrier in the shared memory of the CTA they go to (their bytes count
// towards its transaction count)
__device__ __forceinline__ void st_async(uint32_t a, double v, uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(a),
               "l"(__double_as_longlong(v)), "r"(bar)
               : "memory");
}
template <int DIM>
__device__ __forceinline__ void st_async_node(uint32_t a, const double (&v)[DIM], uint32_t bar) {
  if constexpr (DIM == 2)
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(a),
                 "l"(__double_as_longlong(v[0])), "l"(__double_as_longlong(v[1])), "r"(bar)
                 : "memory");
  else
#pragma unroll
    for (int c = 0; c < DIM; ++c) st_async(a + 8 * c, v[c], bar);
}
template <int DIM>
__device__ __forceinline__ void st_async_node(uint32_t a, const float (&v)[DIM], uint32_t bar) {
  if constexpr (DIM == 2)
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];" ::"r"(a),
                 "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(bar)
                 : "memory");
  else
#pragma unroll
    for (int c = 0; c < DIM; ++c)
      asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(a + 4 * c),
                   "r"(__float_as_uint(v[c])), "r"(bar)
                   : "memory");
}
// One thread per phase: the bytes that the phase waits for
__device__ __forceinline__ void bar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_try(uint32_t bar, uint32_t parity) {   // for a short while
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\t"
               "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
               "selp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok)
               : "r"(bar), "r"(parity)
               : "memory");
  return ok;
}
// Waits for the phase of parity `parity`; false if it does not come in `tries`, each of which the
// hardware suspends for a while.  (A limit by the clock, read at each try or in a second loop after
// the tries, or tries that are no constant cost 0.1 to 0.2 us an iteration on Q4 64 x 64.)
constexpr int kTries = 20000;
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, int tries) {
  for (int k = 0; k < tries; ++k)
    if (bar_try(bar, parity)) return true;
  return false;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sums N values (of the first S warps) over the cluster; `part` is this CTA's [N][kCluster].  The
// CTA's parts are sent to every CTA and are awaited there: on `bar` (ASYNC), else by a cluster
// barrier.  late: a wait of this thread has run out.  True, the same for the whole CTA, if one of
// its threads came late; nothing was sent then.
template <int N, bool ASYNC>
__device__ __forceinline__ bool cluster_sum(double (&v)[N], int S, double* sh, double* part,
                                            uint32_t part_addr, uint32_t bar, uint32_t parity,
                                            int tries, bool& late) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp < S) {
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const double s = warp_sum(v[k]);
      if (lane == 0) sh[k * 32 + warp] = s;
    }
  }
  if constexpr (ASYNC) {
    if (__syncthreads_or(late)) return true;
  } else {
    __syncthreads();
  }
  if (warp == 0) {
    if (ASYNC && lane == 0) bar_expect(bar, N * kCluster * 8);
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const double s = warp_sum(lane < S ? sh[k * 32 + lane] : 0.0);
      const uint32_t mine = part_addr + (k * kCluster + cluster_rank()) * 8;
      if (lane < kCluster) {
        if constexpr (ASYNC)
          st_async(map_rank(mine, lane), s, map_rank(bar, lane));
        else
          st_cluster(map_rank(mine, lane), s);
      }
    }
  }
  if constexpr (ASYNC)
    late = !bar_wait(bar, parity, tries);
  else
    cluster_sync();
#pragma unroll
  for (int k = 0; k < N; ++k) {
    double s = part[k * kCluster + (lane & (kCluster - 1))];
#pragma unroll
    for (int o = kCluster / 2; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    v[k] = s;
  }
  return false;
}

struct ClusterArgs {
  int nnodes, S, H, iters, jacobi;   // S slices per CTA, H warps per slice
  double eps;
  int late;                          // LATE: CTA and 256 times the number of its wait that runs out
  const int32_t* __restrict__ perm;
  const int32_t* __restrict__ width;
  const int64_t* __restrict__ off;
  const int32_t* __restrict__ col;
  SolveScalars* sc;
};

// Shared memory besides the slices: sums, directions (COPY: all of them, and the masks), x and
// 1 / diagonal, partial products.
template <int DIM, typename V, bool COPY>
__host__ __device__ constexpr size_t cluster_vectors(int S, int H, int nnodes) {
  return sizeof(double) * (3 * kCluster + 64 + 4) + sizeof(V) * DIM * 32 * (size_t)S * (1 + H) +
         (COPY ? (sizeof(V) * DIM * nnodes + 15) / 16 * 16 + sizeof(uint32_t) * 32 * S
               : sizeof(V) * DIM * 32 * (size_t)S);
}

// LATE: for the tests, one wait of one CTA runs out (and soon those of the others).
template <int DIM, typename V, bool COPY, bool LATE>
__global__ void __launch_bounds__(kThreadsMax)
k_pcg_cluster(ClusterArgs A, const V* __restrict__ val, const V* __restrict__ dinv,
              V* __restrict__ x, V* __restrict__ r, V* __restrict__ p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SolveScalars* sc = A.sc;
  if (sc->done) return;   // the same for every CTA, before any barrier
  const int S = A.S, H = A.H, per = 32 * S;
  double* partA = reinterpret_cast<double*>(smem_raw);       // [1][kCluster]
  double* partB = partA + kCluster;                          // [2][kCluster]
  double* sh = partB + 2 * kCluster;                         // [2][32]
  // directions: [per][DIM] of this CTA's nodes, or [nnodes][DIM] where copies are kept
  uint64_t* bars = reinterpret_cast<uint64_t*>(sh + 64);     // p.q; r.z and r.r; directions
  uint32_t* count = reinterpret_cast<uint32_t*>(bars + 3);   // nodes whose directions come here
  uint32_t* gave_up = count + 1;                             // a CTA's wait has run out
  V* sp = reinterpret_cast<V*>(bars + 4);
  uint32_t* smask = reinterpret_cast<uint32_t*>(                // [per] CTAs that read a node's
      reinterpret_cast<unsigned char*>(sp) + (sizeof(V) * DIM * A.nnodes + 15) / 16 * 16);
  V* sx = COPY ? reinterpret_cast<V*>(smask + per) : sp + (size_t)per * DIM;  // [DIM][per] slots
  V* sd = sx + (size_t)per * DIM;                            // [DIM][per]
  V* sq = sd + (size_t)per * DIM;                            // [H - 1][DIM][per]
  V* sv = sq + (size_t)per * DIM * (H - 1);                  // the CTA's slices: values, then
  const uint32_t sp_addr = (uint32_t)__cvta_generic_to_shared(sp);
  const uint32_t pa = (uint32_t)__cvta_generic_to_shared(partA), pb = (uint32_t)__cvta_generic_to_shared(partB);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ks = warp % S, h = warp / S;                     // slice of the CTA, share of it
  const int nslice = (A.nnodes + 31) >> 5;
  const int k0 = min(nslice, (int)blockIdx.x * S), k1 = min(nslice, k0 + S);
  const int64_t o0 = A.off[k0], cnt = A.off[k1] - o0;
  uint32_t* sa = reinterpret_cast<uint32_t*>(sv + cnt * (DIM * DIM));   // addresses of the columns' p
  auto home = [&](int b) {   // address of node b's direction
    return map_rank(sp_addr + (uint32_t)((b % per) * DIM * sizeof(V)), (uint32_t)(b / per));
  };
  auto mask_of = [&](int b) {   // address of node b's mask
    return map_rank((uint32_t)__cvta_generic_to_shared(smask) + (uint32_t)(b % per) * 4, (uint32_t)(b / per));
  };
  const uint32_t bar = (uint32_t)__cvta_generic_to_shared(bars);
  if constexpr (COPY) {
    for (int i = threadIdx.x; i < per; i += blockDim.x) smask[i] = 0;
    if (threadIdx.x == 0) {
      *count = *gave_up = 0;
#pragma unroll
      for (int k = 0; k < 3; ++k)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar + 8 * k) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    cluster_sync();
  }
  for (int64_t i = threadIdx.x; i < cnt * (DIM * DIM); i += blockDim.x) sv[i] = val[o0 * (DIM * DIM) + i];
  for (int64_t i = threadIdx.x; i < cnt; i += blockDim.x) {
    const int b = A.col[o0 + i];
    if constexpr (COPY) {
      sa[i] = (uint32_t)(b * DIM * sizeof(V));
      asm volatile("red.shared::cluster.or.b32 [%0], %1;" ::"r"(mask_of(b)), "r"(1u << cluster_rank()) : "memory");
    } else {
      sa[i] = home(b);
    }
  }
  int w = 0;
  const V* vp = sv + lane;
  const uint32_t* ap = sa + lane;
  if (k0 + ks < k1) {
    w = A.width[k0 + ks];
    const int64_t o = A.off[k0 + ks] - o0;
    vp += o * (DIM * DIM);
    ap += o;
  }
  const int li = ks * 32 + lane, slot = k0 * 32 + li;
  const bool on = h == 0 && k0 + ks < k1 && slot < A.nnodes;
  const int a = on ? A.perm[slot] : 0;
  uint32_t mine = 0, readers = 0;
  if constexpr (COPY) {
    cluster_sync();   // the masks are complete
    for (int i = threadIdx.x; i < per; i += blockDim.x)
      for (uint32_t m = smask[i]; m; m &= m - 1)
        asm volatile("red.shared::cluster.add.u32 [%0], 1;" ::"r"(map_rank(bar + 24, __ffs(m) - 1)) : "memory");
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(readers) : "r"(mask_of(a)) : "memory");
    mine = sp_addr + (uint32_t)(a * DIM * sizeof(V));
    if (!on) readers = 0;
  } else {
    mine = home(a);
  }
  // the lane's direction to where it is read
  auto publish = [&](const V (&v)[DIM]) {
    if constexpr (COPY) {
      for (uint32_t m = readers; m; m &= m - 1) {
        const uint32_t to = __ffs(m) - 1;
        st_async_node<DIM>(map_rank(mine, to), v, map_rank(bar + 16, to));
      }
    } else if (on) {
      st_node<DIM, V>(mine, v);
    }
  };
  V rv[DIM], pv[DIM];
#pragma unroll
  for (int c = 0; c < DIM; ++c) {
    const int64_t i = (int64_t)a * DIM + c;
    rv[c] = on ? r[i] : V(0);
    pv[c] = on ? p[i] : V(0);
    if (h == 0) {
      sx[c * per + li] = on ? x[i] : V(0);
      sd[c * per + li] = on ? (A.jacobi ? dinv[i] : V(1)) : V(0);
    }
  }
  if (COPY) cluster_sync();   // the counts are complete
  const uint32_t bytes = COPY ? *count * (uint32_t)(DIM * sizeof(V)) : 0;
  if (COPY && threadIdx.x == 0) bar_expect(bar + 16, bytes);
  publish(pv);
  bool late = false;
  auto tries = [&](int wait) {
    return !LATE ? kTries : A.late == (int)cluster_rank() + 256 * wait ? 0 : 2;
  };
  double rz = sc->rzn, rr = sc->rr, tol2 = sc->tol2;
  int iter = sc->iter, done = 0;
  const bool fresh = iter == 0;
  if (fresh) {   // p = z: the first sums again, in this kernel's fixed order
    double two[2] = {0.0, 0.0};
    if (h == 0)
#pragma unroll
      for (int c = 0; c < DIM; ++c) {
        two[0] += (double)rv[c] * (double)pv[c];
        two[1] += (double)rv[c] * (double)rv[c];
      }
    cluster_sum<2, false>(two, S, sh, partB, pb, 0, 0, 0, late);
    rz = two[0];
    rr = two[1];
    tol2 = A.eps * A.eps * rr;
  }
  const double rr0 = rr;
  const int maxit = sc->maxit;
  if (!COPY) cluster_sync();
  for (int step = 0; step < A.iters; ++step) {
    const uint32_t parity = step & 1;
    if (COPY) late = !bar_wait(bar + 16, parity, tries(3 * step));
    V q[DIM];
#pragma unroll
    for (int c = 0; c < DIM; ++c) q[c] = V(0);
#pragma unroll 4
    for (int s = h; s < w; s += H) {
      V g[DIM];
      if constexpr (COPY)
        ld_node<DIM, V>(reinterpret_cast<const unsigned char*>(sp) + ap[32 * s], g);
      else
        ld_node<DIM, V>(ap[32 * s], g);
      const V* e = vp + s * (DIM * DIM * 32);
#pragma unroll
      for (int c = 0; c < DIM; ++c)
#pragma unroll
        for (int c2 = 0; c2 < DIM; ++c2) q[c] += e[(c * DIM + c2) * 32] * g[c2];
    }
    if (H > 1) {
      if (h > 0)
#pragma unroll
        for (int c = 0; c < DIM; ++c) sq[((h - 1) * DIM + c) * per + li] = q[c];
      __syncthreads();
      if (h == 0)
        for (int m = 0; m < H - 1; ++m)
#pragma unroll
          for (int c = 0; c < DIM; ++c) q[c] += sq[(m * DIM + c) * per + li];
    }
    double sum[1] = {0.0};
#pragma unroll
    for (int c = 0; c < DIM; ++c) sum[0] += (double)pv[c] * (double)q[c];
    if (cluster_sum<1, COPY>(sum, S, sh, partA, pa, bar, parity, tries(3 * step + 1), late)) {
      done = 4;
      break;
    }
    const double pq = sum[0];
    const bool valid = pq > 0.0 && isfinite(pq);
    const V alpha = (V)(rz / pq);
    double two[2] = {0.0, 0.0};
    V zv[DIM];
#pragma unroll
    for (int c = 0; c < DIM; ++c) {
      zv[c] = V(0);
      if (h == 0 && valid) {
        sx[c * per + li] = fma(alpha, pv[c], sx[c * per + li]);
        rv[c] = fma(-alpha, q[c], rv[c]);
        zv[c] = rv[c] * sd[c * per + li];
        two[0] += (double)rv[c] * (double)zv[c];
        two[1] += (double)rv[c] * (double)rv[c];
      }
    }
    if (cluster_sum<2, COPY>(two, S, sh, partB, pb, bar + 8, parity, tries(3 * step + 2), late)) {
      done = 4;
      break;
    }
    if (!valid) {   // the same everywhere: who came late to p.q has left above
      done = 2;
      break;
    }
    if (COPY && __syncthreads_or(late)) {
      done = 4;
      break;
    }
    const V beta = (V)(two[0] / rz);
    rz = two[0];
    rr = two[1];
    ++iter;
    if (rr <= tol2) done = 1;
    else if (iter >= maxit) done = 3;
#pragma unroll
    for (int c = 0; c < DIM; ++c) pv[c] = fma(beta, pv[c], zv[c]);
    if (done || step + 1 == A.iters) break;   // nobody reads the next directions
    if (COPY && threadIdx.x == 0) bar_expect(bar + 16, bytes);
    publish(pv);
    if (!COPY) cluster_sync();
  }
  if (done == 4 && threadIdx.x < kCluster)   // to every CTA: CTA 0 may have ended as usual
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(map_rank(bar + 28, threadIdx.x)), "r"(1u) : "memory");
  cluster_sync();   // no CTA leaves while another may still write to it
  if (COPY && *gave_up) {
    // nothing is sent any more, but stores to a CTA that gave up may be under way: 0.1 ms
    const long long t0 = clock64();
    for (int k = 0; k < 100000 && clock64() - t0 < 200000; ++k) __nanosleep(200);
    done = 4;
    cluster_sync();
  }
  if (on)
#pragma unroll
    for (int c = 0; c < DIM; ++c) {
      const int64_t i = (int64_t)a * DIM + c;
      x[i] = sx[c * per + li];
      r[i] = rv[c];
      p[i] = pv[c];
    }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (fresh) {
      sc->rr0 = rr0;
      sc->tol2 = tol2;
    }
    sc->rzn = rz;
    sc->rr = rr;
    sc->iter = iter;
    sc->done = done;
  }
}

template <int DIM, typename V, bool COPY>
gf_status run_cluster_as(gf_ctx* ctx, const V* val, const V* dinv, V* x, V* r, V* p, double eps,
                         int iters, int* ran) {
  *ran = kPcgNotRun;
  if (iters < 1) return GF_OK;
  const int nslice = (ctx->nnodes + 31) / 32;
  const int S = (nslice + kCluster - 1) / kCluster;
  if (S > kThreadsMax / 32) return GF_OK;
  // Gathers from other CTAs: about 3 ns (2-D: 2 ns) for each separate piece that a warp's lanes
  // read.  Us an iteration by pieces per CTA, and of the three-kernel loop: FP32 Brick8 13^3 965
  // 10.5, 2014 13.1, 3093 17.0, 9187 37.1, loop 13.5; FP64 Brick8 10^3 480 9.3, 2202 14.7, 3047
  // 15.8, loop 14.9; FP32 Q4 124^2 549 5.0, 2680 9.0, 3870 11.5, 7662 24.4, loop 11.0; FP64 Q4 85^2
  // 265 4.3, 2767 8.7, 3458 11.7, loop 10.7 (ordered meshes first, random ones last).
  const double pieces = (double)S * 32 * (ctx->W / DIM) * (DIM == 2 ? 1 : 3) * ctx->gather;
  if (!COPY && pieces > (DIM == 2 ? 3300 : 2100)) return GF_OK;
  // a CTA's slices at the widest row
  const size_t slices = (size_t)S * 32 * (ctx->W / DIM) * (DIM * DIM * sizeof(V) + 4);
  int H = 1;
  while (S * H * 2 <= 16 && cluster_vectors<DIM, V, COPY>(S, H * 2, ctx->nnodes) + slices <= kSmemMax) H *= 2;
  const size_t sm = cluster_vectors<DIM, V, COPY>(S, H, ctx->nnodes) + slices;
  if (sm > kSmemMax) return GF_OK;
  auto kern = k_pcg_cluster<DIM, V, COPY, false>;
  if constexpr (DIM == 2 && sizeof(V) == 8 && COPY) {
    if (ctx->pcg_late >= 0) kern = k_pcg_cluster<DIM, V, COPY, true>;
  }
  GF_CUDA(ctx, gf_smem_attr(kern, sm));
  GF_CUDA(ctx, gf_func_attr((const void*)kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  ClusterArgs A{ctx->nnodes, S, H, iters, dinv != nullptr, eps, ctx->pcg_late, ctx->d_sell_perm,
                ctx->d_sell_w, ctx->d_sell_off, ctx->d_sell_col, ctx->d_scal};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kCluster;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(kCluster);
  cfg.blockDim = dim3(S * H * 32);
  cfg.dynamicSmemBytes = sm;
  cfg.stream = ctx->stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, kern, A, val, dinv, x, r, p) != cudaSuccess) {
    cudaGetLastError();   // no room for such a cluster here: nothing was done
    return GF_OK;
  }
  ctx->launches++;
  GF_CUDA(ctx, cudaMemcpyAsync(ctx->h_pinned, ctx->d_scal, sizeof(SolveScalars), cudaMemcpyDeviceToHost,
                               ctx->stream));
  GF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  *ran = static_cast<const SolveScalars*>(ctx->h_pinned)->done == 4 ? kPcgGaveUp : kPcgRan;
  return GF_OK;
}

// With copies of the direction where they fit.
template <int DIM, typename V>
gf_status run_cluster(gf_ctx* ctx, const V* val, const V* dinv, V* x, V* r, V* p, double eps, int iters,
                      int* ran) {
  const gf_status st = run_cluster_as<DIM, V, true>(ctx, val, dinv, x, r, p, eps, iters, ran);
  if (st != GF_OK || *ran != kPcgNotRun) return st;
  return run_cluster_as<DIM, V, false>(ctx, val, dinv, x, r, p, eps, iters, ran);
}

}  // namespace

// Runs up to `iters` iterations of the (P)CG to the tolerance eps whose state is in x, r, p and the
// context's scalars (iter, rr, rzn, done updated and read back to the pinned copy).  *ran =
// kPcgNotRun: the system is not one for this kernel, and nothing was done; kPcgGaveUp: a wait ran
// out, and the state is lost.  dinv = null: no preconditioner.
gf_status gf_pcg_cluster(gf_ctx* ctx, const double* val, const double* dinv, double* x, double* r,
                         double* p, double eps, int iters, int* ran) {
  *ran = kPcgNotRun;
  if (ctx->sell_bdim == 2) return run_cluster<2, double>(ctx, val, dinv, x, r, p, eps, iters, ran);
  if (ctx->sell_bdim == 3) return run_cluster<3, double>(ctx, val, dinv, x, r, p, eps, iters, ran);
  return GF_OK;
}
gf_status gf_pcg_cluster(gf_ctx* ctx, const float* val, const float* dinv, float* x, float* r,
                         float* p, double eps, int iters, int* ran) {
  *ran = kPcgNotRun;
  if (ctx->sell_bdim == 2) return run_cluster<2, float>(ctx, val, dinv, x, r, p, eps, iters, ran);
  if (ctx->sell_bdim == 3) return run_cluster<3, float>(ctx, val, dinv, x, r, p, eps, iters, ran);
  return GF_OK;
}

// For the tests only: FP64 solves of 2-D systems with copies lose a wait (3 to an iteration) of a
// CTA; a negative CTA: none.
extern "C" __attribute__((visibility("default"))) void gftest_pcg_late(gf_ctx* ctx, int cta, int wait) {
  ctx->pcg_late = cta < 0 ? -1 : cta + 256 * wait;
}
