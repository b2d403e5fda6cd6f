// Owner-computes assembly of Q4, Q8 and Brick8 meshes (GF_SCATTER_OWNER, what
// GF_SCATTER_AUTO takes): every ELL entry of K is written exactly once, with coalesced
// stores; no global atomics, colouring or zero-fill, and the sum over a node's elements has
// a fixed order.  Same arithmetic as gf_assemble.cu (node-pair blocks lam1 g_i g_j^T +
// mu1 g_j g_i^T + mu1 (g_i . g_j) I, weighted by w detJ E), organised by rows.  Reference:
// the scatter of StiffAlgo::AssembleK (src/FEM/StiffAlgo.cc:304-401).
//
//   k_geometry       J^-1 and w detJ E of every (element, Gauss point).  Element-local
//                    coordinates x_i - x_0 are formed in FP64; J, J^-1 are FP64 for the FP64
//                    path and for FP32 elements whose max/min |detJ| over the Gauss points
//                    exceeds 10.
//   k_node_rows_2d   a thread per owned node walks the node's incident elements, forms its
//   k_node_rows_b8   block row of each element matrix from that geometry and adds it into the
//                    node's own rows of a shared-memory tile, which is then stored to K,
//                    padding included.
#include <algorithm>
#include <cmath>

#include "gf_elem.cuh"

namespace {

// ---------------------------------------------------------------------------
// Geometry layout.  An element's values (per Gauss point J^-1 row by row, then w detJ E) form
// 16-byte units.  Where consecutive nodes lie in elements of like numbers, IL = 8 consecutive
// elements interleave their units, so that the lanes of a warp, whose nodes walk those elements,
// read whole 128-byte lines: unit u of element e is at 16-byte index ((e / 8) * units + u) * 8 +
// e % 8.  On a scattered numbering (gf_ctx::scattered) a lane would read a sector and a line for
// each 16 bytes: there an element's units lie in one piece (IL = 1), whose sectors the lane uses
// whole.  Us per call with IL = 8 and 1, by the share of distinct groups of eight among the
// elements of 32 consecutive nodes (FP32; FP64):
//   Q8 512^2     0.11 164, 200; 316, 362   0.34 204, 202; 390, 369   1 296, 229; 709, 424
//   Q4 1024^2    0.15 130, 143; 205, 247   0.36 159, 156; 274, 282   1 281, 197; 503, 323
//   Brick8 80^3  0.15 425, 565; 1008, 1273 0.36 854, 690; 1722, 1598 1 2098, 784; 4373, 1634
// (0.27: Brick8 667, 600; 1373, 1434.)  In 3-D each layer of Gauss points (first natural
// coordinate) is padded to whole units.
template <int ET, typename T, int NG1, int IL>
struct Geo {
  static constexpr int DIM = gf_elem_info(ET).dim, GV = DIM * DIM + 1;
  static constexpr int U = 16 / (int)sizeof(T);                         // values per unit
  static constexpr int LAYERS = DIM == 3 ? NG1 : 1;
  static constexpr int PER = NG1 * NG1 * GV;                            // values per layer
  static constexpr int LU = (PER + U - 1) / U;                          // units per layer
  static constexpr int UNITS = LAYERS * LU;
  static constexpr size_t bytes(int nelem) { return (size_t)((nelem + IL - 1) / IL) * IL * UNITS * 16; }
  // unit 0 of element e; its other units are IL further on each
  template <typename P>
  __device__ __forceinline__ static P* at(P* geo, int e) {
    static_assert(IL == 1 || IL == 8, "shifts");
    if constexpr (IL == 1) return geo + (int64_t)e * UNITS;
    return geo + (int64_t)(e >> 3) * (UNITS * 8) + (e & 7);
  }
};

template <typename T> struct Unit;
template <> struct Unit<float> { using type = float4; };
template <> struct Unit<double> { using type = double2; };

__device__ __forceinline__ void unit_get(const float4& q, float* v) { v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w; }
__device__ __forceinline__ void unit_get(const double2& q, double* v) { v[0] = q.x; v[1] = q.y; }
__device__ __forceinline__ void unit_put(float4* p, const float* v) { *p = make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ void unit_put(double2* p, const double* v) { *p = make_double2(v[0], v[1]); }

// J^-1 and w detJ E of one Gauss point in R arithmetic, to out[GV]; returns |detJ|.
template <int ET, typename T, int NG1, typename R, int NEN, int DIM>
__device__ __forceinline__ R point_geometry(int g, const R (&X)[NEN][DIM], T Ee, T* out) {
  constexpr GpTable<ET, NG1> Tab = gf_gp_table<ET, NG1>();
  constexpr double w1[3] = {NG1 == 2 ? 1.0 : 5.0 / 9.0, NG1 == 2 ? 1.0 : 8.0 / 9.0, 5.0 / 9.0};
  const int gi = DIM == 2 ? g / NG1 : g / (NG1 * NG1);
  const int gj = DIM == 2 ? g % NG1 : (g / NG1) % NG1;
  const int gk = DIM == 2 ? 0 : g % NG1;
  const double wg = w1[gi] * w1[gj] * (DIM == 2 ? 1.0 : w1[gk]);
  R J[3][3], Ji[3][3];
#pragma unroll
  for (int a = 0; a < DIM; ++a)
#pragma unroll
    for (int c = 0; c < DIM; ++c) {
      R s = R(0);
#pragma unroll
      for (int i = 0; i < NEN; ++i)
        s += (sizeof(R) == 8 ? R(Tab.d64[(g * DIM + a) * NEN + i]) : R(Tab.d32[(g * DIM + a) * NEN + i])) * X[i][c];
      J[a][c] = s;
    }
  const R d = gf_det_inv<DIM, R>(J, Ji);
#pragma unroll
  for (int a = 0; a < DIM; ++a)
#pragma unroll
    for (int c = 0; c < DIM; ++c) out[a * DIM + c] = T(Ji[a][c]);
  out[DIM * DIM] = T(R(wg) * d) * Ee;
  return d < R(0) ? -d : d;
}

// All Gauss points of one element in R arithmetic; returns whether max/min |detJ| > 10.
template <int ET, typename T, int NG1, int IL, typename R, int NEN, int DIM>
__device__ __forceinline__ bool element_geometry(const R (&X)[NEN][DIM], T Ee,
                                                 typename Unit<T>::type* out) {
  using G = Geo<ET, T, NG1, IL>;
  R dmin = R(3.4e38), dmax = R(0);
#pragma unroll
  for (int l = 0; l < G::LAYERS; ++l) {
    T buf[G::LU * G::U];
#pragma unroll
    for (int k = G::PER; k < G::LU * G::U; ++k) buf[k] = T(0);
#pragma unroll
    for (int g = 0; g < NG1 * NG1; ++g) {
      const R d = point_geometry<ET, T, NG1, R>(l * NG1 * NG1 + g, X, Ee, buf + g * G::GV);
      dmin = d < dmin ? d : dmin;
      dmax = d > dmax ? d : dmax;
      // the units that this point completes
#pragma unroll
      for (int u = g * G::GV / G::U; u < ((g + 1) * G::GV) / G::U; ++u)
        unit_put(out + (l * G::LU + u) * IL, buf + u * G::U);
    }
    if constexpr (G::PER % G::U != 0)
      unit_put(out + (l * G::LU + G::LU - 1) * IL, buf + (G::LU - 1) * G::U);
  }
  return dmax > R(10) * dmin;
}

constexpr int kGT = 128;

// Geometry of element e to `out` (its unit 0).
template <int ET, typename T, int NG1, int IL>
__device__ __forceinline__ void one_element(int e, const int32_t* __restrict__ conn,
                                            const double* __restrict__ coords,
                                            const T* __restrict__ Eel, typename Unit<T>::type* out) {
  constexpr int NEN = gf_elem_info(ET).nen, DIM = gf_elem_info(ET).dim;
  double X[NEN][DIM];
  double x0[DIM];
#pragma unroll
  for (int i = 0; i < NEN; ++i) {
    const int node = __ldg(conn + (int64_t)e * NEN + i);
#pragma unroll
    for (int c = 0; c < DIM; ++c) {
      const double x = __ldg(coords + (int64_t)node * DIM + c);
      if (i == 0) x0[c] = x;
      X[i][c] = x - x0[c];
    }
  }
  const T Ee = __ldg(Eel + e);
  if constexpr (sizeof(T) == 4) {
    float Xf[NEN][DIM];
#pragma unroll
    for (int i = 0; i < NEN; ++i)
#pragma unroll
      for (int c = 0; c < DIM; ++c) Xf[i][c] = (float)X[i][c];
    if (!element_geometry<ET, T, NG1, IL, float>(Xf, Ee, out)) return;
  }
  element_geometry<ET, T, NG1, IL, double>(X, Ee, out);
}

// A thread per element: its local coordinates stay in registers and the Gauss rule is a
// compile-time table.  With IL = 8 the stores of a warp are whole lines by the layout; with IL = 1
// they pass through shared memory where the block's units fit 48 KB (all but FP64 Brick8 and
// Brick8 with 3^3 points): Q8 512^2 FP64 397 -> 362 us the assembly, Brick8 80^3 FP32 592 -> 565.
template <int ET, typename T, int NG1, int IL>
__global__ void __launch_bounds__(kGT)
k_geometry(int nelem, const int32_t* __restrict__ conn, const double* __restrict__ coords,
           const T* __restrict__ Eel, T* __restrict__ geo) {
  using G = Geo<ET, T, NG1, IL>;
  using UT = typename Unit<T>::type;
  constexpr int ROW = G::UNITS | 1;   // units of an element in shared memory
  constexpr bool kStage = IL == 1 && kGT * ROW * 16 <= 48 * 1024;
  __shared__ UT stage[kStage ? kGT * ROW : 1];
  const int e0 = blockIdx.x * kGT, e = e0 + threadIdx.x;
  UT* all = reinterpret_cast<UT*>(geo);
  if (e < nelem)
    one_element<ET, T, NG1, IL>(e, conn, coords, Eel, kStage ? stage + threadIdx.x * ROW : G::at(all, e));
  if constexpr (kStage) {
    __syncthreads();
    const int cnt = min(kGT, nelem - e0) * G::UNITS;
    for (int k = threadIdx.x; k < cnt; k += kGT)
      all[(int64_t)e0 * G::UNITS + k] = stage[k / G::UNITS * ROW + k % G::UNITS];
  }
}

// ---------------------------------------------------------------------------
// 2-D.  The CTA orders its nodes by degree (stable counting sort, highest first: the nodes
// of a warp walk the same number of elements and keep ascending rows).  Per Gauss point
// g_i = w detJ E J^-T dN_i (dN_i from shared memory: i is known at run time) and
// g_j = J^-T dN_j (dN_j instruction constants) form H_j += g_i g_j^T; FP32 takes two entries
// per packed FMA.
// Bound by issue and latency at the 16 warps per SM that the row tile leaves (Q8 512 x 512
// FP32: 128 us, issue slots 50%, L1 68%, K alone would take 41 us; 144 us before the next
// element's geometry was loaded ahead).  FP64 (Q8 301 x 173): 65 us, 104 us with a thread per
// (node, element) and shared-memory atomics.
constexpr int kDegBuckets = 32;

template <typename T> struct Vec2;
template <> struct Vec2<float> { using type = float2; };
template <> struct Vec2<double> { using type = double2; };

__device__ __forceinline__ double2 fma2(double2 a, double2 b, double2 c) {
  return make_double2(fma(a.x, b.x, c.x), fma(a.y, b.y, c.y));
}

template <int ET, typename T, int NG1, int NB>
size_t node_rows_2d_smem(int W) {
  return sizeof(T) * ((size_t)W * 2 * NB + 2 * NG1 * NG1 * gf_elem_info(ET).nen) +
         sizeof(int) * (3 * NB + 1 + (NB / 32 + 1) * kDegBuckets);
}

template <int ET, typename T, int NG1, int IL, int NB>
__global__ void __launch_bounds__(NB)
k_node_rows_2d(int nnodes, int n, int W, const int32_t* __restrict__ inc_off,
               const int32_t* __restrict__ inc, const uint8_t* __restrict__ inc_loc,
               const uint16_t* __restrict__ inc_slot, const T* __restrict__ geo,
               const AsmTables* __restrict__ tab, T lam1, T mu1, T* __restrict__ K) {
  using G = Geo<ET, T, NG1, IL>;
  using T2 = typename Vec2<T>::type;
  using UT = typename Unit<T>::type;
  constexpr int NEN = gf_elem_info(ET).nen, NGP = NG1 * NG1, RB = 2 * NB, NW = NB / 32;
  constexpr GpTable<ET, NG1> Tab = gf_gp_table<ET, NG1>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* tile = reinterpret_cast<T*>(smem_raw);                  // [W][RB]
  T2* sdN = reinterpret_cast<T2*>(tile + (size_t)W * RB);    // [NGP][NEN]
  int* soff = reinterpret_cast<int*>(sdN + NGP * NEN);       // [NB + 1]
  int* sord = soff + NB + 1;                                 // [NB] node of a thread
  int* spos = sord + NB;                                     // [NB] thread of a node
  int* wcnt = spos + NB;                                     // [NW][kDegBuckets]

  const int t = threadIdx.x;
  const int a0 = blockIdx.x * NB;
  const int na = min(NB, nnodes - a0);
  {
    uint4* z = reinterpret_cast<uint4*>(tile);
    for (int k = t; k < W * RB * (int)sizeof(T) / 16; k += NB) z[k] = make_uint4(0, 0, 0, 0);
  }
  for (int k = t; k < NGP * NEN; k += NB) {
    const int g = k / NEN, i = k - g * NEN;
    if constexpr (sizeof(T) == 4)
      sdN[k] = make_float2(tab->dN32[(g * 2) * NEN + i], tab->dN32[(g * 2 + 1) * NEN + i]);
    else
      sdN[k] = make_double2(tab->dN64[(g * 2) * NEN + i], tab->dN64[(g * 2 + 1) * NEN + i]);
  }
  for (int k = t; k <= na; k += NB) soff[k] = inc_off[a0 + k];
  for (int k = t; k < NW * kDegBuckets; k += NB) wcnt[k] = 0;
  __syncthreads();
  // A node's position is the count of nodes of higher degree plus the nodes of its degree
  // before it.  The node at position t is summed by thread t into tile row pair t, so a
  // warp's accesses fall on distinct banks; the store maps the pairs back to the nodes' rows.
  const int warp = t >> 5, lane = t & 31;
  const int bkt = t < na ? min(soff[t + 1] - soff[t], kDegBuckets - 1) : -1;
  const unsigned same = __match_any_sync(0xffffffffu, bkt);
  const int wrank = __popc(same & ((1u << lane) - 1u));
  if (bkt >= 0 && wrank == 0) wcnt[warp * kDegBuckets + bkt] = __popc(same);
  __syncthreads();
  if (t < 32) {
    // exclusive positions: lane t scans bucket 31 - t, warps in order
    const int b = kDegBuckets - 1 - t;
    int sum = 0;
#pragma unroll
    for (int w = 0; w < NW; ++w) sum += wcnt[w * kDegBuckets + b];
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (t >= o) incl += v;
    }
    int acc = incl - sum;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      const int c = wcnt[w * kDegBuckets + b];
      wcnt[w * kDegBuckets + b] = acc;
      acc += c;
    }
  }
  __syncthreads();
  if (bkt >= 0) {
    const int pos = wcnt[warp * kDegBuckets + bkt] + wrank;
    sord[pos] = t;
    spos[t] = pos;
  }
  __syncthreads();

  const int al = t < na ? sord[t] : 0;
  const int q0 = soff[al];
  const int deg = t < na ? soff[al + 1] - q0 : 0;
  T* myrows = tile + 2 * t;
  // The geometry of the next element is loaded into the registers that a few Gauss points of
  // the current one have just freed, so that its latency is covered by the other points.
  T gv[G::UNITS * G::U];
  const UT* ge = nullptr;
  int i = 0;
  uint32_t sn[NEN / 2];   // neighbour slots of the element's nodes
  auto meta = [&](int k) {
    const int64_t q = q0 + k;
    const int e = __ldg(inc + q);
    i = __ldg(inc_loc + q);
    ge = G::at(reinterpret_cast<const UT*>(geo), e);
    if constexpr (NEN == 8) {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(inc_slot + q * NEN));
      sn[0] = v.x; sn[1] = v.y; sn[2] = v.z; sn[3] = v.w;
    } else {
      const uint2 v = __ldg(reinterpret_cast<const uint2*>(inc_slot + q * NEN));
      sn[0] = v.x; sn[1] = v.y;
    }
  };
  if (deg > 0) {
    meta(0);
#pragma unroll
    for (int u = 0; u < G::UNITS; ++u) unit_get(__ldg(ge + u * IL), gv + u * G::U);
  }
  for (int k = 0; k < deg; ++k) {
    const T2* dn_i = sdN + i;
    uint32_t sw[NEN / 2];
#pragma unroll
    for (int j = 0; j < NEN / 2; ++j) sw[j] = sn[j];
    const bool more = k + 1 < deg;
    if (more) meta(k + 1);
    T2 H[NEN][2];   // H[j][a] = (H_j[a][0], H_j[a][1])
#pragma unroll
    for (int j = 0; j < NEN; ++j) H[j][0].x = H[j][0].y = H[j][1].x = H[j][1].y = T(0);
#pragma unroll
    for (int g = 0; g < NGP; ++g) {
      const T j00 = gv[g * 5], j01 = gv[g * 5 + 1], j10 = gv[g * 5 + 2], j11 = gv[g * 5 + 3];
      const T wd = gv[g * 5 + 4];   // w detJ E
      const T2 dn = dn_i[g * NEN];
      T2 g0, g1;
      g0.x = g0.y = fma(j01, dn.y, j00 * dn.x) * wd;
      g1.x = g1.y = fma(j11, dn.y, j10 * dn.x) * wd;
#pragma unroll
      for (int j = 0; j < NEN; ++j) {
        const T d0 = sizeof(T) == 4 ? T(Tab.d32[(g * 2) * NEN + j]) : T(Tab.d64[(g * 2) * NEN + j]);
        const T d1 = sizeof(T) == 4 ? T(Tab.d32[(g * 2 + 1) * NEN + j]) : T(Tab.d64[(g * 2 + 1) * NEN + j]);
        T2 gj;
        gj.x = fma(j01, d1, j00 * d0);
        gj.y = fma(j11, d1, j10 * d0);
        H[j][0] = fma2(g0, gj, H[j][0]);
        H[j][1] = fma2(g1, gj, H[j][1]);
      }
      // units that lie wholly in the points done since the last refill
      constexpr int STEP = 4;
      if ((g + 1) % STEP == 0 || g == NGP - 1) {
        const int from = (g / STEP) * STEP * 5 / G::U;
        const int to = g == NGP - 1 ? G::UNITS : (g + 1) * 5 / G::U;
        if (more)
#pragma unroll
          for (int u = from; u < to; ++u) unit_get(__ldg(ge + u * IL), gv + u * G::U);
      }
    }
    // V = lam1 H + mu1 H^T + mu1 tr(H) I; column b of V is rows (2 al, 2 al + 1) of tile
    // column 2 p + b.  The slots are distinct: a batch is read, added to and written back
    // together.
    constexpr int JB = NEN < 8 || sizeof(T) == 8 ? 4 : 8;
#pragma unroll
    for (int jb = 0; jb < NEN; jb += JB) {
      T2 x[JB][2];
#pragma unroll
      for (int u = 0; u < JB; ++u) {
        const int j = jb + u;
        const int p = (int)((sw[j >> 1] >> (16 * (j & 1))) & 0xFFFFu);
        x[u][0] = *reinterpret_cast<const T2*>(myrows + (size_t)(2 * p) * RB);
        x[u][1] = *reinterpret_cast<const T2*>(myrows + (size_t)(2 * p + 1) * RB);
      }
#pragma unroll
      for (int u = 0; u < JB; ++u) {
        const int j = jb + u;
        const int p = (int)((sw[j >> 1] >> (16 * (j & 1))) & 0xFFFFu);
        const T h00 = H[j][0].x, h01 = H[j][0].y, h10 = H[j][1].x, h11 = H[j][1].y;
        const T tr = h00 + h11;
        x[u][0].x += fma(mu1, tr, fma(mu1, h00, lam1 * h00));
        x[u][0].y += fma(mu1, h01, lam1 * h10);
        x[u][1].x += fma(mu1, h10, lam1 * h01);
        x[u][1].y += fma(mu1, tr, fma(mu1, h11, lam1 * h11));
        *reinterpret_cast<T2*>(myrows + (size_t)(2 * p) * RB) = x[u][0];
        *reinterpret_cast<T2*>(myrows + (size_t)(2 * p + 1) * RB) = x[u][1];
      }
    }
  }
  __syncthreads();
  // store: warp w takes slots w, w + NW, ...; lanes stride the block's row pairs (n is even
  // and a0 * 2 a multiple of 4, so every pair starts aligned)
  const int64_t row0 = (int64_t)a0 * 2;
  for (int sl = warp; sl < W; sl += NW) {
    const T2* src = reinterpret_cast<const T2*>(tile + (size_t)sl * RB);
    T2* dst = reinterpret_cast<T2*>(K + (int64_t)sl * n + row0);
    for (int r = lane; r < na; r += 32) __stcs(dst + r, src[spos[r]]);
  }
}

// ---------------------------------------------------------------------------
// Brick8.  N_j = (1 + r_j r)(1 + s_j s)(1 + t_j t) / 8 with signs r_j, s_j, t_j, so the
// gradients of an element's nodes are signed sums of a few vectors of the Gauss point
// (columns J0, J1, J2 of J^-1):
//   8 g_j = r_j J0 + s_j J1 + t_j J2 + r_j s_j (s J0 + r J1) + r_j t_j (t J0 + r J2)
//         + s_j t_j (t J1 + s J2) + r_j s_j t_j (st J0 + rt J1 + rs J2)
// Summing g_i times those instead of times every g_j needs 63 instead of 72 multiply-adds a
// point, and 15 to 27 operations instead of 72 for the vectors; the signed sums are formed
// once per element.
// A lane per node rather than two (each with half of the g_j, 14 instead of 7 warps per SM):
// the instructions halve, and the issue slots bound both (Brick8 64^3 FP32: 191 us at 48%
// issue against 303 us; the atomic element kernel takes 475 us).  FP64, 57 x 43 x 61: 293 us
// with one warp per scheduler, bound by latency; four lanes per node, 18 KB tiles and 13
// warps per SM 346 us (each line of geometry read by four lanes), two lanes 370 us, the
// atomic element kernel 373 us.
template <int NG1>
__host__ __device__ constexpr double gauss_x(int k) {
  return NG1 == 2 ? (k ? 0.57735026918962576451 : -0.57735026918962576451)
                  : (k - 1) * 0.77459666924148337704;
}

template <typename T>
__device__ __forceinline__ typename Vec2<T>::type vec2(T a, T b) {
  typename Vec2<T>::type v;
  v.x = a;
  v.y = b;
  return v;
}

// Nodes per warp: 32 in FP32 (a tile of 31 KB), 28 in FP64 (54 KB: four warps per SM, one for
// each scheduler; 32 nodes would leave three).
template <typename T>
constexpr int b8_nodes() { return sizeof(T) == 4 ? 32 : 28; }

template <typename T, int NG1>
size_t node_rows_b8_smem(int W) {
  return sizeof(T) * ((size_t)W * 3 * b8_nodes<T>() + NG1 * NG1 * NG1 * 8 * 4);
}

// A lane per node, a warp (= CTA) per NB consecutive nodes, each lane's three rows in its own
// columns of the tile [slot][3 NB] (no conflicts where the lanes' slots agree).
template <typename T, int NG1, int IL>
__global__ void __launch_bounds__(32)
k_node_rows_b8(int nnodes, int n, int W, const int32_t* __restrict__ inc_off,
               const int32_t* __restrict__ inc, const uint8_t* __restrict__ inc_loc,
               const uint16_t* __restrict__ inc_slot, const T* __restrict__ geo,
               const AsmTables* __restrict__ tab, T lam1, T mu1, T* __restrict__ K) {
  using G = Geo<GF_BRICK8, T, NG1, IL>;
  using UT = typename Unit<T>::type;
  using T2 = typename Vec2<T>::type;
  constexpr int NB = b8_nodes<T>(), RB = 3 * NB, NGP = NG1 * NG1 * NG1, LP = NG1 * NG1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* sdN = reinterpret_cast<T*>(smem_raw);   // [NGP][8][4]
  T* tile = sdN + NGP * 32;                  // [W][RB]
  const int lane = threadIdx.x;
  for (int k = lane; k < NGP * 8; k += 32) {
    const int g = k >> 3, i = k & 7;
#pragma unroll
    for (int c = 0; c < 3; ++c)
      sdN[k * 4 + c] = sizeof(T) == 4 ? T(tab->dN32[(g * 3 + c) * 8 + i]) : T(tab->dN64[(g * 3 + c) * 8 + i]);
  }
  {
    uint4* z = reinterpret_cast<uint4*>(tile);
    for (int k = lane; k < W * RB * (int)sizeof(T) / 16; k += 32) z[k] = make_uint4(0, 0, 0, 0);
  }
  __syncwarp();
  const int a0 = blockIdx.x * NB;
  const int na = min(NB, nnodes - a0);
  int q0 = 0, deg = 0;
  if (lane < na) {
    q0 = __ldg(inc_off + a0 + lane);
    deg = __ldg(inc_off + a0 + lane + 1) - q0;
  }
  T* mine = tile + 3 * lane;
  // The geometry is loaded in chunks of five units (two Gauss points in FP32, one in FP64)
  // into a ring of RC chunks: once a chunk's values are used, the chunk RC further on, of this
  // element or the next, is loaded in its place.
  constexpr int CP = 5 * G::U / 10;                  // points per chunk
  constexpr int CL = (LP + CP - 1) / CP;             // chunks per layer
  constexpr int NC = NG1 * CL;                       // chunks per element, a multiple of RC
  constexpr int RC = sizeof(T) == 4 ? (NG1 == 2 ? NC : CL) : NG1;
  UT gv[RC][5];
  const UT* ge = nullptr;                            // the element whose chunks are being loaded
  int i = 0;
  uint4 sn = make_uint4(0, 0, 0, 0);                 // neighbour slots of its nodes
  auto meta = [&](int k) {
    const int64_t q = q0 + k;
    const int e = __ldg(inc + q);
    i = __ldg(inc_loc + q);
    sn = __ldg(reinterpret_cast<const uint4*>(inc_slot + q * 8));
    ge = G::at(reinterpret_cast<const UT*>(geo), e);
  };
  auto fetch = [&](int c) {
    const int l = c / CL, m = c % CL;
#pragma unroll
    for (int u = 0; u < 5; ++u)
      if (m * 5 + u < G::LU) gv[c % RC][u] = __ldg(ge + (l * G::LU + m * 5 + u) * IL);
  };
  if (deg > 0) {
    meta(0);
#pragma unroll
    for (int c = 0; c < RC; ++c) fetch(c);
  }
  // with two points per axis |r| = |s| = |t|: their size is taken out of the sums (K1, K2)
  constexpr T K1 = NG1 == 2 ? T(gauss_x<NG1>(1)) : T(1), K2 = NG1 == 2 ? T(1.0 / 3.0) : T(1);
  const T lam = lam1 * T(0.125), mu = mu1 * T(0.125);   // the 1/8 of g_j
  for (int k = 0; k < deg; ++k) {
    const T* dn_i = sdN + 4 * i;
    const uint4 sl = sn;
    const bool more = k + 1 < deg;
    // sums of g_i times the vectors, two vectors at a time: (r, s), (rt, st), (t, rs), rst
    T2 Ha[9], Hb[9], Hc[9];
    T Hd[9];
#pragma unroll
    for (int x = 0; x < 9; ++x) {
      Ha[x] = Hb[x] = Hc[x] = vec2(T(0), T(0));
      Hd[x] = T(0);
    }
#pragma unroll
    for (int c = 0; c < NC; ++c) {
#pragma unroll
      for (int cm = 0; cm < CP; ++cm) {
        const int l = c / CL, m = c % CL * CP + cm;
        if (m >= LP) continue;
        const int g = l * LP + m;
        const T r = NG1 == 2 ? T(l ? 1 : -1) : T(gauss_x<NG1>(l));
        const T s = NG1 == 2 ? T(m / NG1 ? 1 : -1) : T(gauss_x<NG1>(m / NG1));
        const T t = NG1 == 2 ? T(m % NG1 ? 1 : -1) : T(gauss_x<NG1>(m % NG1));
        T v[10];
#pragma unroll
        for (int x = 0; x < 10; ++x) {
          T q[4];
          unit_get(gv[c % RC][(cm * 10 + x) / G::U], q);
          v[x] = q[(cm * 10 + x) % G::U];
        }
        T d[4];
        if constexpr (sizeof(T) == 4) {
          unit_get(reinterpret_cast<const UT*>(dn_i)[g * 8], d);
        } else {
          unit_get(reinterpret_cast<const UT*>(dn_i)[g * 16], d);
          d[2] = dn_i[g * 32 + 2];
        }
        T gi[3];
#pragma unroll
        for (int a = 0; a < 3; ++a)
          gi[a] = fma(v[a * 3 + 2], d[2], fma(v[a * 3 + 1], d[1], v[a * 3] * d[0])) * v[9];
#pragma unroll
        for (int b = 0; b < 3; ++b) {
          const T j0 = v[b * 3], j1 = v[b * 3 + 1], j2 = v[b * 3 + 2];
          const T2 ca = vec2(j0, j1);
          const T2 cb = vec2(fma(t, j0, r * j2), fma(t, j1, s * j2));
          const T2 cc = vec2(j2, fma(s, j0, r * j1));
          const T cd = fma(s * t, j0, fma(r * t, j1, r * s * j2));
#pragma unroll
          for (int a = 0; a < 3; ++a) {
            const T2 ga = vec2(gi[a], gi[a]);
            Ha[a * 3 + b] = fma2(ga, ca, Ha[a * 3 + b]);
            Hb[a * 3 + b] = fma2(ga, cb, Hb[a * 3 + b]);
            Hc[a * 3 + b] = fma2(ga, cc, Hc[a * 3 + b]);
            Hd[a * 3 + b] = fma(gi[a], cd, Hd[a * 3 + b]);
          }
        }
      }
      if (c + RC < NC) {
        fetch(c + RC);
      } else if (more) {
        if (c + RC == NC) meta(k + 1);
        fetch(c + RC - NC);
      }
    }
    // blocks of the nodes by their signs (t, then s, then r); V = lam P + mu P^T + mu tr(P) I
#pragma unroll
    for (int st = -1; st <= 1; st += 2) {
      T Er[9], Es[9], Ers[9];
#pragma unroll
      for (int x = 0; x < 9; ++x) {
        Er[x] = fma(st * K1, Hb[x].x, Ha[x].x);
        Es[x] = fma(st * K1, Hb[x].y, Ha[x].y);
        Ers[x] = fma(st * K2, Hd[x], K1 * Hc[x].y);
      }
#pragma unroll
      for (int ss = -1; ss <= 1; ss += 2) {
        // node j (r = +) and j + 4 (r = -)
        const int j = st < 0 ? (ss < 0 ? 0 : 1) : (ss < 0 ? 3 : 2);
        const uint32_t w0 = j & 2 ? sl.y : sl.x, w1 = j & 2 ? sl.w : sl.z;
        T* o0 = mine + ((w0 >> (16 * (j & 1))) & 0xFFFFu) * (3 * RB);
        T* o1 = mine + ((w1 >> (16 * (j & 1))) & 0xFFFFu) * (3 * RB);
        T x0[9], x1[9];
#pragma unroll
        for (int b = 0; b < 3; ++b)
#pragma unroll
          for (int a = 0; a < 3; ++a) {
            x0[a * 3 + b] = o0[b * RB + a];
            x1[a * 3 + b] = o1[b * RB + a];
          }
        T P[9], M[9];
#pragma unroll
        for (int x = 0; x < 9; ++x) {
          const T f0 = st * Hc[x].x + ss * Es[x], fr = Er[x] + ss * Ers[x];
          P[x] = f0 + fr;
          M[x] = f0 - fr;
        }
        const T tp = mu * (P[0] + P[4] + P[8]), tm = mu * (M[0] + M[4] + M[8]);
#pragma unroll
        for (int b = 0; b < 3; ++b)
#pragma unroll
          for (int a = 0; a < 3; ++a) {
            const int x = a * 3 + b, y = b * 3 + a;
            T p = fma(lam, P[x], mu * P[y]), m = fma(lam, M[x], mu * M[y]);
            if (a == b) { p += tp; m += tm; }
            o0[b * RB + a] = x0[x] + p;
            o1[b * RB + a] = x1[x] + m;
          }
      }
    }
  }
  __syncwarp();
  const int rows = na * 3;
  const int64_t row0 = (int64_t)a0 * 3;
  for (int s = 0; s < W; ++s) {
    const T* src = tile + (size_t)s * RB;
    T* dst = K + (int64_t)s * n + row0;
#pragma unroll
    for (int r = 0; r < 96; r += 32)
      if (r + lane < rows) __stcs(dst + r + lane, src[r + lane]);
  }
}

// ---------------------------------------------------------------------------
constexpr size_t kNodeSmem = 56 * 1024;

template <int ET, typename T, int NG1, int IL>
gf_status launch_geometry(gf_ctx* ctx) {
  const T* Eel = sizeof(T) == 8 ? (const T*)ctx->d_Eel : (const T*)ctx->d_Eel32;
  gf_status st = gf_geo_buffer(ctx, Geo<ET, T, NG1, IL>::bytes(ctx->nelem));
  if (st != GF_OK) return st;
  k_geometry<ET, T, NG1, IL><<<gf_blocks(ctx->nelem, kGT), kGT, 0, ctx->stream>>>(
      ctx->nelem, ctx->d_conn, ctx->d_coords64, Eel, (T*)ctx->d_geo);
  GF_LAUNCH_CHECK(ctx, "k_geometry");
  cudaEventRecord(ctx->asm_now.em, ctx->stream);
  return GF_OK;
}

template <int ET, typename T, int NG1, int IL, int NB>
gf_status launch_2d(gf_ctx* ctx, T* K, const AsmTables* d_tab) {
  const size_t sm = node_rows_2d_smem<ET, T, NG1, NB>(ctx->W);
  auto kern = k_node_rows_2d<ET, T, NG1, IL, NB>;
  GF_CUDA(ctx, gf_smem_attr(kern, sm));
  kern<<<(ctx->nnodes + NB - 1) / NB, NB, sm, ctx->stream>>>(
      ctx->nnodes, ctx->n, ctx->W, ctx->d_inc_off, ctx->d_inc, ctx->d_inc_loc, ctx->d_inc_slot,
      (const T*)ctx->d_geo, d_tab, T(ctx->lam1), T(ctx->mu1), K);
  GF_LAUNCH_CHECK(ctx, "k_node_rows_2d");
  return GF_OK;
}

// Blocks of 128 nodes while four CTAs fit an SM and every SM gets one; smaller blocks for wider
// rows (FP64 Q8: 64) and smaller meshes.
template <int ET, typename T, int NG1, int IL>
gf_status assemble_2d(gf_ctx* ctx, T* K, const AsmTables* d_tab) {
  gf_status st = launch_geometry<ET, T, NG1, IL>(ctx);
  if (st != GF_OK) return st;
  if (node_rows_2d_smem<ET, T, NG1, 128>(ctx->W) <= kNodeSmem && ctx->nnodes >= 128 * ctx->sm_count)
    return launch_2d<ET, T, NG1, IL, 128>(ctx, K, d_tab);   // four or five CTAs per SM
  if (node_rows_2d_smem<ET, T, NG1, 64>(ctx->W) <= kNodeSmem && ctx->nnodes >= 64 * ctx->sm_count)
    return launch_2d<ET, T, NG1, IL, 64>(ctx, K, d_tab);
  return launch_2d<ET, T, NG1, IL, 32>(ctx, K, d_tab);
}

template <typename T, int NG1, int IL>
gf_status assemble_b8(gf_ctx* ctx, T* K, const AsmTables* d_tab) {
  gf_status st = launch_geometry<GF_BRICK8, T, NG1, IL>(ctx);
  if (st != GF_OK) return st;
  const size_t sm = node_rows_b8_smem<T, NG1>(ctx->W);
  auto kern = k_node_rows_b8<T, NG1, IL>;
  GF_CUDA(ctx, gf_smem_attr(kern, sm));
  constexpr int NB = b8_nodes<T>();
  kern<<<(ctx->nnodes + NB - 1) / NB, 32, sm, ctx->stream>>>(
      ctx->nnodes, ctx->n, ctx->W, ctx->d_inc_off, ctx->d_inc, ctx->d_inc_loc, ctx->d_inc_slot,
      (const T*)ctx->d_geo, d_tab, T(ctx->lam1), T(ctx->mu1), K);
  GF_LAUNCH_CHECK(ctx, "k_node_rows_b8");
  return GF_OK;
}

template <typename T, int NG1, int IL>
gf_status node_dispatch(gf_ctx* ctx, T* K, const AsmTables* d_tab) {
  switch (ctx->elem_type) {
    case GF_Q4: return assemble_2d<GF_Q4, T, NG1, IL>(ctx, K, d_tab);
    case GF_Q8: return assemble_2d<GF_Q8, T, NG1, IL>(ctx, K, d_tab);
    default: return assemble_b8<T, NG1, IL>(ctx, K, d_tab);
  }
}

template <typename T>
gf_status node_assemble(gf_ctx* ctx, T* K, const AsmTables* d_tab) {
  if (ctx->scattered)
    return ctx->ngauss == 2 ? node_dispatch<T, 2, 1>(ctx, K, d_tab) : node_dispatch<T, 3, 1>(ctx, K, d_tab);
  return ctx->ngauss == 2 ? node_dispatch<T, 2, 8>(ctx, K, d_tab) : node_dispatch<T, 3, 8>(ctx, K, d_tab);
}

}  // namespace

// Geometry buffer of at least `bytes` bytes (kept across assemblies).
gf_status gf_geo_buffer(gf_ctx* ctx, size_t bytes) {
  if (ctx->geo_bytes >= bytes) return GF_OK;
  if (ctx->d_geo) cudaFree(ctx->d_geo);
  ctx->d_geo = nullptr;
  ctx->geo_bytes = 0;
  if (gf_malloc_retry(ctx, &ctx->d_geo, bytes) != cudaSuccess)
    return gf_fail(ctx, GF_ERR_OOM, "geometry buffer (%zu bytes)", bytes);
  ctx->geo_bytes = bytes;
  return GF_OK;
}

// Whether this file's kernels take the mesh: Q4, Q8 and Brick8 whose rows fit their tiles (32
// nodes; 28 in FP64 Brick8) within 112 KB, two CTAs per SM.  FP64 Brick8 meshes of less than a
// warp per SM stay with a thread per (node, element): 36 against 42 us at 8^3 (16^3: 48 and 45).
bool gf_assemble_node_fits(const gf_ctx* ctx, int dtype) {
  if (ctx->elem_type == GF_BRICK20) return false;
  if (ctx->elem_type == GF_BRICK8 && dtype == GF_F64 && ctx->nnodes <= 24 * (int64_t)ctx->sm_count)
    return false;
  const size_t es = dtype == GF_F64 ? 8 : 4;
  const size_t rows = ctx->dim == 2 ? 64 : 3 * (dtype == GF_F64 ? b8_nodes<double>() : b8_nodes<float>());
  return es * (rows * (size_t)ctx->W + 27 * 8 * 4) + 4 * 1024 <= 112 * 1024;
}

// Launches the assembly on the context's stream (no sync).
gf_status gf_assemble_node(gf_ctx* ctx, int dtype, const AsmTables* d_tab) {
  if (dtype == GF_F64) return node_assemble(ctx, ctx->d_K64, d_tab);
  return node_assemble(ctx, ctx->d_K32, d_tab);
}
