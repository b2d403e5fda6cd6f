// Brick20 assembly by coalesced reductions (GF_SCATTER_ATOMIC, what GF_SCATTER_AUTO takes for
// Brick20).  Same arithmetic as gf_assemble.cu (node-pair blocks lam1 g_i g_j^T +
// mu1 g_j g_i^T + mu1 (g_i . g_j) I, weighted by w detJ E); K starts from zero.
// Reference: StiffAlgo::AssembleK (src/FEM/StiffAlgo.cc:304-401).
//
// What bounds the scatter is the number of 128-byte lines that a warp's reduction touches, not
// the values: the rows of one node are only 12 bytes, so a lane per (element, node pair) pays
// a line for each pair or single value.  Here a CTA holds its consecutive elements' matrices
// in shared memory, and a warp adds one column of the same node pair for all of them at once,
// lanes (element, row): the rows of neighbouring elements' nodes lie 12 or 24 bytes apart in
// a column of the ELL, so the lanes share lines.  Now L2 takes 140-150 G sectors of reductions
// a second that miss it (1300 sectors per FP32 element; DRAM reads and writes K once), whatever
// the order of the elements; from 52^3 (FP32) that is all that is left of the time, and where the
// mesh is ordered the lines are fetched to L2 ahead of the reductions.
//   us, against a thread per node pair:    FP32  FP64
//   Brick20   8^3                    32 -> 26   35 -> 30
//   Brick20  24^3                  191 -> 160  375 -> 277
//   Brick20  48^3                1353 -> 1060  2770 -> 2490
//   Brick20  64^3                3159 -> 2959  6519 -> 6433
// A warp per element, so that only the reductions need the whole CTA; eight elements (four in
// FP64) fill 24 lanes of a reduction and two CTAs an SM.  CTAs start the reductions at
// different nodes (FP64 48^3 2474 -> 2171 us when its K was resident, nothing else).
#include <algorithm>
#include <cmath>

#include "gf_elem.cuh"

namespace {

constexpr int NEN = 20, DIM = 3, RAW = 60, GD = 12;
// Matrices in shared memory: the 12 x 12 tiles (I, J), I <= J, of the node groups of four, row
// by row, rows 6 to 11 from PO on.  The strides put the lanes that write (half tile) and the
// lanes of the reductions (element, row) on distinct banks.
// (element e's matrix starts at e * (GS + 1), its gradients 16-byte aligned at e * GS.)
constexpr int NTILE = 15, PO = 80, TS = 153, SV = NTILE * TS, GS = 2344;
__host__ __device__ constexpr int tile_of(int I, int J) { return I * 5 - I * (I - 1) / 2 + J - I; }
__host__ __device__ constexpr int row_of(int r) { return r < 6 ? r * GD : PO + (r - 6) * GD; }

// A warp per element: E elements to a CTA.
template <typename T, int NG1>
struct B20 {
  static constexpr int NGP = NG1 * NG1 * NG1;
  static constexpr int E = sizeof(T) == 4 ? 8 : 4, THREADS = 32 * E;
  static_assert(GS % 32 == 8 && GS >= NGP * RAW && GS >= SV + E, "room for both");
  static constexpr int SS = NEN * NEN;        // slots of one element
  static constexpr int N = E * NEN;           // nodes of a group
  static constexpr size_t vals = (size_t)E * GS + (size_t)RAW * NGP + NGP + (size_t)N * 4 + (size_t)E * NGP;
  // two groups' coordinates and slots, three groups' node ids and incidences
  static constexpr size_t bytes = (sizeof(T) * vals + 15) / 16 * 16 + sizeof(double) * 2 * N * DIM +
                                  sizeof(uint16_t) * 2 * E * SS + sizeof(int) * 3 * 2 * N;
};

// BYTES (4 or 8) from global to shared memory without passing registers.
template <int BYTES>
__device__ __forceinline__ void cp_async(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "n"(BYTES)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
      "mul.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}

// N values from shared memory, 16 bytes at a time.
template <int N, typename T>
__device__ __forceinline__ void lds_vec(const T* p, T (&v)[N]) {
  if constexpr (sizeof(T) == 4) {
    static_assert(N % 4 == 0, "16-byte groups");
#pragma unroll
    for (int k = 0; k < N / 4; ++k) {
      const float4 q = reinterpret_cast<const float4*>(p)[k];
      v[4 * k] = q.x; v[4 * k + 1] = q.y; v[4 * k + 2] = q.z; v[4 * k + 3] = q.w;
    }
  } else {
#pragma unroll
    for (int k = 0; k < N / 2; ++k) {
      const double2 q = reinterpret_cast<const double2*>(p)[k];
      v[2 * k] = q.x; v[2 * k + 1] = q.y;
    }
  }
}

// The same 8 bytes at a time.
template <int N>
__device__ __forceinline__ void lds_pairs(const float* p, float (&v)[N]) {
#pragma unroll
  for (int k = 0; k < N / 2; ++k) {
    const float2 q = reinterpret_cast<const float2*>(p)[k];
    v[2 * k] = q.x; v[2 * k + 1] = q.y;
  }
}

// Gradients of one Gauss point from shared memory: J, J^-1 and g_i = J^-1 dN_i, written to
// g[i * DIM + c]; returns detJ.
template <typename T, int NGP>
__device__ __forceinline__ T b20_gradients(const T* dN /* [DIM * NEN][NGP] at the point */,
                                          const T* X /* [NEN][4] */, T* g) {
  T J[3][3], Ji[3][3];
#pragma unroll
  for (int a = 0; a < DIM; ++a)
#pragma unroll
    for (int b = 0; b < DIM; ++b) J[a][b] = T(0);
#pragma unroll
  for (int i = 0; i < NEN; ++i) {
    T x[4];
    lds_vec(X + i * 4, x);
#pragma unroll
    for (int a = 0; a < DIM; ++a) {
      const T d = dN[(a * NEN + i) * NGP];
#pragma unroll
      for (int b = 0; b < DIM; ++b) J[a][b] += d * x[b];
    }
  }
  const T det = gf_det_inv<DIM, T>(J, Ji);
  constexpr int V = 16 / (int)sizeof(T);   // four nodes' gradients are whole 16-byte groups
#pragma unroll
  for (int i0 = 0; i0 < NEN; i0 += 4) {
    T out[4 * DIM];
#pragma unroll
    for (int ii = 0; ii < 4; ++ii)
#pragma unroll
      for (int c = 0; c < DIM; ++c) {
        T s = T(0);
#pragma unroll
        for (int a = 0; a < DIM; ++a) s += Ji[c][a] * dN[(a * NEN + i0 + ii) * NGP];
        out[ii * DIM + c] = s;
      }
#pragma unroll
    for (int k = 0; k < 4 * DIM / V; ++k) {
      if constexpr (sizeof(T) == 4)
        reinterpret_cast<float4*>(g + i0 * DIM)[k] =
            make_float4(out[4 * k], out[4 * k + 1], out[4 * k + 2], out[4 * k + 3]);
      else
        reinterpret_cast<double2*>(g + i0 * DIM)[k] = make_double2(out[2 * k], out[2 * k + 1]);
    }
  }
  return det;
}

// The same point of a distorted element of the FP32 path in FP64, from the mesh's own
// coordinates (rare: kept small rather than fast); returns w detJ.
__device__ __forceinline__ float b20_gradients_f64(const AsmTables* __restrict__ tab, int gp,
                                                   const double* x /* [NEN][DIM] */, float* g) {
  const double* dN = tab->dN64 + gp * DIM * NEN;
  double J[3][3], Ji[3][3];
#pragma unroll
  for (int a = 0; a < DIM; ++a)
#pragma unroll
    for (int b = 0; b < DIM; ++b) J[a][b] = 0.0;
#pragma unroll 1
  for (int i = 0; i < NEN; ++i)
#pragma unroll
    for (int a = 0; a < DIM; ++a)
#pragma unroll
      for (int b = 0; b < DIM; ++b) J[a][b] += dN[a * NEN + i] * (x[i * DIM + b] - x[b]);
  const double det = gf_det_inv<DIM, double>(J, Ji);
#pragma unroll 1
  for (int i = 0; i < NEN; ++i)
#pragma unroll
    for (int c = 0; c < DIM; ++c)
      g[i * DIM + c] = (float)(Ji[c][0] * dN[i] + Ji[c][1] * dN[NEN + i] + Ji[c][2] * dN[2 * NEN + i]);
  return (float)(tab->w64[gp] * det);
}

// ---------------------------------------------------------------------------
// einc: incidence of (element, local node), inc_slot: the slots of the element's nodes in that
// node's rows, 20 to an incidence.  What a group of E elements reads is on its way while the
// group before it is computed (node ids and incidences two groups ahead, since coordinates and
// slots are found through them).
template <typename T, int NG1>
__global__ void __launch_bounds__(B20<T, NG1>::THREADS, 2)
k_assemble_b20(int nelem, int n, const int32_t* __restrict__ conn,
               const double* __restrict__ coords, const T* __restrict__ Eel,
               const int32_t* __restrict__ einc, const uint16_t* __restrict__ inc_slot,
               const AsmTables* __restrict__ tab, T lam1, T mu1, bool ahead, T* __restrict__ K) {
  using L = B20<T, NG1>;
  constexpr int NGP = L::NGP, E = L::E, SS = L::SS, N = L::N, kBT = L::THREADS;
  constexpr bool f64 = sizeof(T) == 8;
  static_assert(NGP <= 32 && N <= kBT, "a lane per Gauss point, a thread per node");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* sG = reinterpret_cast<T*>(smem_raw);        // [E][GS] gradients, then matrices
  T* sX = sG + E * GS;                           // [E][NEN][4]
  T* sdN = sX + N * 4;                           // [RAW: a * NEN + i][NGP]
  T* sw = sdN + RAW * NGP;                       // [NGP]
  T* swd = sw + NGP;                             // [E][NGP]  w detJ E
  double* scoord = reinterpret_cast<double*>(smem_raw + (sizeof(T) * L::vals + 15) / 16 * 16);  // [2][N][3]
  uint16_t* sslots = reinterpret_cast<uint16_t*>(scoord + 2 * N * DIM);     // [2][E][SS]
  int* sconn = reinterpret_cast<int*>(sslots + 2 * E * SS);                 // [3][N]
  int* sinc = sconn + 3 * N;                                                // [3][N]

  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  for (int k = t; k < RAW * NGP; k += kBT) {
    const int g = k % NGP, r = k / NGP;
    sdN[k] = f64 ? T(tab->dN64[g * RAW + r]) : T(tab->dN32[g * RAW + r]);
  }
  for (int k = t; k < NGP; k += kBT) sw[k] = f64 ? T(tab->w64[k]) : T(tab->w32[k]);

  // this lane's half (rows 6 part .. 6 part + 5) of a tile (I, J); lanes 30 and 31 have none
  int I = 0, J = lane >> 1;
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (J >= 5) { ++I; J -= 5 - I; }
  const int part = lane & 1;
  // this lane's place in a reduction: node i + lane / (3 E), element, row
  constexpr int LPB = 3 * E, BPW = 32 / LPB;
  const int64_t n3 = (int64_t)n * 3;
  const int rb = lane / LPB, re = (lane - rb * LPB) / 3, ra = lane % 3;

  const int groups = (nelem + E - 1) / E;
  auto count = [&](int grp) { return grp < groups ? min(E, nelem - grp * E) * NEN : 0; };
  auto fetch_ids = [&](int grp, int ring) {
    if (t < count(grp)) {
      const int64_t q = (int64_t)grp * E * NEN + t;
      cp_async<4>(sconn + ring * N + t, conn + q);
      cp_async<4>(sinc + ring * N + t, einc + q);
    }
  };
  auto fetch_data = [&](int grp, int ring, int buf) {
    const int cnt = count(grp);
    for (int k = t; k < cnt * 3; k += kBT) {
      const int a = k / 3, c = k - a * 3;
      cp_async<8>(scoord + buf * N * DIM + k, coords + (int64_t)sconn[ring * N + a] * DIM + c);
    }
    for (int k = t; k < cnt * 5; k += kBT) {
      const int a = k / 5, c = k - a * 5;
      cp_async<8>(sslots + buf * E * SS + k * 4, inc_slot + (int64_t)sinc[ring * N + a] * NEN + c * 4);
    }
  };
  int ring = 0, buf = 0;
  fetch_ids(blockIdx.x, 0);
  cp_async_wait();
  __syncthreads();
  fetch_data(blockIdx.x, 0, 0);
  fetch_ids(blockIdx.x + gridDim.x, 1);
  for (int grp = blockIdx.x; grp < groups; grp += gridDim.x) {
    const int eb = grp * E;
    const int ne = min(E, nelem - eb);
    const T Ee = warp < ne ? __ldg(Eel + eb + warp) : T(0);
    cp_async_wait();
    __syncthreads();   // this group's data is there; the previous group's matrices are read
    const int* snode = sconn + ring * N;
    const uint16_t* sslot = sslots + buf * E * SS;
    const double* x = scoord + buf * N * DIM + warp * NEN * DIM;
    ring = ring == 2 ? 0 : ring + 1;
    buf ^= 1;
    fetch_data(grp + gridDim.x, ring, buf);
    fetch_ids(grp + 2 * gridDim.x, ring == 2 ? 0 : ring + 1);
    if (ahead) {
      // the lines that this group's reductions touch, to L2 during the products: lanes
      // (pair, element), one prefetch where neighbouring elements share a line
      const int e = lane % E, last = ne - 1;
      for (int pr = warp * (32 / E) + lane / E; pr < SS; pr += kBT / 32 * (32 / E)) {
        const T* q = K + (int64_t)snode[min(e, last) * NEN + pr / NEN] * DIM +
                     (int64_t)sslot[min(e, last) * SS + pr] * n3;
#pragma unroll
        for (int b = 0; b < 3; ++b) {
          const uint64_t line = (uint64_t)(q + b * (int64_t)n) / 128;
          const uint64_t end = ((uint64_t)(q + b * (int64_t)n + 3) - 1) / 128;
          const uint64_t left = __shfl_up_sync(0xffffffffu, line, 1);
          if (e == 0 || line != left) asm volatile("prefetch.global.L2 [%0];" ::"l"(line * 128));
          if (e == E - 1 && end != line) asm volatile("prefetch.global.L2 [%0];" ::"l"(end * 128));
        }
      }
    }
    if (warp < ne) {
      T* G = sG + warp * GS;
      T* X = sX + warp * NEN * 4;
      T* wd = swd + warp * NGP;
      if (lane < NEN) {
#pragma unroll
        for (int c = 0; c < DIM; ++c) X[lane * 4 + c] = T(x[lane * 3 + c] - x[c]);
      }
      __syncwarp();
      T det = T(0);
      if (lane < NGP) det = b20_gradients<T, NGP>(sdN + lane, X, G + lane * RAW);
      T w = lane < NGP ? sw[lane] * det : T(0);
      if constexpr (!f64) {
        // an element whose max/min |detJ| over the Gauss points exceeds 10 is redone in FP64
        float dmin = lane < NGP ? fabsf((float)det) : 3.4e38f, dmax = lane < NGP ? dmin : 0.f;
#pragma unroll
        for (int o = 16; o; o >>= 1) {
          dmin = fminf(dmin, __shfl_xor_sync(0xffffffffu, dmin, o));
          dmax = fmaxf(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
        }
        if (dmax > 10.f * dmin && lane < NGP)
          w = b20_gradients_f64(tab, lane, x, reinterpret_cast<float*>(G + lane * RAW));
      }
      if (lane < NGP) wd[lane] = w * Ee;
      __syncwarp();

      // products: H = sum_gp (w detJ E) g_i g_j^T of this lane's 6 rows and 12 columns
      T H[6][GD];
      const T* gI = G + (I * 4 + part * 2) * DIM;
      const T* gJ = G + J * GD;
      if (lane < 2 * NTILE) {
        if constexpr (!f64) {
          // two neighbouring columns per packed FMA
          float2 h[6][GD / 2];
#pragma unroll
          for (int r = 0; r < 6; ++r)
#pragma unroll
            for (int p = 0; p < GD / 2; ++p) h[r][p] = make_float2(0.f, 0.f);
#pragma unroll 1
          for (int g = 0; g < NGP; ++g) {
            T gi[6], gj[GD];
            lds_vec(gJ + g * RAW, gj);
            lds_pairs(gI + g * RAW, gi);
            const float2 ww = make_float2(wd[g], wd[g]);
            float2 c[GD / 2];
#pragma unroll
            for (int p = 0; p < GD / 2; ++p) c[p] = mul2(make_float2(gj[2 * p], gj[2 * p + 1]), ww);
#pragma unroll
            for (int r = 0; r < 6; ++r)
#pragma unroll
              for (int p = 0; p < GD / 2; ++p) h[r][p] = fma2(make_float2(gi[r], gi[r]), c[p], h[r][p]);
          }
#pragma unroll
          for (int r = 0; r < 6; ++r)
#pragma unroll
            for (int p = 0; p < GD / 2; ++p) {
              H[r][2 * p] = h[r][p].x;
              H[r][2 * p + 1] = h[r][p].y;
            }
        } else {
#pragma unroll
          for (int r = 0; r < 6; ++r)
#pragma unroll
            for (int c = 0; c < GD; ++c) H[r][c] = T(0);
#pragma unroll 1
          for (int g = 0; g < NGP; ++g) {
            T gi[6], gj[GD];
            lds_vec(gI + g * RAW, gi);
            lds_vec(gJ + g * RAW, gj);
            const T ww = wd[g];
#pragma unroll
            for (int r = 0; r < 6; ++r) {
              const T y = gi[r] * ww;
#pragma unroll
              for (int c = 0; c < GD; ++c) H[r][c] += y * gj[c];
            }
          }
        }
      }
      __syncwarp();   // the gradients are read: the matrix takes their place
      if (lane < 2 * NTILE) {
        T* out = G + warp + (lane >> 1) * TS + part * PO;
#pragma unroll
        for (int ii = 0; ii < 2; ++ii)
#pragma unroll
          for (int jj = 0; jj < 4; ++jj) {
            T tr = T(0);
#pragma unroll
            for (int a = 0; a < DIM; ++a) tr += H[ii * DIM + a][jj * DIM + a];
#pragma unroll
            for (int a = 0; a < DIM; ++a)
#pragma unroll
              for (int b = 0; b < DIM; ++b) {
                T v = lam1 * H[ii * DIM + a][jj * DIM + b] + mu1 * H[ii * DIM + b][jj * DIM + a];
                if (a == b) v += mu1 * tr;
                out[(ii * DIM + a) * GD + jj * DIM + b] = v;
              }
          }
      }
    }
    __syncthreads();

    // reductions: a warp takes node i of its elements and the columns of every node j
    if (rb < BPW && re < ne) {
      const uint16_t* slots = sslot + re * SS;
      for (int ii = warp * BPW + rb; ii < NEN; ii += kBT / 32 * BPW) {
        const int i = (ii + blockIdx.x * 7) % NEN;
        const int ig = i >> 2, ir = (i & 3) * DIM + ra, irow = row_of(ir);
        T* row = K + (int64_t)snode[re * NEN + i] * DIM + ra;
#pragma unroll
        for (int jg = 0; jg < 5; ++jg) {
          // rows of a stored tile (ig <= jg), or its columns
          const bool up = ig <= jg;
          const T* v = sG + re * (GS + 1) + (up ? tile_of(ig, jg) * TS + irow : tile_of(jg, ig) * TS + ir);
          T x[GD];
          if (up) {
#pragma unroll
            for (int c = 0; c < GD; ++c) x[c] = v[c];
          } else {
#pragma unroll
            for (int c = 0; c < GD; ++c) x[c] = v[row_of(c)];
          }
#pragma unroll
          for (int jj = 0; jj < 4; ++jj) {
            T* dst = row + (int64_t)slots[i * NEN + jg * 4 + jj] * n3;
            atomicAdd(dst, x[jj * 3]);
            atomicAdd(dst + n, x[jj * 3 + 1]);
            atomicAdd(dst + n + n, x[jj * 3 + 2]);
          }
        }
      }
    }
  }
}

template <typename T, int NG1>
gf_status launch_b20(gf_ctx* ctx, const AsmTables* d_tab, T* K) {
  using L = B20<T, NG1>;
  auto kern = k_assemble_b20<T, NG1>;
  GF_CUDA(ctx, gf_smem_attr(kern, L::bytes));
  const T* Eel = sizeof(T) == 8 ? (const T*)ctx->d_Eel : (const T*)ctx->d_Eel32;
  const int groups = (ctx->nelem + L::E - 1) / L::E;
  // Lines fetched ahead on large matrices of ordered meshes.  Us with and without, FP32: 44^3 (1.0
  // GB of K) 926, 952; 48^3 1197, 1113; 50^3 (1.5 GB) 1349, 1376; 52^3 1519, 1651; 64^3 3088, 3320;
  // FP64: 28^3 446, 433; 32^3 642, 618; 38^3 (1.4 GB) 1052, 1191; 44^3 1915, 1990; 60^3 5137, 5288;
  // 64^3 6573, 6552.  What a prefetch brings is a line; where the rows of consecutive elements'
  // nodes do not fill the lines in order, most of it is fetched for nothing, and twice: FP32 56^3
  // with the nodes shuffled in runs of 128, 16, 1 3128, 7372, 13869 against 2544, 4303, 9451, rows
  // of 8 elements (8 x 8 x 3200) 2964 against 2412, of 16 2521 against 2451, of 52 1819 against 2047.
  const int64_t kbytes = (int64_t)ctx->n * ctx->W * (int64_t)sizeof(T);
  const bool ahead = ctx->consecutive && kbytes > 1500000000;
  // CTAs that stay for several groups drift apart, and with them the elements in flight, whose lines
  // L2 has to hold at once.  An ordered mesh's are few, and the loads ahead pay: FP32 28^3 249 us,
  // 263 with a CTA per group, 40^3 702, 665, 56^3 1932, 1976; FP64 36^3 932, 1085.  Shuffled in runs
  // of 16 nodes: FP32 28^3 351, 344; 32^3 582, 486; 36^3 941, 739; 56^3 4325, 3016 (N = 1: 36^3 2107,
  // 1850; elements in runs of 16: 651, 690); FP64 36^3 1392, 1377.
  const bool stay = sizeof(T) == 8 || !ctx->shuffled || kbytes <= 300000000;
  kern<<<stay ? std::min(groups, ctx->sm_count * 2) : groups, L::THREADS, L::bytes, ctx->stream>>>(
      ctx->nelem, ctx->n, ctx->d_conn, ctx->d_coords64, Eel, ctx->d_einc, ctx->d_inc_slot, d_tab,
      T(ctx->lam1), T(ctx->mu1), ahead, K);
  GF_LAUNCH_CHECK(ctx, "k_assemble_b20");
  return GF_OK;
}

}  // namespace

// Adds every Brick20 element matrix into K (zero on entry) on the context's stream (no sync).
gf_status gf_assemble_b20(gf_ctx* ctx, int dtype, const AsmTables* d_tab) {
  if (dtype == GF_F64)
    return ctx->ngauss == 2 ? launch_b20<double, 2>(ctx, d_tab, ctx->d_K64)
                            : launch_b20<double, 3>(ctx, d_tab, ctx->d_K64);
  return ctx->ngauss == 2 ? launch_b20<float, 2>(ctx, d_tab, ctx->d_K32)
                          : launch_b20<float, 3>(ctx, d_tab, ctx->d_K32);
}
