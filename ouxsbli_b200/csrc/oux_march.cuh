// Marching sweeps of 3D grids whose tile fields are all plain copies (the high-order
// viscous stencils, their node velocity gradients read from fields).
//
// Every warp is on its own: it marches along the sweep, 32 faces a chunk, one per lane.
// The cells of its stencils pass through a ring in its part of shared memory; while a
// chunk is evaluated the next chunk's cells are on their way (cp.async), so each cell is
// loaded once and no chunk waits for memory.  ME4 face positions (SHARE) and the flux of
// the face below a chunk's first cell come from the chunk before, so each position and
// each face is evaluated once.
//
// No block barrier: a face takes KEEP or, where the sensor says so, the several times
// longer SLAU reconstruction, and warps that meet at barriers wait for the slowest of
// them.  Measured on B200 at 512^3 (Hybrid-6 / ME4, FP64, ms per sweep x / y / z): tiles
// of one block with barriers 8.8 / 9.5 / 9.8; blocks of 8 warps marching a shared ring,
// three barriers a chunk, y / z 8.6 / 9.1; these 5.1-5.8 / 6.3-6.6 / 8.1 (the clock falls under
// the power cap as they get faster).  What bounds them (ncu at 184^3, x / y / z): L1 (88 / 86 /
// 65 % busy: the rings' reads and cp.async lines), instruction issue (54 / 42 / 48 %) and the FP64 pipe (45 / 38 / 40 %), with
// load latency in y (2.2 long-scoreboard stalls an issue).  Resident warps are limited by
// what the rings leave of L1: copies in flight need its lines (y 8.2 ms at 16 warps and 220 KB
// of shared memory, 6.3 at 12 and 165 KB; z 10.2 at 10 and 197 KB, 8.1 at 8 and 178 KB).
#pragma once
#include <algorithm>
#include "oux_sweep.cuh"

namespace oux {

constexpr int MARCH_WARPS = 2;  // per block; the warps do not share anything

template <bool LES> __host__ __device__ constexpr int march_fields() { return LES ? TF_COUNT : TF_COUNT - 2; }
// ring slab of a tile field (no slabs for mut and qc2 without LES)
template <bool LES> __host__ __device__ constexpr int march_slab(int field) {
  return !LES && field > TF_QC2 ? field - 2 : field;
}

// cp(field, source array) for each tile field of the sweep
template <int DIR, bool LES, class T, class CP>
__device__ __forceinline__ void march_fields_of(const StepArgs<T>& A, CP cp) {
  cp(TF_RHO, A.W.rho); cp(TF_U, A.W.u); cp(TF_V, A.W.v); cp(TF_W, A.W.w); cp(TF_P, A.W.p); cp(TF_T, A.W.T_);
  cp(TF_MU, A.W.mu);
  if constexpr (LES) { cp(TF_MUT, A.W.mut); cp(TF_QC2, A.W.qc2); }
  if (A.scheme != 0) cp(TF_SEN, A.W.sensor);
  constexpr int n = DIR, a1 = (n + 1) % 3, a2 = (n + 2) % 3;
  constexpr int ca = n == 0 ? 1 : 0, cb = n == 2 ? 1 : 2;
  cp(TF_D0, A.W.grad[3 * a1 + a1]); cp(TF_D1, A.W.grad[3 * a2 + a2]);
  cp(TF_D2, A.W.grad[3 * n + ca]); cp(TF_D3, A.W.grad[3 * n + cb]);
}

// ---- y sweep -----------------------------------------------------------------------
// A warp owns YM_C adjacent x-columns (aligned to YM_C cells, whole 32-byte sectors) of one
// plane, over a segment of the y axis; lane = (column, face), YM_R faces a chunk.
constexpr int YM_C = 8, YM_R = 4;
constexpr int YM_RING = 14;  // rows f-2 .. f+3 of a chunk's and the next one's faces (13); even: 16 (8-byte) banks
template <class T> __host__ __device__ constexpr int ym_minb() { return sizeof(T) == 8 ? 6 : 7; }

template <class T, bool LES, bool SHARE> __host__ __device__ constexpr size_t ym_warp_smem() {
  return sizeof(double) * 5 * YM_C + sizeof(T) * march_fields<LES>() * YM_RING * YM_C +
         (SHARE ? sizeof(T) * me4_terms<LES>() * (YM_R + 2) * YM_C : 0);
}

template <int ORDER, int VK, bool LES, class T, bool SHARE>
__global__ void __launch_bounds__(32 * MARCH_WARPS, ym_minb<T>()) k_march_y(StepArgs<T> A, int seg) {
  step_begin();
  constexpr int DIR = 1, R = YM_R, MC = YM_C, NR = YM_RING, FS = NR * MC, NP = (R + 2) * MC;
  extern __shared__ __align__(16) unsigned char smraw[];
  const Geo& G = A.G;
  const int lane = threadIdx.x & 31;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  unsigned char* ws = smraw + warp * ym_warp_smem<T, LES, SHARE>();
  double* Fc = reinterpret_cast<double*>(ws);           // [5][MC] fluxes of the face below the chunk
  T* ring = reinterpret_cast<T*>(Fc + 5 * MC);          // [field][NR][MC]
  T* Vs = ring + march_fields<LES>() * FS;              // [term][R + 2][MC] ME4 positions, a ring of rows
  const int cx = lane % MC, ry = lane / MC;
  const int i = (blockIdx.x * MARCH_WARPS + warp) * MC + cx;
  const bool xok = i >= G.gx && i < G.nx - G.gx;
  const int c0 = G.gy + blockIdx.y * seg, c1 = min(G.ny - G.gy, c0 + seg);  // cells of the segment
  const int k = G.sk0 + blockIdx.z;
  const int64_t col = G.at(i, 0, k);
  const int r0 = c0 - 3;  // the segment's first row; ring row of row r: (r - r0) mod NR

  auto load_row = [&](int r) {  // rows the segment does not read, and rows off the grid, are skipped
    if (!xok || r < 0 || r >= G.ny || r > c1 + 2) return;
    T* d = ring + ((unsigned)(r - r0) % NR) * MC + cx;
    const int64_t o = col + r * G.sx;
    march_fields_of<DIR, LES>(A, [&](int field, const T* src) {
      cp_async<sizeof(T)>(d + march_slab<LES>(field) * FS, src + o);
    });
  };
  // the first chunk's rows c0-3 .. c0+R+1
#pragma unroll 1
  for (int q = ry; q < R + 5; q += R) load_row(r0 + q);
  cp_async_commit();

  const double cm = xok ? A.coef * face_metric<3, DIR>(A, i, 1, k) : 0.0;
  const T inv = SHARE ? (T)A.M.inv_dy[0] : T(0);  // the spacings are all the same

  int s0 = ry;  // ring row of row f - 2
  int p0 = ry;  // SHARE: position-ring row of position f - 1
  for (int a = c0 - 1; a < c1; a += R) {  // faces a .. a+R-1; this lane's is f
    const int f = a + ry;
    const bool valid = xok && f < c1, cell = valid && f >= c0;
    cp_async_wait_all();
    __syncwarp();  // the chunk's rows have landed
    if (a + R < c1) load_row(f + R + 3);
    cp_async_commit();
    double* racc = A.Racc + col + f * G.sx;
    double ra[5] = {};  // the cell's accumulator travels while its face is evaluated
    if (cell) {
#pragma unroll
      for (int l = 0; l < 5; ++l) ra[l] = load_here(racc + l * G.vs);
    }
    int off[6];
#pragma unroll
    for (int m = 0; m < 6; ++m) off[m] = (s0 + m < NR ? s0 + m : s0 + m - NR) * MC + cx;
    auto st0 = [&](int field, int m) -> T { return ring[march_slab<LES>(field) * FS + off[m]]; };
    if constexpr (SHARE) {
      // position f + 1; the segment's first chunk also positions a - 1 and a
      auto put = [&](int row, int m0) {
        auto sp = [&](int field, int m) -> T { return st0(field, m0 + m); };
        T v[9];
        me4_position<LES>(A, sp, DIR, inv, v);
        row = (row < R + 2 ? row : row - (R + 2)) * MC + cx;
#pragma unroll
        for (int q = 0; q < me4_terms<LES>(); ++q) Vs[q * NP + row] = v[q];
      };
      if (a == c0 - 1 && ry < 2) put(p0, 0);
      put(p0 + 2, 2);
    }
    T F[5] = {};
    if (valid) {
      const int fc[3] = {i, f, k};
      face_flux<3, DIR, ORDER, VK, LES, T, false, SHARE>(A, st0, fc, F);
    }
    if constexpr (SHARE) {
      __syncwarp();  // the chunk's positions are written
      int pr[3];
#pragma unroll
      for (int m = 0; m < 3; ++m) pr[m] = (p0 + m < R + 2 ? p0 + m : p0 + m - (R + 2)) * MC + cx;
      auto P = [&](int q, int m) -> T { return Vs[q * NP + pr[m]]; };
      T vo[4];
      me4_face<LES>(A, P, DIR, inv, vo);
      F[1] = F[1] - vo[0]; F[2] = F[2] - vo[1]; F[3] = F[3] - vo[2]; F[4] = F[4] - vo[3];
    }
    double Rr[5];
#pragma unroll
    for (int l = 0; l < 5; ++l) {
      double Fl = (double)__shfl_up_sync(0xffffffffu, F[l], MC);
      if (ry == 0) Fl = Fc[l * MC + cx];
      Rr[l] = ra[l] + cm * (-Fl + (double)F[l]);
    }
    __syncwarp();  // the carried fluxes, and the positions, have been read
    if (ry == R - 1) {
#pragma unroll
      for (int l = 0; l < 5; ++l) Fc[l * MC + cx] = (double)F[l];
    }
    if (cell) {
#pragma unroll
      for (int l = 0; l < 5; ++l) racc[l * G.vs] = Rr[l];
    }
    s0 += R; s0 = s0 < NR ? s0 : s0 - NR;
    p0 += R; p0 = p0 < R + 2 ? p0 : p0 - (R + 2);
  }
}

// Warps a march has resident at `blocks` blocks per SM on the device (0: the kernel cannot
// be launched), asked once per kernel; allows the kernel its shared memory.
template <class K>
int march_slots(K kern, int warps, int blocks, size_t smem) {
  int dev = 0, sms = 0;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
      cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return 0;
  return sms * blocks * warps;
}

// The segment length (rows per warp in the x sweep) of an axis of n cells on `lines` warp
// lines, by the fewest rounds on the busiest of the resident warps; `start` rounds are
// what a warp's start costs (its ring is empty).  For a given number of waves of warps
// the most segments that fit are the best, so only those are tried.
template <class F>
int march_split(int n, int64_t slots, int64_t lines, double start, F rounds) {
  int best = n;
  double cost = ((lines + slots - 1) / slots) * (rounds(n) + start);
  for (int64_t w = 1; w <= 32; ++w) {
    const int64_t p = std::min<int64_t>(n, w * slots / lines);  // segments
    if (p < 1) continue;
    const int seg = (int)((n + p - 1) / p);
    const int64_t waves = (lines * ((n + seg - 1) / seg) + slots - 1) / slots;
    const double c = (double)waves * (rounds(seg) + start);
    if (c < cost) { cost = c; best = seg; }
    if (p == n) break;
  }
  return best;
}

template <int ORDER, int VK, bool LES, class T, bool SHARE>
int launch_march_y(const StepArgs<T>& A, cudaStream_t s) {
  auto kern = k_march_y<ORDER, VK, LES, T, SHARE>;
  constexpr size_t smem = MARCH_WARPS * ym_warp_smem<T, LES, SHARE>();
  static const int slots = march_slots(kern, MARCH_WARPS, ym_minb<T>(), smem);
  if (!slots) return 1;
  const Geo& G = A.G;
  const int Ny = G.ny - 2 * G.gy, Nz = G.sk1 - G.sk0;
  if (Nz <= 0) return 0;  // an empty part of a split stage
  const int groups = (G.nx - G.gx + YM_C - 1) / YM_C;
  const int seg = march_split(Ny, slots, (int64_t)groups * Nz, 2.0, [](int c) { return (c + YM_R) / YM_R; });
  const dim3 grid((unsigned)((groups + MARCH_WARPS - 1) / MARCH_WARPS), (unsigned)((Ny + seg - 1) / seg), (unsigned)Nz);
  return launch_step(G, kern, grid, dim3(32 * MARCH_WARPS), smem, s, A, seg) == cudaSuccess ? 0 : 1;
}

// ---- z sweep -----------------------------------------------------------------------
// A warp owns 32 adjacent x-columns of one y row, lane = column (the warps of a block take
// consecutive such lines, whatever their number in a row), and marches along z over a
// segment of cells, one face a round.  A lane's stencil, its cp.async copies, the two
// ME4 positions and the face flux before its current one are its own: no synchronisation
// at all.  Rows are 256 contiguous bytes of a plane: the y sweep's 8 columns by 4 faces a
// warp took 12.0 ms here and 16 by 2 took 10.5 (512^3, ME4, FP64; 8.1 this way), every load
// instruction touching 4 or 2 planes 2 MB apart.  Bulk copies instead of cp.async: 8.3.
constexpr int ZM_ROWS = 7;  // rows f-2 .. f+3 of the convective fields, and the next row
constexpr int ZM_CONV = 6;  // rho, u, v, w, p, T
template <bool SHARE> __host__ __device__ constexpr int zm_aux_rows() {
  return SHARE ? 5 : 7;  // rows f .. f+3 (ME4 positions) or f-2 .. f+3 (Central), and the next row
}
constexpr int ZM_OPS = 15;  // operands of a row's cell updates: Racc, Q^n, and Qs or Rs
template <class T, bool LES, bool SHARE> __host__ __device__ constexpr size_t zm_warp_smem() {
  return sizeof(double) * 32 * ZM_OPS +
         sizeof(T) * 32 * (ZM_CONV * ZM_ROWS + (march_fields<LES>() - ZM_CONV) * zm_aux_rows<SHARE>());
}
// warps per block and blocks per SM: 8 (FP64) / 16 (mixed) resident warps; more leave
// the L1 too small for the copies in flight.  The mixed Central and LES rings are larger
// (58 KB a block and more): 3 blocks, 12 warps, fit the 228 KB of an SM.
template <class T> __host__ __device__ constexpr int zm_warps() { return sizeof(T) == 8 ? 2 : 4; }
constexpr int ZM_MINB = 4;
template <class T, bool LES, bool SHARE> constexpr int zm_blocks() {
  constexpr int fit = (int)(228 * 1024 / (zm_warps<T>() * zm_warp_smem<T, LES, SHARE>() + 1024));
  return fit < ZM_MINB ? fit : ZM_MINB;
}

template <int ORDER, int VK, bool LES, class T, bool SHARE>
__global__ void __launch_bounds__(32 * zm_warps<T>(), ZM_MINB) k_march_z(StepArgs<T> A, int seg) {
  step_begin();
  constexpr int DIR = 2, NC = ZM_ROWS, NA = zm_aux_rows<SHARE>();
  constexpr bool MXC = sizeof(T) < sizeof(double);
  extern __shared__ __align__(16) unsigned char smraw[];
  const Geo& G = A.G;
  const int lane = threadIdx.x & 31;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);  // warp-uniform
  const int groups = (G.nx - 2 * G.gx + 31) / 32, line = blockIdx.x * zm_warps<T>() + warp;
  const int row = line / groups, x0 = G.gx + 32 * (line - row * groups);
  if (row >= G.ny - 2 * G.gy) return;
  unsigned char* ws = smraw + warp * zm_warp_smem<T, LES, SHARE>();
  double* ops = reinterpret_cast<double*>(ws) + lane;                       // [operand][32]
  T* conv = reinterpret_cast<T*>(ws + sizeof(double) * 32 * ZM_OPS) + lane;  // [field][NC][32]
  T* aux = conv + ZM_CONV * NC * 32;                                        // [field - 6][NA][32]
  const int i = x0 + lane, t = G.gy + row;
  const bool xok = i < G.nx - G.gx;
  const int c0 = G.sk0 + blockIdx.y * seg, c1 = min(G.sk1, c0 + seg);  // cells of the segment
  const int64_t col = G.at(i, t, 0);
  const int f0 = c0 - 1;  // the segment's first face
  const int r0 = f0 - 2;  // and first row, in slot 0 of both rings

  auto load_row = [&](int r, int slotc, int slota) {  // rows off the grid or not read are skipped
    if (!xok || r < 0 || r >= G.nz || r > c1 + 2) return;
    const int64_t o = col + r * G.plane;
    march_fields_of<DIR, LES>(A, [&](int field, const T* src) {
      T* d = field < ZM_CONV ? conv + (field * NC + slotc) * 32
                             : aux + ((march_slab<LES>(field) - ZM_CONV) * NA + slota) * 32;
      cp_async<sizeof(T)>(d, src + o);
    });
  };
  // the rows before the first prefetched one
  constexpr int PRE = SHARE ? 4 : 6;
#pragma unroll 1
  for (int m = 0; m < PRE; ++m) load_row(r0 + m, m, m);
  cp_async_commit();

  const double cm = xok ? A.coef * face_metric<3, DIR>(A, i, t, 1) : 0.0;
  const int md = A.mode;  // the z sweep is the stage's last
  const bool needQn = (!MXC && (md == CM_RK3_1 || md == CM_RK3_2 || md == CM_RK4_S)) || md == CM_RK3_3 ||
                      md == CM_RK4_4;
  const bool needQs = md == CM_RK3_2 || md == CM_RK3_3;
  const bool needRs = md == CM_RK4_S || md == CM_RK4_4;
  const T inv = SHARE ? (T)A.M.inv_dz[0] : T(0);  // the spacings are all the same

  T Fp[5] = {};                           // the flux of face f - 1
  T P0[SHARE ? me4_terms<LES>() : 1] = {}, P1[SHARE ? me4_terms<LES>() : 1] = {};  // positions f - 1 and f
  // SHARE: two rounds before the first face evaluate its positions f0 - 1 and f0.
  // sc / sa: ring slot of row f - 2 (conv) and of the first row the viscous terms read
  int sc = SHARE ? NC - 2 : 0, sa = 0;
#pragma unroll 1
  for (int f = SHARE ? f0 - 2 : f0; f < c1; ++f) {
    cp_async_wait_all();  // this lane's rows have landed
    const int64_t o = col + f * G.plane;
    const bool cell = xok && f >= c0;
    if (cell) {  // the operands of the cell's update travel while its face is evaluated
#pragma unroll
      for (int l = 0; l < 5; ++l) {
        cp_async<8>(ops + l * 32, A.Racc + o + l * G.vs);
        if (needQn) cp_async<8>(ops + (5 + l) * 32, A.Qn + o + l * G.vs);
        if (needRs) cp_async<8>(ops + (10 + l) * 32, A.Rs + o + l * G.vs);
        else if (needQs) cp_async<sizeof(T)>(ops + (10 + l) * 32, A.Qs + o + l * G.vs);
      }
    }
    cp_async_commit();
    {
      const int n = sc + 6 < NC ? sc + 6 : sc + 6 - NC;
      if (f + 1 < c1) load_row(f + 4, n, SHARE ? (sa + 4 < NA ? sa + 4 : sa + 4 - NA) : n);
      cp_async_commit();
    }
    int oc[6], oa[6];  // warp-uniform slot offsets of rows f-2+m
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      oc[m] = (sc + m < NC ? sc + m : sc + m - NC) * 32;
      if (SHARE) oa[m] = m < 2 ? 0 : (sa + m - 2 < NA ? sa + m - 2 : sa + m - 2 - NA) * 32;
      else oa[m] = oc[m];
    }
    auto st0 = [&](int field, int m) -> T {
      return field < ZM_CONV ? conv[field * NC * 32 + oc[m]]
                             : aux[(march_slab<LES>(field) - ZM_CONV) * NA * 32 + oa[m]];
    };
    T v[9];
    if constexpr (SHARE) {  // position f + 1
      auto sp = [&](int field, int m) -> T { return st0(field, 2 + m); };
      me4_position<LES>(A, sp, DIR, inv, v);
    }
    if (xok && f >= f0) {
      T F[5];
      const int fc[3] = {i, t, f};
      face_flux<3, DIR, ORDER, VK, LES, T, false, SHARE>(A, st0, fc, F);
      if constexpr (SHARE) {
        auto P = [&](int k, int m) -> T { return m == 0 ? P0[k] : m == 1 ? P1[k] : v[k]; };
        T vo[4];
        me4_face<LES>(A, P, DIR, inv, vo);
        F[1] = F[1] - vo[0]; F[2] = F[2] - vo[1]; F[3] = F[3] - vo[2]; F[4] = F[4] - vo[3];
      }
      if (cell) {
        cp_async_wait_group<1>();  // the operands; the next row may still be on its way
        double Rr[5];
#pragma unroll
        for (int l = 0; l < 5; ++l) Rr[l] = ops[l * 32] + cm * (-(double)Fp[l] + (double)F[l]);
        combine_cell<3>(
            A, i, t, f, o, Rr, [&](int l) -> double { return ops[(5 + l) * 32]; },
            [&](int l) -> T { return *reinterpret_cast<const T*>(ops + (10 + l) * 32); },
            [&](int l) -> double { return ops[(10 + l) * 32]; });
      }
#pragma unroll
      for (int l = 0; l < 5; ++l) Fp[l] = F[l];
    }
    if constexpr (SHARE) {
#pragma unroll
      for (int k = 0; k < me4_terms<LES>(); ++k) { P0[k] = P1[k]; P1[k] = v[k]; }
      sa = sa + 1 < NA ? sa + 1 : 0;
    }
    sc = sc + 1 < NC ? sc + 1 : 0;
  }
}

template <int ORDER, int VK, bool LES, class T, bool SHARE>
int launch_march_z(const StepArgs<T>& A, cudaStream_t s) {
  auto kern = k_march_z<ORDER, VK, LES, T, SHARE>;
  constexpr size_t smem = zm_warps<T>() * zm_warp_smem<T, LES, SHARE>();
  static const int slots = march_slots(kern, zm_warps<T>(), zm_blocks<T, LES, SHARE>(), smem);
  if (!slots) return 1;
  const Geo& G = A.G;
  const int Nx = G.nx - 2 * G.gx, Ny = G.ny - 2 * G.gy, Nz = G.sk1 - G.sk0;
  if (Nz <= 0) return 0;  // an empty part of a split stage
  const int groups = (Nx + 31) / 32;
  const int seg = march_split(Nz, slots, (int64_t)groups * Ny, 4.0, [](int c) { return c; });
  const dim3 grid((unsigned)(((int64_t)groups * Ny + zm_warps<T>() - 1) / zm_warps<T>()), (unsigned)((Nz + seg - 1) / seg));
  return launch_step(G, kern, grid, dim3(32 * zm_warps<T>()), smem, s, A, seg) == cudaSuccess ? 0 : 1;
}

// ---- x sweep ---------------------------------------------------------------------
// A warp marches along the rows it owns (consecutive j of one plane) as one stream, lane
// = face.  A row of Nx cells is E stream elements: its
// Nx + 1 faces (and, with shared ME4 positions, the two positions left of the first
// face), at least 32; a chunk may end one row and start the next, so no lane idles at a
// row's last face, which costs a tile of 32 cells and 33 faces a fifth warp per 4 rows.
// The ring holds XM_RING cells: a chunk's and the next one's 64 faces reach 69 cells, and
// 5 more for each of at most two row ends; its first 5 cells are repeated after its end
// so that a face's 6 cells are consecutive.
constexpr int XM_RING = 80;  // a multiple of 16 (8-byte) banks

template <class T, bool LES, bool SHARE> __host__ __device__ constexpr size_t march_x_warp_smem() {
  return (sizeof(double) * 5 * 33 + sizeof(T) * march_fields<LES>() * (XM_RING + 5) +
          (SHARE ? sizeof(T) * me4_terms<LES>() * 34 : 0) + 15) / 16 * 16;
}

template <class T> __host__ __device__ constexpr int march_x_minb() { return 8; }  // 16 resident warps

template <int ORDER, int VK, bool LES, class T, bool SHARE>
__global__ void __launch_bounds__(32 * MARCH_WARPS, march_x_minb<T>()) k_march_x(StepArgs<T> A, int nrow, int E) {
  step_begin();
  constexpr int FS = XM_RING + 5, E0 = SHARE ? 2 : 0, CX = SHARE ? 3 : 5;
  extern __shared__ __align__(16) unsigned char smraw[];
  const Geo& G = A.G;
  const int lane = threadIdx.x & 31;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int Nx = G.nx - 2 * G.gx, j1 = G.ny - G.gy;
  const int j0 = G.gy + (blockIdx.x * MARCH_WARPS + warp) * nrow;
  const int k = G.sk0 + blockIdx.y;
  if (j0 >= j1) return;
  const int rows = min(nrow, j1 - j0), total = rows * E, C = E + CX;
  unsigned char* ws = smraw + warp * march_x_warp_smem<T, LES, SHARE>();
  double* Fs = reinterpret_cast<double*>(ws);          // [5][33] the chunk's fluxes after the one before them
  T* ring = reinterpret_cast<T*>(Fs + 5 * 33);         // [field][FS]
  T* Vs = ring + march_fields<LES>() * FS;             // [term][34] positions after the two before them

  // cell `idx` of the warp's stream: cell gx - 3 + rel of its row
  auto load_cell = [&](int idx) {
    const int r = idx / C, rel = idx - r * C;
    const int ci = G.gx - 3 + rel;
    if (r >= rows || rel >= Nx + 6 || ci < 0 || ci >= G.nx) return;
    const int64_t o = G.at(ci, j0 + r, k);
    const int slot = (unsigned)idx % XM_RING;
    auto stage = [&](T* d) {
      march_fields_of<0, LES>(A, [&](int field, const T* src) {
        cp_async<sizeof(T)>(d + march_slab<LES>(field) * FS, src + o);
      });
    };
    stage(ring + slot);
    if (slot < 5) stage(ring + slot + XM_RING);
  };
  int loaded = 0;         // stream cells issued so far
  int e31 = 31, r31 = 0;  // element and row of the last lane of the chunk being loaded (E >= 32)
  auto load_chunk = [&]() {
    const int end = r31 * C + e31 - E0 + 6;
    for (int idx = loaded + lane; idx < end; idx += 32) load_cell(idx);
    loaded = end;
    cp_async_commit();
  };
  load_chunk();
  int e = lane, r = 0;
  const T inv0 = (T)A.M.inv_dx[0];
  for (int s = 0; s < total; s += 32) {
    cp_async_wait_all();
    __syncwarp();
    if (s + 32 < total) {
      e31 += 32;
      if (e31 >= E) { e31 -= E; ++r31; }
      load_chunk();
    }
    const int f = G.gx - 1 - E0 + e, j = j0 + r;
    const bool valid = r < rows && e >= E0 && f <= G.nx - G.gx - 1;
    const T* cell0 = ring + (unsigned)(r * C + e - E0 + XM_RING) % XM_RING;
    auto st0 = [&](int field, int m) -> T { return cell0[march_slab<LES>(field) * FS + m]; };
    if constexpr (SHARE) {
      auto sp = [&](int field, int m) -> T { return st0(field, 2 + m); };
      T v[9];
      me4_position<LES>(A, sp, 0, inv0, v);
#pragma unroll
      for (int q = 0; q < me4_terms<LES>(); ++q) Vs[q * 34 + lane + 2] = v[q];
    }
    T F[5] = {};
    if (valid) {
      const int fc[3] = {f, j, k};
      face_flux<3, 0, ORDER, VK, LES, T, false, SHARE>(A, st0, fc, F);
    }
    if constexpr (SHARE) {
      __syncwarp();
      auto P = [&](int q, int m) -> T { return Vs[q * 34 + lane + m]; };
      T vo[4];
      me4_face<LES>(A, P, 0, inv0, vo);
      F[1] = F[1] - vo[0]; F[2] = F[2] - vo[1]; F[3] = F[3] - vo[2]; F[4] = F[4] - vo[3];
    }
#pragma unroll
    for (int l = 0; l < 5; ++l) Fs[l * 33 + lane + 1] = (double)F[l];
    __syncwarp();
    if (valid && e > E0) {
      const int64_t o = G.at(f, j, k);
      const double cm = A.coef * face_metric<3, 0>(A, f, j, k);
#pragma unroll
      for (int l = 0; l < 5; ++l) A.Racc[o + l * G.vs] = cm * (-Fs[l * 33 + lane] + (double)F[l]);
    }
    if constexpr (SHARE) {
      if (lane >= 30) {
#pragma unroll
        for (int q = 0; q < me4_terms<LES>(); ++q) Vs[q * 34 + lane - 30] = Vs[q * 34 + lane + 2];
      }
    }
    __syncwarp();
    if (lane == 31) {
#pragma unroll
      for (int l = 0; l < 5; ++l) Fs[l * 33] = (double)F[l];
    }
    e += 32;
    if (e >= E) { e -= E; ++r; }
  }
}

template <int ORDER, int VK, bool LES, class T, bool SHARE>
int launch_march_x(const StepArgs<T>& A, cudaStream_t s) {
  auto kern = k_march_x<ORDER, VK, LES, T, SHARE>;
  constexpr size_t smem = MARCH_WARPS * march_x_warp_smem<T, LES, SHARE>();
  static const int slots = march_slots(kern, MARCH_WARPS, march_x_minb<T>(), smem);
  if (!slots) return 1;
  const Geo& G = A.G;
  const int Nx = G.nx - 2 * G.gx, Ny = G.ny - 2 * G.gy, Nz = G.sk1 - G.sk0;
  if (Nz <= 0) return 0;  // an empty part of a split stage
  const int E = std::max(Nx + 1 + (SHARE ? 2 : 0), 32);
  const int nrow = std::min(16, march_split(Ny, slots, Nz, 1.5, [&](int r) { return ((int64_t)r * E + 31) / 32; }));
  const int warps = (Ny + nrow - 1) / nrow;
  const dim3 grid((unsigned)((warps + MARCH_WARPS - 1) / MARCH_WARPS), (unsigned)Nz, 1);
  return launch_step(G, kern, grid, dim3(32 * MARCH_WARPS), smem, s, A, nrow, E) == cudaSuccess ? 0 : 1;
}

template <int DIR, int ORDER, int VK, bool LES, class T, bool SHARE>
int launch_march_dir(const StepArgs<T>& A, cudaStream_t s) {
  if constexpr (DIR == 0) return launch_march_x<ORDER, VK, LES, T, SHARE>(A, s);
  else if constexpr (DIR == 1) return launch_march_y<ORDER, VK, LES, T, SHARE>(A, s);
  else return launch_march_z<ORDER, VK, LES, T, SHARE>(A, s);
}

// Interior cells from which a direction's sweep marches; below, the tile sweeps of
// oux_sweep.cuh give more blocks.  Measured on B200 on cubes, us per sweep, march / tile:
//   FP64          64^3     72^3     96^3     128^3     176^3     192^3     256^3
//   x KEEP ME4    21 / 23  25 / 35  46 / 64  96 / 137  252 / 348 274 / 430 627 / 996
//   x Hybrid ME4  31 / 28  37 / 41  68 / 76  157 / 158 352 / 402 367 / 493 774 / 1124
//   x SLAU C6     32 / 29  37 / 42  72 / 78  162 / 163 392 / 424 404 / 515 850 / 1187
//   x Hybrid ME4, stretched axes (positions not shared)
//                 33 / 28  39 / 40  81 / 76  172 / 157 409 / 397 433 / 490 872 / 1107
//   x KEEP C6 walled in y
//                 21 / 23  26 / 35  51 / 64  104 / 131 263 / 330 283 / 407 652 / 940
//   y Hybrid ME4  34 / 31  40 / 46  76 / 81  134 / 172 298 / 446 389 / 532 863 / 1208
//   y KEEP C6     22 / 23  26 / 35  54 / 60  90 / 129  210 / 343 273 / 408 608 / 956
//   z KEEP ME4    22 / 25  32 / 39  53 / 68  116 / 148 285 / 397 329 / 473 787 / 1105
//   z Hybrid ME4  40 / 30  61 / 47  96 / 82  214 / 175 477 / 454 540 / 545 1026 / 1248
//   z SLAU ME4    39 / 32  58 / 50  93 / 86  209 / 186 496 / 492 553 / 587 1139 / 1359
//   z Hybrid C6   42 / 29  64 / 45  108 / 79 244 / 170 573 / 440 642 / 528 1330 / 1209
//   z Hybrid ME4 walled in y
//                 43 / 29  60 / 47  124 / 76 327 / 165 864 / 433 979 / 515 1384 / 1201
//   mixed         40^3     48^3     64^3     96^3      160^3     224^3     256^3
//   x Hybrid C6   13 / 13  13 / 16  23 / 21  49 / 54   172 / 218 418 / 566 526 / 834
//   x LES C6      13 / 13  13 / 16  21 / 21  44 / 58   166 / 242 418 / 647 582 / 958
//   y LES ME4     13 / 15  17 / 15  23 / 21  52 / 54   166 / 200 400 / 539 584 / 782
//   z Hybrid C6   17 / 14  21 / 16  25 / 22  60 / 56   212 / 218 548 / 560 641 / 831
//   z Hybrid ME4  17 / 15  20 / 16  27 / 23  60 / 59   228 / 228 538 / 585 758 / 870
//   z KEEP C6     13 / 12  14 / 13  17 / 18  37 / 48   146 / 188 380 / 494 523 / 747
// so the FP64 z march is for shared ME4 positions alone (the viscous rows of Central-6, and
// of walled grids, double its ring), from where it pays for SLAU faces too; FP64 x marches
// of faces that mix KEEP and SLAU stay within 10 % of the tiles either way up to 176^3.
// In x a warp takes whole rows, so a grid with few of them leaves the SMs idle whatever its
// size; MARCH_MIN_ROWS is half the resident warps, in rows as the tiles count them (they
// work on four at a time).  us per x sweep, march / tile, FP64 Hybrid-6 ME4 and KEEP-6:
// 600 rows of 1024 67 / 49 and 51 / 41, of 4096 255 / 166 and 180 / 137; 1200 of 1024
// 88 / 88 and 68 / 74, of 4096 303 / 315 and 244 / 262; 640 x 1 x 640 48 / 94 and 45 / 80.
constexpr int64_t MARCH_MIN_ROWS = 1184;
template <int DIR, class T, bool SHARE> constexpr int64_t march_min_cells() {
  constexpr bool mx = sizeof(T) < sizeof(double);
  if (DIR < 2) return mx ? 100000 : 370000;
  return mx ? 11000000 : SHARE ? 6000000 : INT64_MAX;
}

}  // namespace oux
