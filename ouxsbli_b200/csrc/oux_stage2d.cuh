// One Runge-Kutta stage of a 2D inviscid solve in one kernel: primitives and sensor of a
// tile and its halo, the x and y face fluxes, the stage combination, and the ghost /
// boundary cells of the cells it writes.
//
// Measured on B200 (us, separate passes -> this): 513 x 7 shock tube, SLAU-6 RK3, ten steps
// 1085 -> 382; 252^2 vortex, KEEP-6 RK4, ten steps 901 -> 334; 64 vortices of 64^2 to 512^2 in one
// batched step 2115 -> 968 (FP64) and 1599 -> 966 (mixed).  What bounds it: load latency and
// barriers at small grids; on large ones L1 (73 % busy in FP64, 63 % mixed, at 2048^2) and
// latency that the two other resident blocks have to hide (2.6 long-scoreboard and 1.4
// barrier stalls an issue; the combination's operands are fetched during the fluxes: without
// that the batched step took 2883).
//
// A 2D stage as separate passes (primitives, sensor, two sweeps, ghost fill) is bound by
// launches on the grids 2D cases have: five kernels of 5 to 10 us each whatever the size
// up to 250^2, and on larger ones by the primitive fields and flux differences it sends
// through memory between the passes.  Here a stage reads its source and writes its
// result.  A block owns 32 x 8 cells and decodes them with a halo of order / 2 cells (1.5
// to 2.1x the cells, from L2); 288 threads own its 33 x 8 x faces, then its 32 x 9 y faces.
//
// The source is read with a halo, so a stage never writes the array it reads: the stage
// states alternate between two buffers (run_fused_2d in oux_api.cu).
#pragma once
#include "oux_sweep.cuh"

namespace oux {

template <int N> struct IntC { static constexpr int value = N; };

constexpr int S2_TX = 32, S2_TY = 8, S2_THREADS = S2_TX * (S2_TY + 1);

// halo of the decoded tile: the face stencils', and two cells for the sensor of the cells
// next to the tile
template <int ORDER, bool KONLY> __host__ __device__ constexpr int s2_halo() {
  return !KONLY && ORDER == 2 ? 2 : ORDER / 2;
}
template <int ORDER, bool KONLY> __host__ __device__ constexpr int s2_cells() {
  return (S2_TX + 2 * s2_halo<ORDER, KONLY>()) * (S2_TY + 2 * s2_halo<ORDER, KONLY>());
}
// tile fields: rho, u, v, p, T [, sensor, and in the mixed form the FP64 u, v it is formed from]
template <int ORDER, bool KONLY, class T> __host__ __device__ constexpr size_t stage2d_smem() {
  return sizeof(double) * (4 * ((S2_TX + 1) * S2_TY + S2_TX * (S2_TY + 1)) + 8 * S2_TX * S2_TY) +
         (!KONLY && sizeof(T) < sizeof(double) ? sizeof(double) * 2 * s2_cells<ORDER, KONLY>() : 0) +
         sizeof(T) * (KONLY ? 5 : 6) * s2_cells<ORDER, KONLY>();
}

// src: the stage's source, FP64 form: the full state; mixed form: the FP32 increment over
// A.Qn (null: none).  dst: the array the stage writes (FP64: a full state; mixed: an
// increment, or the full FP64 state in the last stage).  keep (mixed form, first stage):
// a copy of Q^n the later stages read, so that the last one can write the state in place.
template <int ORDER, bool KONLY, class T>
__global__ void __launch_bounds__(S2_THREADS, KONLY ? 3 : 2)
k_stage2d(StepArgs<T> A, const void* src, void* dst, double* keep) {
  step_begin();
  constexpr bool MX = sizeof(T) < sizeof(double);
  constexpr int H = s2_halo<ORDER, KONLY>(), LX = S2_TX + 2 * H, LY = S2_TY + 2 * H, NC = LX * LY;
  constexpr int NFX = (S2_TX + 1) * S2_TY, NFY = S2_TX * (S2_TY + 1);
  extern __shared__ __align__(16) unsigned char smraw[];
  double* Fx = reinterpret_cast<double*>(smraw);  // [4][S2_TY][S2_TX + 1]
  double* Fy = Fx + 4 * NFX;                      // [4][S2_TY + 1][S2_TX]
  double* ops = Fy + 4 * NFY;                     // [8][cell] operands of the combination
  double* vel = ops + 8 * S2_TX * S2_TY;          // mixed form with a sensor: FP64 u, v
  T* tile = reinterpret_cast<T*>(vel + (!KONLY && MX ? 2 * NC : 0));  // [field][LY][LX]
  const Geo& G = A.G;
  const int tid = threadIdx.x;
  const int bx = G.gx + S2_TX * blockIdx.x, by = G.gy + S2_TY * blockIdx.y;
  const int ex = G.nx - G.gx, ey = G.ny - G.gy;  // ends of the interior
  const double* Sd = reinterpret_cast<const double*>(src);
  const float* Sf = reinterpret_cast<const float*>(src);

  // the combination's operands (Q^n, and the source's own value or Rs) travel while the
  // fluxes are evaluated
  const int tx = tid % S2_TX, ty = tid / S2_TX;
  const bool own = ty < S2_TY && bx + tx < ex && by + ty < ey;
  const bool needS = A.mode == CM_RK3_2 || A.mode == CM_RK3_3, rk4 = A.mode == CM_RK4_S || A.mode == CM_RK4_4;
  if (own) {
    const int64_t o = G.at(bx + tx, by + ty, 0);
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      const int64_t q = o + l * G.vs;
      cp_async<8>(ops + l * S2_TX * S2_TY + tid, A.Qn + q);
      double* d = ops + (4 + l) * S2_TX * S2_TY + tid;
      if (rk4) cp_async<8>(d, A.Rs + q);
      else if (needS) cp_async<sizeof(T)>(d, reinterpret_cast<const T*>(src) + q);
    }
  }
  cp_async_commit();

  // ---- primitives of the tile and its halo (prim_cell / prim_mx_cell); a thread's loads
  // all go out before its first store ----
  constexpr int ND = (NC + S2_THREADS - 1) / S2_THREADS;  // cells a thread decodes
  double q[ND][4], Jv[ND];
  bool in[ND];
#pragma unroll
  for (int n = 0; n < ND; ++n) {
    const int c = tid + n * S2_THREADS;
    const int i = bx - H + c % LX, j = by - H + c / LX;
    in[n] = c < NC && i >= 0 && i < min(G.nx, ex + H) && j >= 0 && j < min(G.ny, ey + H);
    if (!in[n]) continue;
    const int64_t o = G.at(i, j, 0);
    Jv[n] = A.M.jac[(int64_t)j * G.nx + i];
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      if constexpr (MX) q[n][l] = A.Qn[o + l * G.vs] + (Sf ? (double)Sf[o + l * G.vs] : 0.0);
      else q[n][l] = Sd[o + l * G.vs];
    }
  }
#pragma unroll
  for (int n = 0; n < ND; ++n) {
    if (!in[n]) continue;
    const int c = tid + n * S2_THREADS;
    double v[3], rho, p, temp;
    prim_decode<2>(q[n], Jv[n], A.K, rho, v, p, temp);
    tile[c] = (T)rho;
    tile[NC + c] = (T)v[0];
    tile[2 * NC + c] = (T)v[1];
    tile[3 * NC + c] = MX ? (T)(p - A.K.p_ref) : (T)p;
    tile[4 * NC + c] = MX ? (T)(temp - A.K.T_ref) : (T)temp;
    if constexpr (!KONLY && MX) { vel[c] = v[0]; vel[NC + c] = v[1]; }
  }
  __syncthreads();

  // ---- Ducros sensor of the tile and a one-cell ring; cells of the outermost layer take
  // their inner neighbour's (the copies of calc_Ducros) ----
  if constexpr (!KONLY) {
    const double* U = vel;
    if constexpr (!MX) U = tile + NC;
    for (int c = tid; c < (S2_TX + 2) * (S2_TY + 2); c += S2_THREADS) {
      const int i = bx - 1 + c % (S2_TX + 2), j = by - 1 + c / (S2_TX + 2);
      if (i > ex || j > ey) continue;
      const int ci = min(max(i, 1), G.nx - 2), cj = min(max(j, 1), G.ny - 2);
      const int o = (cj - by + H) * LX + ci - bx + H;
      const double dxt = ducros_scale<double>(A.M.inv_dx, ci), dyt = ducros_scale<double>(A.M.inv_dy, cj);
      const double dudx = (-U[o - 1] + U[o + 1]) * dxt, dvdx = (-U[NC + o - 1] + U[NC + o + 1]) * dxt;
      const double dudy = (-U[o - LX] + U[o + LX]) * dyt, dvdy = (-U[NC + o - LX] + U[NC + o + LX]) * dyt;
      tile[5 * NC + (j - by + H) * LX + i - bx + H] =
          (T)ducros_value<2, double>(dudx + dvdy, 0.0, 0.0, dvdx - dudy);
    }
    __syncthreads();
  }

  // ---- x faces, then y faces ----
  // cell f - 2 + m of a face's stencil lies `m - 2` cells from its left cell at base
  auto face = [&](auto dir, int fi, int fj, double* out, int stride) {
    constexpr int D = decltype(dir)::value;
    const int base = (fj - by + H) * LX + fi - bx + H;
    auto st0 = [&](int field, int m) -> T {
      constexpr int step = D == 0 ? 1 : LX;
      if (field == TF_W) return T(0);
      const int slab = field <= TF_V ? field : field == TF_P ? 3 : field == TF_T ? 4 : 5;
      return tile[slab * NC + base + (m - 2) * step];
    };
    const int fc[3] = {fi, fj, 0};
    T F[5];
    face_flux<2, D, ORDER, VK_EULER, false, T, KONLY, false>(A, st0, fc, F);
    out[0] = (double)F[0];
    out[stride] = (double)F[1];
    out[2 * stride] = (double)F[2];
    out[3 * stride] = (double)F[4];
  };
  if (tid < NFX) {
    const int fi = bx - 1 + tid % (S2_TX + 1), fj = by + tid / (S2_TX + 1);
    if (fi < ex && fj < ey) face(IntC<0>{}, fi, fj, Fx + tid, NFX);
  }
  {
    const int fi = bx + tid % S2_TX, fj = by - 1 + tid / S2_TX;
    if (fi < ex && fj < ey) face(IntC<1>{}, fi, fj, Fy + tid, NFY);
  }
  __syncthreads();

  // ---- cells ----
  if (!own) return;
  cp_async_wait_all();
  const int i = bx + tx, j = by + ty;
  const int64_t o = G.at(i, j, 0);
  const double cx = A.coef * face_metric<2, 0>(A, i, j, 0), cy = A.coef * face_metric<2, 1>(A, i, j, 0);
  const double* fx = Fx + ty * (S2_TX + 1) + tx;
  const double* fy = Fy + ty * S2_TX + tx;
  const bool full = !MX || A.mode == CM_RK3_3 || A.mode == CM_RK4_4;  // dst holds a full state
  double* Dd = reinterpret_cast<double*>(dst);
  float* Df = reinterpret_cast<float*>(dst);
  double w[5];  // the cell's new full state
  float wf[4];  // its increment (mixed form, not the last stage)
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    const int64_t q = o + l * G.vs;
    const double dE = cx * (-fx[l * NFX] + fx[l * NFX + 1]);
    const double R = dE + cy * (-fy[l * NFY] + fy[l * NFY + S2_TX]);
    const double qn = ops[l * S2_TX * S2_TY + tid];
    const double* op = ops + (4 + l) * S2_TX * S2_TY + tid;
    const double s = needS ? (double)*reinterpret_cast<const T*>(op) : 0.0, rs = rk4 ? *op : 0.0;
    if (MX && keep) keep[q] = qn;
    switch (A.mode) {
      case CM_RK3_1:
        if constexpr (MX) wf[l] = (T)(-R);
        else w[l] = qn - R;
        break;
      case CM_RK3_2:
        if constexpr (MX) wf[l] = (T)((A.c2 * s - R) * A.c4);  // c1 + c2 = 1
        else w[l] = (A.c1 * qn + A.c2 * s - R) * A.c4;
        break;
      case CM_RK3_3:
        if constexpr (MX) w[l] = qn + (A.c1 * s - R) * A.c4;  // (c1 + c2) c4 = 1
        else w[l] = (A.c1 * s + A.c2 * qn - R) * A.c4;
        break;
      case CM_RK4_S:
        if constexpr (MX) wf[l] = (T)(-A.c1 * R);
        else w[l] = qn - A.c1 * R;
        A.Rs[q] = rs + A.c2 * R;
        break;
      default: {  // CM_RK4_4
        const double r = rs + R;
        w[l] = qn - r * (1.0 / 6.0);
        A.Rs[q] = 0.0;
      }
    }
    if (full) {
      Dd[q] = w[l];
    } else {
      Df[q] = wf[l];
      w[l] = qn + (double)wf[l];
    }
  }

  // ---- the ghost / boundary cells this cell is the source of (ghost_cell's rules) ----
  // per axis, the indices this cell is the source of: every index a multiple of the period
  // away (periodic), or the boundary cell beside it; `from`, `to` and `step` enumerate them
  struct Range { int from, to, step; };
  auto sources = [](int c, int n, int gw, bool wall) -> Range {
    const int N = n - 2 * gw;
    if (wall) return {c == 1 ? 0 : c, c == n - 2 ? n - 1 : c, 1};
    return {c - c / N * N, n - 1, N};
  };
  const Range ri = sources(i, G.nx, G.gx, G.bcx), rj = sources(j, G.ny, G.gy, G.bcy);
  if (ri.from == i && i + ri.step > ri.to && rj.from == j && j + rj.step > rj.to) return;
  for (int gj = rj.from; gj <= rj.to; gj += rj.step)
    for (int gi = ri.from; gi <= ri.to; gi += ri.step) {
      if (gi == i && gj == j) continue;
      const int64_t p = G.at(gi, gj, 0);
      const bool bnd = (G.bcx && gi != i) || (G.bcy && gj != j);
      double v[5] = {w[0], w[1], w[2], w[3], 0.0};
      if (bnd) bc_2d(G, 4, v, gi, gj, i, j);
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        const int64_t q = p + l * G.vs;
        if (MX && keep) keep[q] = A.Qn[q];
        if (full) Dd[q] = v[l];
        else Df[q] = bnd ? (float)(v[l] - A.Qn[q]) : wf[l];
      }
    }
}

template <int ORDER, bool KONLY, class T>
int launch_stage2d(const StepArgs<T>& A, const void* src, void* dst, double* keep, cudaStream_t s) {
  auto kern = k_stage2d<ORDER, KONLY, T>;
  constexpr size_t smem = stage2d_smem<ORDER, KONLY, T>();
  static const cudaError_t attr = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (attr != cudaSuccess) return 1;
  const Geo& G = A.G;
  const dim3 grid((unsigned)((G.nx - 2 * G.gx + S2_TX - 1) / S2_TX), (unsigned)((G.ny - 2 * G.gy + S2_TY - 1) / S2_TY));
  return launch_step(G, kern, grid, dim3(S2_THREADS), smem, s, A, src, dst, keep) == cudaSuccess ? 0 : 1;
}

template <class T>
int launch_stage2d_any(int order, const StepArgs<T>& A, const void* src, void* dst, double* keep, cudaStream_t s) {
  const bool konly = A.scheme == 0;
  if (order == 6) return konly ? launch_stage2d<6, true, T>(A, src, dst, keep, s) : launch_stage2d<6, false, T>(A, src, dst, keep, s);
  if (order == 4) return konly ? launch_stage2d<4, true, T>(A, src, dst, keep, s) : launch_stage2d<4, false, T>(A, src, dst, keep, s);
  return konly ? launch_stage2d<2, true, T>(A, src, dst, keep, s) : launch_stage2d<2, false, T>(A, src, dst, keep, s);
}

}  // namespace oux
