// Batched BiCGSTAB: many independent systems (the diagonal blocks of one
// block-diagonal matrix) times R right-hand sides each, solved together.
//
// Every (system, right-hand side) pair runs the recurrences of
// cublas2_pbicgstabv2 (include/bicgstab/bicgstab_solver.h:33-275) with its own
// rho, alpha, omega, beta and stop test; pairs that converge are frozen (x no
// longer changes) while the others continue.  Layout: A and M in SELL-32 over
// all N rows; vectors row-major N x R.  R threads share a row, one per
// right-hand side, so every matrix entry read from HBM serves R products (a
// warp broadcast) and a gathered column is R contiguous doubles read by R
// neighbouring lanes.  Thread blocks are tiles of 256 rows inside one
// system; each dot product leaves one partial per tile and the last tile of a
// system to finish sums that system's partials in tile order (deterministic)
// and updates the system's scalars.
#include <algorithm>
#include <climits>
#include <cmath>

#include "internal.cuh"

namespace dcu {
namespace {

constexpr int BT = 256;           // rows per tile (= threads per block)
constexpr int BT_WARPS = BT / 32;
constexpr int BCHUNK = 8;         // iterations per graph launch

struct BState {                   // per (system, rhs) pair, length S * R
  double* rho;
  double* alpha;
  double* omega;
  double* beta;
  double* res;
  double* thr;
  double* bnorm;
  int* active;                    // 1 while iterating
  int* sys_live;                  // per system: pairs still iterating
  int* conv_it;                   // iteration counter when it stopped
  int* status;                    // dcu_solve_status
};

struct BGlobal {
  int it;                         // the reference's counter, shared by all pairs
  int done;
  int active_count;
  int systems_done;               // systems finished in the current kernel
  int pidx;
  int maxiter;
  int pad[2];
};

template <int R>
struct BArgs {
  int n, nsys, ntiles;
  const int* sys_off;             // [nsys + 1]
  const int* tile_sys;            // [ntiles]
  const int* tile_row0;           // [ntiles]
  const int* tile_off;            // [nsys + 1] first tile of each system
  const long long* off;
  const int* kd;                  // per (slice, k) offset descriptors
  const int* su;                  // per slice: all of its k uniform
  const int* ix;
  const double* aval;
  const double* mval;
  const double* b;
  double* x;
  double* r;
  double* rs;
  double* p0;
  double* p1;
  double* y;
  double* ay;
  double* s;
  double* z;
  double* az;
  double* part;                   // [ntiles][3][R]
  unsigned* cnt;                  // [nsys] tiles finished, per kernel
  BState st;
  BGlobal* g;
};

// out[q] = sum_k val * X[col][q], q < R, X row-major with R columns.
// V right-hand sides per thread: 2 (one 16-byte load per gathered column)
// when R >= 2, else 1.
template <int R>
__host__ __device__ constexpr int vals_per_thread() {
  return R >= 2 ? 2 : 1;
}

template <int V>
__device__ __forceinline__ void ldv(const double* __restrict__ p, double (&o)[V]) {
  if constexpr (V == 2) {
    const double2 t = __ldg(reinterpret_cast<const double2*>(p));
    o[0] = t.x;
    o[1] = t.y;
  } else {
    o[0] = __ldg(p);
  }
}
template <int V>
__device__ __forceinline__ void ldp(const double* p, double (&o)[V]) {  // plain load (data written this launch)
  if constexpr (V == 2) {
    const double2 t = *reinterpret_cast<const double2*>(p);
    o[0] = t.x;
    o[1] = t.y;
  } else {
    o[0] = *p;
  }
}
template <int V>
__device__ __forceinline__ void stv(double* p, const double (&o)[V]) {
  if constexpr (V == 2) *reinterpret_cast<double2*>(p) = make_double2(o[0], o[1]);
  else *p = o[0];
}

// One SELL-32 row for V right-hand sides: acc[e] = sum_k val[q] * xf(col[q])[e].
// A slice whose every k has one column offset (su, kd: SellPlan) forms its
// columns from the row and reads no index.
template <int V, typename F>
__device__ __forceinline__ void sell_row_v(const long long* __restrict__ off, const int* __restrict__ kd,
                                           const int* __restrict__ su, const double* __restrict__ val,
                                           const int* __restrict__ ix, int row, F xf, double (&acc)[V]) {
  const int sl = row >> 5;
  const long long o0 = __ldg(off + sl), o1 = __ldg(off + sl + 1);
  const long long base = o0 + (row & 31);
  const int w = (int)((o1 - o0) >> 5);
#pragma unroll
  for (int e = 0; e < V; ++e) acc[e] = 0.0;
  auto step = [&](const double (&av)[8], const int (&cv)[8], int k0) {
#pragma unroll
    for (int t = 0; t < 8; ++t)
      if (k0 + t < w) {
        double xv[V];
        xf(cv[t], xv);
#pragma unroll
        for (int e = 0; e < V; ++e) acc[e] += av[t] * xv[e];
      }
  };
  if (__ldg(su + sl) & 1) {
    const int* __restrict__ kp = kd + (o0 >> 5);
    for (int k0 = 0; k0 < w; k0 += 8) {
      double av[8];
      int cv[8];
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        av[t] = (k0 + t < w) ? __ldcs(val + base + 32ll * (k0 + t)) : 0.0;
        cv[t] = (k0 + t < w) ? row + (__ldg(kp + k0 + t) >> 1) : row;
      }
      step(av, cv, k0);
    }
    return;
  }
  for (int k0 = 0; k0 < w; k0 += 8) {
    double av[8];
    int cv[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const long long q = base + 32ll * (k0 + t);
      av[t] = (k0 + t < w) ? __ldcs(val + q) : 0.0;
      cv[t] = (k0 + t < w) ? __ldcs(ix + q) : row;
    }
    step(av, cv, k0);
  }
}

// Thread layout: a block covers one tile of BT rows of one system.  T = R / V
// threads share a row; thread t owns right-hand sides q0 .. q0 + V - 1 with
// q0 = (t % T) * V and takes the tile's rows in T passes of BT / T
// consecutive rows (row = row0 + pass * BT / T + t / T).  A warp reads 32 x V
// consecutive doubles of each row-major N x R vector and gathers 32 / T
// neighbouring rows x R right-hand sides (contiguous) per column offset.
template <int R>
struct TileRows {
  static constexpr int V = vals_per_thread<R>();
  static constexpr int T = R / V;
  int row0, row_end, q0, j;
  __device__ TileRows(const int* tile_row0, const int* sys_off, int tile, int sys) {
    row0 = tile_row0[tile];
    row_end = min(row0 + BT, sys_off[sys + 1]);
    q0 = (threadIdx.x % T) * V;
    j = threadIdx.x / T;
  }
  __device__ int row(int pass) const { return row0 + pass * (BT / T) + j; }
};

// Block sums of ND x V values per thread (value [d][e] belongs to right-hand
// side q0 + e) into part[tile][d * R + q]; the last tile of the system to
// finish gets a pointer to the system totals (summed in tile order, entry
// d * R + q, in shared memory), every other tile nullptr.
template <int ND, int R>
__device__ __forceinline__ const double* system_reduce(double (&v)[ND][vals_per_thread<R>()],
                                                       double* __restrict__ part, unsigned* cnt, int tile, int t0,
                                                       int t1, int sys) {
  constexpr int V = vals_per_thread<R>(), T = R / V;
  __shared__ double red[ND * R][BT_WARPS];
  __shared__ double totals[ND * R];
  __shared__ int amlast;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int d = 0; d < ND; ++d)
#pragma unroll
    for (int e = 0; e < V; ++e) {
      double xs = v[d][e];
      // lanes j * T + qt of a warp share qt: fold over the row bits
#pragma unroll
      for (int o = 16; o >= T; o >>= 1) xs += __shfl_xor_sync(0xffffffffu, xs, o);
      if (lane < T) red[d * R + lane * V + e][wid] = xs;
    }
  __syncthreads();
  if (threadIdx.x < ND * R) {
    double ssum = 0.0;
#pragma unroll
    for (int w = 0; w < BT_WARPS; ++w) ssum += red[threadIdx.x][w];
    part[(size_t)tile * (3 * R) + threadIdx.x] = ssum;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned done = atomicAdd(&cnt[sys], 1u);
    amlast = (done == (unsigned)(t1 - t0 - 1)) ? 1 : 0;
  }
  __syncthreads();
  if (!amlast) return nullptr;
  __threadfence();
  // thread j < ND * R sums slot j over the system's tiles in order
  if (threadIdx.x < ND * R) {
    double ssum = 0.0;
    for (int t = t0; t < t1; ++t) ssum += __ldcg(part + (size_t)t * (3 * R) + threadIdx.x);
    totals[threadIdx.x] = ssum;
  }
  __syncthreads();
  if (threadIdx.x == 0) cnt[sys] = 0u;
  return totals;
}

// Every kernel of the batched iteration starts here: it lets the next kernel
// (programmatic dependent launch) be scheduled once all its blocks have
// passed this point, waits for the previous kernel to complete with its
// memory visible, then reads the batch's stop flag.
__device__ __forceinline__ bool g_finished(const BGlobal* g) {
  cudaTriggerProgrammaticLaunchCompletion();
  cudaGridDependencySynchronize();
  return *(volatile const int*)&g->done != 0;
}

// Launch with programmatic dependent launch (inside the captured graph: a
// programmatic edge from the previous kernel).
template <typename K, typename A>
cudaError_t launch_pdl_b(K kernel, int grid, int block, cudaStream_t st, const A& args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args);
}

// A system whose every pair stopped is skipped by all its tiles (nothing reads
// its vectors or partials any more).
template <int R>
__device__ __forceinline__ bool system_idle(const BArgs<R>& a, int sys) { return a.st.sys_live[sys] == 0; }

template <int R>
__global__ void __launch_bounds__(BT) kb_init(BArgs<R> a, double tol, int tol_mode) {
  constexpr int V = vals_per_thread<R>(), T = R / V;
  const int tile = blockIdx.x, sys = a.tile_sys[tile];
  const TileRows<R> tr(a.tile_row0, a.sys_off, tile, sys);
  double v[3][V] = {};
#pragma unroll 1
  for (int pass = 0; pass < T; ++pass) {
    const int row = tr.row(pass);
    if (row >= tr.row_end) break;
    double ax[V], bb[V], rr[V], zero[V];
    sell_row_v<V>(a.off, a.kd, a.su, a.aval, a.ix, row,
                  [&](int c, double (&o)[V]) { ldv<V>(a.x + (size_t)c * R + tr.q0, o); }, ax);
    const size_t i = (size_t)row * R + tr.q0;
    ldv<V>(a.b + i, bb);
#pragma unroll
    for (int e = 0; e < V; ++e) {
      rr[e] = bb[e] + (-1.0) * ax[e];
      zero[e] = 0.0;
      v[0][e] += rr[e] * rr[e];   // (r*, r) = (r, r) at the start
      v[1][e] += rr[e] * rr[e];
      v[2][e] += bb[e] * bb[e];
    }
    stv<V>(a.r + i, rr);
    stv<V>(a.rs + i, rr);
    stv<V>(a.p0 + i, zero);
    stv<V>(a.p1 + i, zero);
    stv<V>(a.ay + i, zero);
  }
  const double* tot = system_reduce<3, R>(v, a.part, a.cnt, tile, a.tile_off[sys], a.tile_off[sys + 1], sys);
  if (tot && threadIdx.x == 0) {
    int live = 0;
    for (int qq = 0; qq < R; ++qq) {
      const int i = sys * R + qq;
      a.st.rho[i] = tot[0 * R + qq];
      a.st.res[i] = sqrt(tot[1 * R + qq]);
      a.st.bnorm[i] = sqrt(tot[2 * R + qq]);
      a.st.thr[i] = (tol_mode == DCU_TOL_REL) ? tol * a.st.bnorm[i] : tol;
      a.st.alpha[i] = 0.0;
      a.st.omega[i] = 1.0;
      a.st.beta[i] = 0.0;
      const bool run = a.st.res[i] != 0.0 && a.g->maxiter > 1;
      a.st.active[i] = run ? 1 : 0;
      a.st.conv_it[i] = 1;
      a.st.status[i] = run ? -1 : (a.st.res[i] == 0.0 ? DCU_SOLVE_CONVERGED : DCU_SOLVE_MAXITER);
      live += run ? 1 : 0;
    }
    atomicAdd(&a.g->active_count, live);
    a.st.sys_live[sys] = live;
  }
}

// K1: p = r + beta (p - omega ay) at gathered columns; y = M p
template <int R>
__global__ void __launch_bounds__(BT) kb_py(BArgs<R> a) {
  constexpr int V = vals_per_thread<R>(), T = R / V;
  if (g_finished(a.g)) return;
  const int tile = blockIdx.x, sys = a.tile_sys[tile];
  if (system_idle(a, sys)) return;
  const TileRows<R> tr(a.tile_row0, a.sys_off, tile, sys);
  double beta[V], omega[V];
#pragma unroll
  for (int e = 0; e < V; ++e) {
    beta[e] = a.st.beta[sys * R + tr.q0 + e];
    omega[e] = a.st.omega[sys * R + tr.q0 + e];
  }
  const int pidx = a.g->pidx;
  const double* __restrict__ pold = pidx ? a.p1 : a.p0;
  double* __restrict__ pnew = pidx ? a.p0 : a.p1;
  auto pf = [&](int c, double (&o)[V]) {
    const size_t i = (size_t)c * R + tr.q0;
    double rr[V], pp[V], yy[V];
    ldv<V>(a.r + i, rr);
    ldv<V>(pold + i, pp);
    ldv<V>(a.ay + i, yy);
#pragma unroll
    for (int e = 0; e < V; ++e) o[e] = rr[e] + beta[e] * (pp[e] - omega[e] * yy[e]);
  };
#pragma unroll 1
  for (int pass = 0; pass < T; ++pass) {
    const int row = tr.row(pass);
    if (row >= tr.row_end) break;
    double yv[V], pv[V];
    sell_row_v<V>(a.off, a.kd, a.su, a.mval, a.ix, row, pf, yv);
    pf(row, pv);
    const size_t i = (size_t)row * R + tr.q0;
    stv<V>(pnew + i, pv);
    stv<V>(a.y + i, yv);
  }
}

// K2: ay = A y; alpha = rho / (r*, ay)
template <int R>
__global__ void __launch_bounds__(BT) kb_ay(BArgs<R> a) {
  constexpr int V = vals_per_thread<R>(), T = R / V;
  if (g_finished(a.g)) return;
  const int tile = blockIdx.x, sys = a.tile_sys[tile];
  if (system_idle(a, sys)) return;
  const TileRows<R> tr(a.tile_row0, a.sys_off, tile, sys);
  double v[1][V] = {};
#pragma unroll 1
  for (int pass = 0; pass < T; ++pass) {
    const int row = tr.row(pass);
    if (row >= tr.row_end) break;
    double ayv[V], rsv[V];
    sell_row_v<V>(a.off, a.kd, a.su, a.aval, a.ix, row,
                  [&](int c, double (&o)[V]) { ldv<V>(a.y + (size_t)c * R + tr.q0, o); }, ayv);
    const size_t i = (size_t)row * R + tr.q0;
    ldv<V>(a.rs + i, rsv);
    stv<V>(a.ay + i, ayv);
#pragma unroll
    for (int e = 0; e < V; ++e) v[0][e] += rsv[e] * ayv[e];
  }
  const double* tot = system_reduce<1, R>(v, a.part, a.cnt, tile, a.tile_off[sys], a.tile_off[sys + 1], sys);
  if (tot && threadIdx.x == 0) {
    for (int qq = 0; qq < R; ++qq) {
      const int i = sys * R + qq;
      if (!a.st.active[i]) continue;
      const double alpha = a.st.rho[i] / tot[0 * R + qq];
      a.st.alpha[i] = alpha;
      if (tot[0 * R + qq] == 0.0 || !isfinite(alpha)) {
        a.st.active[i] = 0;
        a.st.status[i] = DCU_SOLVE_BREAKDOWN;
        a.st.alpha[i] = a.st.omega[i] = a.st.beta[i] = 0.0;
        atomicSub(&a.g->active_count, 1);
        a.st.sys_live[sys] -= 1;
      }
    }
  }
}

// K3: s = r - alpha ay (on the fly at gathered columns); z = M s
template <int R>
__global__ void __launch_bounds__(BT) kb_sz(BArgs<R> a) {
  constexpr int V = vals_per_thread<R>(), T = R / V;
  if (g_finished(a.g)) return;
  const int tile = blockIdx.x, sys = a.tile_sys[tile];
  if (system_idle(a, sys)) return;
  const TileRows<R> tr(a.tile_row0, a.sys_off, tile, sys);
  double nalpha[V];
#pragma unroll
  for (int e = 0; e < V; ++e) nalpha[e] = -1.0 * a.st.alpha[sys * R + tr.q0 + e];
  auto sf = [&](int c, double (&o)[V]) {
    const size_t i = (size_t)c * R + tr.q0;
    double rr[V], yy[V];
    ldv<V>(a.r + i, rr);
    ldv<V>(a.ay + i, yy);
#pragma unroll
    for (int e = 0; e < V; ++e) o[e] = rr[e] + nalpha[e] * yy[e];
  };
#pragma unroll 1
  for (int pass = 0; pass < T; ++pass) {
    const int row = tr.row(pass);
    if (row >= tr.row_end) break;
    double zv[V], sv[V];
    sell_row_v<V>(a.off, a.kd, a.su, a.mval, a.ix, row, sf, zv);
    sf(row, sv);
    const size_t i = (size_t)row * R + tr.q0;
    stv<V>(a.s + i, sv);
    stv<V>(a.z + i, zv);
  }
}

// K4: az = A z; omega = (az, s) / (az, az)
template <int R>
__global__ void __launch_bounds__(BT) kb_az(BArgs<R> a) {
  constexpr int V = vals_per_thread<R>(), T = R / V;
  if (g_finished(a.g)) return;
  const int tile = blockIdx.x, sys = a.tile_sys[tile];
  if (system_idle(a, sys)) return;
  const TileRows<R> tr(a.tile_row0, a.sys_off, tile, sys);
  double v[2][V] = {};
#pragma unroll 1
  for (int pass = 0; pass < T; ++pass) {
    const int row = tr.row(pass);
    if (row >= tr.row_end) break;
    double azv[V], sv[V];
    sell_row_v<V>(a.off, a.kd, a.su, a.aval, a.ix, row,
                  [&](int c, double (&o)[V]) { ldv<V>(a.z + (size_t)c * R + tr.q0, o); }, azv);
    const size_t i = (size_t)row * R + tr.q0;
    ldv<V>(a.s + i, sv);
    stv<V>(a.az + i, azv);
#pragma unroll
    for (int e = 0; e < V; ++e) {
      v[0][e] += azv[e] * sv[e];
      v[1][e] += azv[e] * azv[e];
    }
  }
  const double* tot = system_reduce<2, R>(v, a.part, a.cnt, tile, a.tile_off[sys], a.tile_off[sys + 1], sys);
  if (tot && threadIdx.x == 0) {
    for (int qq = 0; qq < R; ++qq) {
      const int i = sys * R + qq;
      if (!a.st.active[i]) continue;
      // Az = 0 (s = 0 when the half step solved the pair): omega = 0
      const double omega = (tot[1 * R + qq] == 0.0) ? 0.0 : tot[0 * R + qq] / tot[1 * R + qq];
      a.st.omega[i] = omega;
      if (!isfinite(omega)) {
        a.st.active[i] = 0;
        a.st.status[i] = DCU_SOLVE_BREAKDOWN;
        a.st.alpha[i] = a.st.omega[i] = a.st.beta[i] = 0.0;
        atomicSub(&a.g->active_count, 1);
        a.st.sys_live[sys] -= 1;
      }
    }
  }
}

// K5: x += alpha y + omega z (active pairs); r = s - omega az; rho, beta, ||r||
template <int R>
__global__ void __launch_bounds__(BT) kb_xr(BArgs<R> a) {
  constexpr int V = vals_per_thread<R>(), T = R / V;
  if (g_finished(a.g)) return;
  const int tile = blockIdx.x, sys = a.tile_sys[tile];
  if (system_idle(a, sys)) return;
  const TileRows<R> tr(a.tile_row0, a.sys_off, tile, sys);
  double alpha[V], omega[V];
  bool active[V];
#pragma unroll
  for (int e = 0; e < V; ++e) {
    const int ip = sys * R + tr.q0 + e;
    alpha[e] = a.st.alpha[ip];
    omega[e] = a.st.omega[ip];
    active[e] = a.st.active[ip] != 0;
  }
  double v[2][V] = {};
#pragma unroll 1
  for (int pass = 0; pass < T; ++pass) {
    const int row = tr.row(pass);
    if (row >= tr.row_end) break;
    const size_t i = (size_t)row * R + tr.q0;
    double xv[V], yv[V], zv[V], sv[V], azv[V], rsv[V], rn[V];
    ldp<V>(a.x + i, xv);
    ldv<V>(a.y + i, yv);
    ldv<V>(a.z + i, zv);
    ldv<V>(a.s + i, sv);
    ldv<V>(a.az + i, azv);
    ldv<V>(a.rs + i, rsv);
#pragma unroll
    for (int e = 0; e < V; ++e) {
      if (active[e]) {
        double t = xv[e] + alpha[e] * yv[e];
        xv[e] = t + omega[e] * zv[e];
      }
      rn[e] = sv[e] + (-1.0 * omega[e]) * azv[e];
      v[0][e] += rsv[e] * rn[e];
      v[1][e] += rn[e] * rn[e];
    }
    stv<V>(a.x + i, xv);
    stv<V>(a.r + i, rn);
  }
  const double* tot = system_reduce<2, R>(v, a.part, a.cnt, tile, a.tile_off[sys], a.tile_off[sys + 1], sys);
  if (tot && threadIdx.x == 0) {
    const int it = a.g->it;
    for (int qq = 0; qq < R; ++qq) {
      const int i = sys * R + qq;
      if (!a.st.active[i]) continue;
      const double rho_new = tot[0 * R + qq];
      const double beta = (rho_new / a.st.rho[i]) * (a.st.alpha[i] / a.st.omega[i]);
      a.st.rho[i] = rho_new;
      a.st.beta[i] = beta;
      a.st.res[i] = sqrt(tot[1 * R + qq]);
      a.st.conv_it[i] = it;
      // the stop test first, as in the reference (it never examines beta)
      if (!isfinite(a.st.res[i])) {
        a.st.active[i] = 0;
        a.st.status[i] = DCU_SOLVE_BREAKDOWN;
      } else if (a.st.res[i] < a.st.thr[i]) {
        a.st.active[i] = 0;
        a.st.status[i] = DCU_SOLVE_CONVERGED;
      } else if (!isfinite(beta) || rho_new == 0.0) {
        a.st.active[i] = 0;
        a.st.status[i] = DCU_SOLVE_BREAKDOWN;
      } else if (it + 1 >= a.g->maxiter) {
        a.st.status[i] = DCU_SOLVE_MAXITER;
        a.st.conv_it[i] = it + 1;
      }
      if (!a.st.active[i]) {
        a.st.alpha[i] = a.st.omega[i] = a.st.beta[i] = 0.0;
        atomicSub(&a.g->active_count, 1);
        a.st.sys_live[sys] -= 1;
      }
    }
  }
}

// K6: one thread advances the shared counter after K5 and decides whether the
// batch is done.
template <int R>
__global__ void kb_step(BArgs<R> a) {
  if (g_finished(a.g)) return;
  BGlobal* g = a.g;
  g->pidx ^= 1;
  if (g->active_count <= 0) {
    g->done = 1;
  } else {
    g->it += 1;
    if (g->it >= g->maxiter) g->done = 1;
  }
}

// ---------------------------------------------------------------------------
// A cluster per system.
//
// The kernels above run every system's tiles in each launch: an iteration of
// the whole batch streams all its vectors through HBM and costs six launches.
// Here one cluster takes a
// system through its whole solve before the next one, its rows split over the
// cluster's CTAs, so that the vectors of the systems in flight stay in L2 (and
// r*, Az and x, which only their own row reads, in shared memory where they
// fit); the five steps of an iteration are separated by the cluster's hardware
// barrier, and a system costs its own iterations, not the batch's.  s and p are
// not stored: s = r - alpha Ay and p = r + beta q (q = p - omega Ay of the last
// iteration, published with r) are formed where they are used, by the same
// operations.  Systems are taken from a queue, the large ones from one end by
// the even clusters, the small ones from the other by the odd ones, so that
// large systems do not all share L2 at once.  Each CTA sums the same partials
// in the same order; a system's result does not depend on the order of the
// queue.
// ---------------------------------------------------------------------------
constexpr int BC_THREADS = 512;   // (1024 hold 64 registers each and spill: 265 -> 340 ms on 512 systems x 8)
constexpr int BC_MAXC = 16;

struct BCArgs {
  int count;                // systems of this launch ...
  const int* order;         // ... by size, descending
  int* head;                // [0] taken, [1] from the front, [2] from the back
  const int* sys_off;
  const long long* off;
  const int* ix;
  const double* aval;
  const double* mval;
  const double* b;
  double* x;
  double *r, *q, *y, *ay, *z, *rs, *az;
  double tol;
  int tol_mode, maxiter;
  int cap;                  // doubles of dynamic shared memory
  int* last;                // the batch's iteration counter: the latest that any system reached
  int* iters;
  int* status;
};

__device__ __forceinline__ unsigned bc_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned bc_size() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned bc_id() {
  unsigned r;
  asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned bc_remote(const void* p, unsigned rank) {
  unsigned o;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(o) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
  return o;
}
__device__ __forceinline__ void bc_barrier() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// A row's entries reach the CTA's shared memory a pass ahead of their use
// (cp.async, each row's copies by the T threads that share it, so a warp waits
// for its own copies only): a pass then waits for one gather instead of the
// chain slice offset -> values and columns -> gather.
constexpr int BC_W = 8;           // entries of a row that are prefetched (the rest are read in place)
constexpr int BC_LD = BC_W + 1;   // row stride (rows in different banks)
constexpr int BC_STAGES = 2;
constexpr int BC_SLICES = 256;    // 32-row slices of one CTA, at most

template <int R>
struct BCEntries {
  static constexpr int ROWS = BC_THREADS / (R / vals_per_thread<R>());  // rows of a pass
  double val[BC_STAGES][ROWS * BC_LD];
  int col[BC_STAGES][ROWS * BC_LD];
  int off[BC_SLICES + 1];         // first slot of each of the CTA's slices, from the first one's
};
template <int R>
__host__ __device__ constexpr size_t bc_entry_bytes() {
  static_assert(sizeof(BCEntries<R>) <= 128 * 1024, "room for the rows' own vectors, and for the entries at all");
  return (sizeof(BCEntries<R>) + 15) / 16 * 16;
}

__device__ __forceinline__ void bc_copy8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" : : "r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void bc_copy4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" : : "r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

// The rows of one CTA: entries ahead of their use, and their sums.
template <int R>
struct BCRows {
  static constexpr int V = vals_per_thread<R>(), T = R / V, ROWS = BCEntries<R>::ROWS;
  BCEntries<R>& E;
  const int* ix;
  int c0, rows, sl0;
  long long ob;   // first slot of the CTA's first slice

  __device__ __forceinline__ void prefetch(const double* val, int pass) const {
    const int jr = threadIdx.x / T, j = pass * ROWS + jr;
    if (j < rows) {
      const int row = c0 + j, sl = (row >> 5) - sl0;
      const int o = E.off[sl], w = min(BC_W, (E.off[sl + 1] - o) >> 5);
      const long long at = ob + o + (row & 31);
      double* dv = &E.val[pass % BC_STAGES][jr * BC_LD];
      int* dc = &E.col[pass % BC_STAGES][jr * BC_LD];
      for (int k = threadIdx.x % T; k < w; k += T) {
        bc_copy8(dv + k, val + at + 32ll * k);
        bc_copy4(dc + k, ix + at + 32ll * k);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  // The first pass of a phase over `val` (called before the barrier that opens
  // the phase: the matrix does not change).
  __device__ __forceinline__ void begin(const double* val) const {
    __syncwarp();
    prefetch(val, 0);
  }
  // The entries of `pass` are there; those of the next one are on their way
  // (into the stage that the pass before used).
  __device__ __forceinline__ void take(const double* val, int pass) const {
    __syncwarp();
    prefetch(val, pass + 1);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
  }
  // acc[e] = sum_k val[row, k] xf(col)[e] for this thread's row of `pass`
  template <typename F>
  __device__ __forceinline__ void sum(const double* val, int pass, int row, F xf, double (&acc)[V]) const {
    const int jr = threadIdx.x / T, sl = (row >> 5) - sl0;
    const int o = E.off[sl], w = (E.off[sl + 1] - o) >> 5;
    const double* sv = &E.val[pass % BC_STAGES][jr * BC_LD];
    const int* sc = &E.col[pass % BC_STAGES][jr * BC_LD];
#pragma unroll
    for (int e = 0; e < V; ++e) acc[e] = 0.0;
    const int wn = min(w, BC_W);
#pragma unroll
    for (int k0 = 0; k0 < BC_W; k0 += 4) {
      double xv[4][V];
#pragma unroll
      for (int t = 0; t < 4; ++t)
        if (k0 + t < wn) xf(sc[k0 + t], xv[t]);
#pragma unroll
      for (int t = 0; t < 4; ++t)
        if (k0 + t < wn) {
          const double av = sv[k0 + t];
#pragma unroll
          for (int e = 0; e < V; ++e) acc[e] += av * xv[t][e];
        }
    }
    for (int k = BC_W; k < w; ++k) {
      const long long at = ob + o + (row & 31) + 32ll * k;
      const double av = __ldg(val + at);
      double xv[V];
      xf(__ldg(ix + at), xv);
#pragma unroll
      for (int e = 0; e < V; ++e) acc[e] += av * xv[e];
    }
  }
};

// Sums of ND x V values per thread over the rows of a cluster's system; on
// return red[d * R + q][0] holds right-hand side q's total d for the threads of
// warp 0.  Everything stored before it is visible to the cluster after it.
template <int ND, int R>
__device__ __forceinline__ void bc_sum(double (&v)[ND][vals_per_thread<R>()], double (*red)[BC_THREADS / 32 + 1],
                                       double (*part)[BC_MAXC], unsigned rank, unsigned C) {
  constexpr int V = vals_per_thread<R>(), T = R / V, WARPS = BC_THREADS / 32;
  static_assert(2 * R <= WARPS, "a warp to a sum");
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
#pragma unroll
  for (int d = 0; d < ND; ++d)
#pragma unroll
    for (int e = 0; e < V; ++e) {
      double t = v[d][e];
#pragma unroll
      for (int o = 16; o >= T; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (lane < T) red[d * R + lane * V + e][wid] = t;
    }
  __syncthreads();
  if (wid < ND * R) {
    double t = lane < WARPS ? red[wid][lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane < (int)C)
      asm volatile("st.shared::cluster.f64 [%0], %1;" : : "r"(bc_remote(&part[wid][rank], (unsigned)lane)), "d"(t)
                   : "memory");
  }
  bc_barrier();
  if (wid == 0) {
    if (lane < ND * R) {
      double t = 0.0;
      for (unsigned c = 0; c < C; ++c) t += part[lane][c];
      red[lane][0] = t;  // (the warps' parts were read before the barrier)
    }
    __syncwarp();
  }
}

template <int R>
__global__ void __launch_bounds__(BC_THREADS, 1) k_batch_cluster(BCArgs a) {
  constexpr int V = vals_per_thread<R>(), T = R / V;
  constexpr int ROWS = BCEntries<R>::ROWS, THREADS = BC_THREADS;
  extern __shared__ __align__(16) unsigned char bc_raw[];
  BCEntries<R>& E = *reinterpret_cast<BCEntries<R>*>(bc_raw);
  double* bc_sm = reinterpret_cast<double*>(bc_raw + bc_entry_bytes<R>());
  __shared__ double red[2 * R][BC_THREADS / 32 + 1];
  __shared__ double part[2][2 * R][BC_MAXC];
  __shared__ double rho[R], alpha[R], omega[R], beta[R], res[R], thr[R];
  __shared__ int active[R], stat[R], conv[R];
  __shared__ int next;
  const int tid = threadIdx.x;
  const unsigned rank = bc_rank(), C = bc_size();
  const int q0 = (tid % T) * V;
  unsigned par = 0;
  bc_barrier();  // every CTA of the cluster has started

  // total d of right-hand side tid (threads below R; ND * R <= 32: one warp)
  auto total = [&](int d) { return red[d * R + tid][0]; };

  for (;;) {
    if (rank == 0 && tid == 0) {
      int s = -1;
      if (atomicAdd(a.head, 1) < a.count)
        s = (bc_id() & 1) ? a.order[a.count - 1 - atomicAdd(a.head + 2, 1)] : a.order[atomicAdd(a.head + 1, 1)];
      for (unsigned c = 0; c < C; ++c)
        asm volatile("st.shared::cluster.s32 [%0], %1;" : : "r"(bc_remote(&next, c)), "r"(s) : "memory");
    }
    bc_barrier();
    const int sys = next;
    if (sys < 0) break;
    const int s0 = a.sys_off[sys], s1 = a.sys_off[sys + 1];
    const int rpc = ((s1 - s0 + (int)C - 1) / (int)C + 7) & ~7;  // rows of a CTA
    const int c0 = min(s0 + rpc * (int)rank, s1), rows = min(rpc, s1 - c0);
    const size_t g0 = (size_t)c0 * R;
    // own-row vectors: shared memory while they fit (the same choice in every CTA)
    const int need = rpc * R;
    double* rs = need <= a.cap ? bc_sm : a.rs + g0;
    double* az = 2 * need <= a.cap ? bc_sm + need : a.az + g0;
    double* xs = 3 * need <= a.cap ? bc_sm + 2 * need : a.x + g0;
    const bool x_in = 3 * need <= a.cap;

    // the CTA's slice offsets
    const int sl0 = c0 >> 5, nsl = rows > 0 ? ((c0 + rows - 1) >> 5) - sl0 + 1 : 0;
    const long long ob = __ldg(a.off + sl0);
    for (int t = tid; t <= nsl; t += THREADS) E.off[t] = (int)(__ldg(a.off + sl0 + t) - ob);
    __syncthreads();
    const int npass = (rpc + ROWS - 1) / ROWS;
    const int jr = tid / T;        // this thread's row of a pass
    const BCRows<R> rw{E, a.ix, c0, rows, sl0, ob};
    rw.begin(a.aval);

    // r = b - A x, r* = r, q = 0
    {
      double v[2][V] = {};
      for (int pass = 0; pass < npass; ++pass) {
        rw.take(a.aval, pass);
        const int j = pass * ROWS + jr;
        if (j >= rows) continue;
        const int row = c0 + j, li = j * R + q0;
        const size_t i = g0 + li;
        double ax[V], bb[V], rr[V], zero[V] = {};
        rw.sum(a.aval, pass, row, [&](int c, double (&o)[V]) { ldp<V>(a.x + (size_t)c * R + q0, o); }, ax);
        ldv<V>(a.b + i, bb);
#pragma unroll
        for (int e = 0; e < V; ++e) {
          rr[e] = bb[e] + (-1.0) * ax[e];
          v[0][e] += rr[e] * rr[e];
          v[1][e] += bb[e] * bb[e];
        }
        stv<V>(a.r + i, rr);
        stv<V>(rs + li, rr);
        stv<V>(a.q + i, zero);
        stv<V>(a.ay + i, zero);
        if (x_in) {
          double xv[V];
          ldp<V>(a.x + i, xv);
          stv<V>(xs + li, xv);
        }
      }
      rw.begin(a.mval);
      par ^= 1u;
      bc_sum<2, R>(v, red, part[par], rank, C);
      if (tid < R) {
        rho[tid] = total(0);
        res[tid] = sqrt(total(0));
        const double bn = sqrt(total(1));
        thr[tid] = (a.tol_mode == DCU_TOL_REL) ? a.tol * bn : a.tol;
        alpha[tid] = 0.0;
        omega[tid] = 1.0;
        beta[tid] = 0.0;
        const bool run = res[tid] != 0.0 && a.maxiter > 1;
        active[tid] = run ? 1 : 0;
        conv[tid] = 1;
        stat[tid] = run ? -1 : (res[tid] == 0.0 ? DCU_SOLVE_CONVERGED : DCU_SOLVE_MAXITER);
      }
    }
    int it = 1;
    int live = __syncthreads_count(tid < R && active[tid < R ? tid : 0]);
    // a pair that stopped keeps alpha = omega = beta = 0: its x no longer changes
    auto freeze = [&](int status) {
      active[tid] = 0;
      stat[tid] = status;
      alpha[tid] = omega[tid] = beta[tid] = 0.0;
    };
    while (live > 0 && it < a.maxiter) {
      double be[V];
#pragma unroll
      for (int e = 0; e < V; ++e) be[e] = beta[q0 + e];
      // y = M p
      for (int pass = 0; pass < npass; ++pass) {
        rw.take(a.mval, pass);
        const int j = pass * ROWS + jr;
        if (j >= rows) continue;
        const int row = c0 + j;
        double yv[V];
        rw.sum(a.mval, pass, row, [&](int c, double (&o)[V]) {
          double rr[V], qq[V];
          ldp<V>(a.r + (size_t)c * R + q0, rr);
          ldp<V>(a.q + (size_t)c * R + q0, qq);
#pragma unroll
          for (int e = 0; e < V; ++e) o[e] = rr[e] + be[e] * qq[e];
        }, yv);
        stv<V>(a.y + g0 + j * R + q0, yv);
      }
      rw.begin(a.aval);
      bc_barrier();
      // Ay, alpha
      {
        double v[1][V] = {};
        for (int pass = 0; pass < npass; ++pass) {
          rw.take(a.aval, pass);
          const int j = pass * ROWS + jr;
          if (j >= rows) continue;
          const int row = c0 + j, li = j * R + q0;
          double t[V], s[V];
          ldp<V>(rs + li, s);
          rw.sum(a.aval, pass, row, [&](int c, double (&o)[V]) { ldp<V>(a.y + (size_t)c * R + q0, o); }, t);
          stv<V>(a.ay + g0 + li, t);
#pragma unroll
          for (int e = 0; e < V; ++e) v[0][e] += s[e] * t[e];
        }
        rw.begin(a.mval);
        par ^= 1u;
        bc_sum<1, R>(v, red, part[par], rank, C);
        if (tid < R && active[tid]) {
          const double d = total(0), al = rho[tid] / d;
          alpha[tid] = al;
          if (d == 0.0 || !isfinite(al)) freeze(DCU_SOLVE_BREAKDOWN);
        }
        __syncthreads();
      }
      double na[V];
#pragma unroll
      for (int e = 0; e < V; ++e) na[e] = -1.0 * alpha[q0 + e];
      // z = M s
      for (int pass = 0; pass < npass; ++pass) {
        rw.take(a.mval, pass);
        const int j = pass * ROWS + jr;
        if (j >= rows) continue;
        const int row = c0 + j;
        double zv[V];
        rw.sum(a.mval, pass, row, [&](int c, double (&o)[V]) {
          double rr[V], yy[V];
          ldp<V>(a.r + (size_t)c * R + q0, rr);
          ldp<V>(a.ay + (size_t)c * R + q0, yy);
#pragma unroll
          for (int e = 0; e < V; ++e) o[e] = rr[e] + na[e] * yy[e];
        }, zv);
        stv<V>(a.z + g0 + j * R + q0, zv);
      }
      rw.begin(a.aval);
      bc_barrier();
      // Az, omega
      {
        double v[2][V] = {};
        for (int pass = 0; pass < npass; ++pass) {
          rw.take(a.aval, pass);
          const int j = pass * ROWS + jr;
          if (j >= rows) continue;
          const int row = c0 + j, li = j * R + q0;
          double t[V], rr[V], yy[V];
          ldp<V>(a.r + g0 + li, rr);
          ldp<V>(a.ay + g0 + li, yy);
          rw.sum(a.aval, pass, row, [&](int c, double (&o)[V]) { ldp<V>(a.z + (size_t)c * R + q0, o); }, t);
          stv<V>(az + li, t);
#pragma unroll
          for (int e = 0; e < V; ++e) {
            v[0][e] += t[e] * (rr[e] + na[e] * yy[e]);
            v[1][e] += t[e] * t[e];
          }
        }
        rw.begin(a.mval);
        par ^= 1u;
        bc_sum<2, R>(v, red, part[par], rank, C);
        if (tid < R && active[tid]) {
          // Az = 0 (s = 0 when the half step solved the pair): omega = 0
          const double om = (total(1) == 0.0) ? 0.0 : total(0) / total(1);
          omega[tid] = om;
          if (!isfinite(om)) freeze(DCU_SOLVE_BREAKDOWN);
        }
        __syncthreads();
      }
      // x, r, q; rho, beta, ||r||
      {
        double al[V], om[V], be2[V];
        bool act[V];
#pragma unroll
        for (int e = 0; e < V; ++e) {
          al[e] = alpha[q0 + e];
          om[e] = omega[q0 + e];
          be2[e] = beta[q0 + e];
          act[e] = active[q0 + e] != 0;
        }
        double v[2][V] = {};
        for (int j = tid / T; j < rows; j += THREADS / T) {
          const int li = j * R + q0;
          const size_t i = g0 + li;
          double xv[V], yv[V], zv[V], rr[V], qq[V], yy[V], tt[V], s[V];
          ldp<V>(xs + li, xv);
          ldp<V>(a.y + i, yv);
          ldp<V>(a.z + i, zv);
          ldp<V>(a.r + i, rr);
          ldp<V>(a.q + i, qq);
          ldp<V>(a.ay + i, yy);
          ldp<V>(az + li, tt);
          ldp<V>(rs + li, s);
#pragma unroll
          for (int e = 0; e < V; ++e) {
            if (act[e]) {
              const double t = xv[e] + al[e] * yv[e];
              xv[e] = t + om[e] * zv[e];
            }
            const double p = rr[e] + be2[e] * qq[e];
            const double sv = rr[e] + (-1.0 * al[e]) * yy[e];
            const double rn = sv + (-1.0 * om[e]) * tt[e];
            qq[e] = p - om[e] * yy[e];
            rr[e] = rn;
            v[0][e] += s[e] * rn;
            v[1][e] += rn * rn;
          }
          stv<V>(xs + li, xv);
          stv<V>(a.r + i, rr);
          stv<V>(a.q + i, qq);
        }
        par ^= 1u;
        bc_sum<2, R>(v, red, part[par], rank, C);
        if (tid < R && active[tid]) {
          const double rho_new = total(0);
          const double bt = (rho_new / rho[tid]) * (alpha[tid] / omega[tid]);
          rho[tid] = rho_new;
          beta[tid] = bt;
          res[tid] = sqrt(total(1));
          conv[tid] = it;
          // the stop test first, as in the reference (it never examines beta)
          if (!isfinite(res[tid])) freeze(DCU_SOLVE_BREAKDOWN);
          else if (res[tid] < thr[tid]) freeze(DCU_SOLVE_CONVERGED);
          else if (!isfinite(bt) || rho_new == 0.0) freeze(DCU_SOLVE_BREAKDOWN);
          else if (it + 1 >= a.maxiter) conv[tid] = it + 1;
        }
        live = __syncthreads_count(tid < R && active[tid < R ? tid : 0]);
        ++it;
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (x_in)
      for (int j = tid / T; j < rows; j += THREADS / T) {
        double xv[V];
        ldp<V>(xs + j * R + q0, xv);
        stv<V>(a.x + g0 + j * R + q0, xv);
      }
    if (rank == 0 && tid < R) {
      a.iters[(size_t)sys * R + tid] = conv[tid];
      a.status[(size_t)sys * R + tid] = stat[tid] < 0 ? DCU_SOLVE_MAXITER : stat[tid];
      // (kb_step's counter: it stays on the iteration in which the last pair stopped)
      if (tid == 0) atomicMax(a.last, live == 0 ? max(1, it - 1) : it);
    }
    __syncthreads();
  }
  bc_barrier();  // no CTA leaves while another may still write into its shared memory
}

// The padding slots of an offset-aligned slice (value 0, column row + offset)
// reach over a system's ends.  The neighbour's vectors may not have been
// written yet, or hold a NaN of its own, and 0 * NaN would end this system too:
// such a slot gets its own row as column, and its slice is read by index.
// Once a call: 512 systems x 8 take 217 ms before and 216 with it; holding every
// gathered column to its system's rows instead cost the tile kernels 1.2%.
__global__ void kb_own_columns(const int* __restrict__ sys_off, int nsys, int n, const long long* __restrict__ off,
                               int* __restrict__ ix, int* __restrict__ kd, int* __restrict__ su) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    // the first system that ends after the row
    int lo = 0, hi = nsys - 1;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (sys_off[mid + 1] > r) hi = mid;
      else lo = mid + 1;
    }
    const int s0 = sys_off[lo], s1 = sys_off[lo + 1];
    if (r < s0 || r >= s1) continue;  // in no system
    const long long o0 = off[r >> 5];
    const int w = (int)((off[(r >> 5) + 1] - o0) >> 5);
    bool mine = false;
    for (int k = 0; k < w; ++k) {
      const long long q = o0 + 32ll * k + (r & 31);
      const int c = ix[q];
      if (c >= s0 && c < s1) continue;
      ix[q] = r;
      kd[(o0 >> 5) + k] = 0;
      mine = true;
    }
    if (mine) atomicAnd(su + (r >> 5), ~1);
  }
}

__global__ void kb_check_blocks(const int* __restrict__ ptr, const int* __restrict__ idx, const int* __restrict__ sys_off,
                                int nsys, int n, int* __restrict__ bad) {
  // every column's rows lie in its own diagonal block
  for (int s = blockIdx.x; s < nsys; s += gridDim.x) {
    const int c0 = sys_off[s], c1 = sys_off[s + 1];
    if (threadIdx.x == 0 && (c1 < c0 || c0 < 0 || c1 > n)) atomicOr(bad, 1);
    for (int c = c0 + threadIdx.x; c < c1 && c0 >= 0 && c1 <= n; c += blockDim.x)
      for (int e = ptr[c]; e < ptr[c + 1]; ++e)
        if (idx[e] < c0 || idx[e] >= c1) atomicOr(bad, 2);
  }
}

// CTAs of a system's cluster: two passes of rows each, up to 16.
template <int R>
int batch_ctas(int rows) {
  int k = 1;
  while (k < BC_MAXC && rows > 2 * BCEntries<R>::ROWS * k) k <<= 1;
  return k;
}

// Whether a batch goes to the clusters: two estimates of the time of one
// iteration of all its systems, in us on one B200, a system of n rows counted
// sqrt(n / largest) times (the iterations of a stencil grow with its width).
//   clusters  a system's iteration takes 3.7 us and 5.6 to 7.2 us for every pass
//             of its CTAs' rows (a fifth more at 8 right-hand sides once r* of
//             the rows no longer fits shared memory); 148, 74, 33, 15 and 7
//             clusters of 1, 2, 4, 8 and 16 CTAs run at once, one after
//             another.  At least the longest system, and whole rounds of every
//             class.
//   tiles     six launches, the tiles, their rows, and the last tile's sum over
//             its system's tiles.
// The constants are fitted to batches of 1 to 8192 equal systems of 16 to 90000
// rows.  The clusters may be estimated up to 1.2 times as long: a cluster
// costs a system's own iterations, the tiles' launches go on until the last
// system stops, and equal sizes converge apart too; less with more right-hand
// sides, where rows outweigh launches.  Of 156 batches with random sizes and
// coefficients the rule is never over 1.04 times the tiles' time, nor over 1.18
// times the faster one's.  Solve times, tiles and clusters, ms: 4096 systems of 64
// rows x 1 2.3 and 3.1; 2048 of 100 to 300 x 4 3.7 and 3.1; 1000 of 300 to 1000
// x 1 3.0 and 2.0; 300 of 300 to 4000 x 8 7.6 and 8.8, x 1 2.8 and 1.8; 64 of 20000
// to 50000 x 1 30 and 22, x 8 92 and 120.
template <int R>
bool cluster_batch(const std::vector<int>& so, int nsys) {
  constexpr double pass_us = R == 1 ? 5.6 : R == 2 ? 7.2 : R == 4 ? 6.9 : 7.0;
  constexpr double row_us = R == 1 ? 25e-6 : R == 2 ? 28e-6 : R == 4 ? 33e-6 : 34e-6;
  constexpr double slack = R <= 2 ? 1.2 : 1.15;
  constexpr int own = R == 8 ? (int)((64 * 1024 - bc_entry_bytes<R>()) / (sizeof(double) * R)) : INT_MAX;
  constexpr int resident[5] = {148, 74, 33, 15, 7};
  int tall = 0;
  for (int s = 0; s < nsys; ++s) tall = std::max(tall, so[s + 1] - so[s]);
  if (tall > BC_MAXC * (32 * (BC_SLICES - 2) - 8)) return false;  // slices of a CTA
  double tiles = 23.5 + 2.0 * R * std::min(1.0, tall / (double)BT) + 0.1 * ((tall + BT - 1) / BT);
  double class_us[5] = {}, most = 0.0, all = 0.0;
  int class_n[5] = {};
  for (int s = 0; s < nsys; ++s) {
    const int n = so[s + 1] - so[s];
    if (n <= 0) continue;
    const int k = batch_ctas<R>(n), rpc = (n + k - 1) / k;
    const int passes = (rpc + BCEntries<R>::ROWS - 1) / BCEntries<R>::ROWS;
    const int c = k == 1 ? 0 : k == 2 ? 1 : k == 4 ? 2 : k == 8 ? 3 : 4;
    const double w = std::sqrt((double)n / tall), us = w * (3.7 + (rpc > own ? 1.2 : 1.0) * pass_us * passes);
    ++class_n[c];
    class_us[c] += us;
    most = std::max(most, us);
    tiles += w * ((n + BT - 1) / BT * (0.018 + 0.002 * R) + n * R * row_us);
  }
  for (int c = 0; c < 5; ++c) {
    if (class_n[c] == 0) continue;
    all += class_us[c] / resident[c];
    most = std::max(most, (class_n[c] + resident[c] - 1) / resident[c] * class_us[c] / class_n[c]);
  }
  return std::max(all, most) < slack * tiles;
}

// The systems of a batch through k_batch_cluster: classes by size, the larger
// the system the more CTAs share it.  *ran stays false when the device cannot
// hold the clusters.
template <int R>
int run_batch_clusters(Ctx* c, int nsys, const int* sys_off_d, const std::vector<int>& so, const SellPlan& plan,
                       const double* aval, const double* mval, const double* B, double* X, const dcu_options* opt,
                       int* iters_h, int* status_h, dcu_solve_info* info, bool* ran) {
  const int n = plan.n;
  auto kernel = k_batch_cluster<R>;
  // shared memory: the entries, then the rows' own vectors (more of it made no
  // difference: 60, 120 and 210 KB within 1%)
  const size_t smem = std::max<size_t>(64 * 1024, bc_entry_bytes<R>());
  if (smem + 16 * 1024 > c->smem_optin) return DCU_OK;
  DCU_CUDA(c, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  DCU_CUDA(c, cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  std::vector<int> order(nsys);
  for (int s = 0; s < nsys; ++s) order[s] = s;
  std::stable_sort(order.begin(), order.end(), [&](int p, int q) { return so[p + 1] - so[p] > so[q + 1] - so[q]; });
  struct Class {
    int cta, first, count, grid;
  };
  std::vector<Class> cls;
  for (int i = 0; i < nsys; ++i) {
    const int k = batch_ctas<R>(so[order[i] + 1] - so[order[i]]);
    if (cls.empty() || cls.back().cta != k) cls.push_back({k, i, 0, 0});
    ++cls.back().count;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(BC_THREADS);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  for (auto& k : cls) {
    int fit = 0;
    at[0].val.clusterDim.x = k.cta;
    cfg.gridDim = dim3(k.cta);
    if (cudaOccupancyMaxActiveClusters(&fit, kernel, &cfg) != cudaSuccess || fit < 1) {
      cudaGetLastError();
      return DCU_OK;
    }
    k.grid = std::min(fit, k.count) * k.cta;
  }
  auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
  const size_t vec = al(sizeof(double) * (size_t)n * R), pairs = (size_t)nsys * R;
  const size_t heads = al(sizeof(int) * (3 * cls.size() + 1));
  DCU_TRY(ensure(c, B_VEC, 7 * vec + heads + al(sizeof(int) * nsys) + 2 * al(sizeof(int) * pairs)));
  char* p = bp<char>(c, B_VEC);
  BCArgs a{};
  a.sys_off = sys_off_d;
  a.off = plan.off;
  a.ix = plan.idx;
  a.aval = aval;
  a.mval = mval;
  a.b = B;
  a.x = X;
  double** vecs[7] = {&a.r, &a.q, &a.y, &a.ay, &a.z, &a.rs, &a.az};
  for (int i = 0; i < 7; ++i) *vecs[i] = reinterpret_cast<double*>(p + i * vec);
  int* head = reinterpret_cast<int*>(p + 7 * vec);
  a.last = head + 3 * cls.size();
  int* ord = reinterpret_cast<int*>(p + 7 * vec + heads);
  a.iters = reinterpret_cast<int*>(p + 7 * vec + heads + al(sizeof(int) * nsys));
  a.status = reinterpret_cast<int*>(p + 7 * vec + heads + al(sizeof(int) * nsys) + al(sizeof(int) * pairs));
  a.tol = opt->tol;
  a.tol_mode = opt->tol_mode;
  a.maxiter = opt->maxiter > 0 ? opt->maxiter : n;
  a.cap = (int)((smem - bc_entry_bytes<R>()) / sizeof(double));
  DCU_CUDA(c, cudaMemsetAsync(head, 0, heads, c->stream));
  DCU_CUDA(c, cudaMemcpyAsync(ord, order.data(), sizeof(int) * nsys, cudaMemcpyHostToDevice, c->stream));
  DCU_CUDA(c, cudaEventRecord(c->ev[0], c->stream));
  // every second class on the auxiliary stream: its clusters start as the
  // larger systems' last ones leave the SMs
  DCU_CUDA(c, cudaEventRecord(c->ev[6], c->stream));
  DCU_CUDA(c, cudaStreamWaitEvent(c->aux_stream, c->ev[6], 0));
  for (size_t k = 0; k < cls.size(); ++k) {
    a.count = cls[k].count;
    a.order = ord + cls[k].first;
    a.head = head + 3 * k;
    at[0].val.clusterDim.x = cls[k].cta;
    cfg.gridDim = dim3(cls[k].grid);
    cfg.stream = (k & 1) ? c->aux_stream : c->stream;
    DCU_CUDA(c, cudaLaunchKernelEx(&cfg, kernel, a));
    c->launches++;
  }
  DCU_CUDA(c, cudaEventRecord(c->ev[7], c->aux_stream));
  DCU_CUDA(c, cudaStreamWaitEvent(c->stream, c->ev[7], 0));
  DCU_CUDA(c, cudaEventRecord(c->ev[1], c->stream));
  DCU_CUDA(c, cudaMemcpyAsync(iters_h, a.iters, sizeof(int) * pairs, cudaMemcpyDeviceToHost, c->stream));
  DCU_CUDA(c, cudaMemcpyAsync(status_h, a.status, sizeof(int) * pairs, cudaMemcpyDeviceToHost, c->stream));
  int* last = static_cast<int*>(c->pinned);
  DCU_CUDA(c, cudaMemcpyAsync(last, a.last, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
  DCU_CUDA(c, cudaStreamSynchronize(c->stream));
  *ran = true;
  if (info) {
    info->iters = *last;
    info->status = DCU_SOLVE_CONVERGED;
    for (size_t i = 0; i < pairs; ++i) info->status = std::max(info->status, status_h[i]);
    info->replacements = 0;
    info->res = info->true_res = info->bnorm = 0.0;
    info->a_fp32 = 0;
    cudaEventElapsedTime(&info->ms, c->ev[0], c->ev[1]);
  }
  return DCU_OK;
}

template <int R>
int run_batch(Ctx* c, int nsys, const int* sys_off_d, const SellPlan& plan, const double* aval, const double* mval,
              const double* B, double* X, const dcu_options* opt, int* iters_h, int* status_h,
              dcu_solve_info* info) {
  const int n = plan.n;
  // host copy of the system offsets -> tiles
  std::vector<int> so(nsys + 1);
  DCU_CUDA(c, cudaMemcpyAsync(so.data(), sys_off_d, sizeof(int) * (nsys + 1), cudaMemcpyDeviceToHost, c->stream));
  DCU_CUDA(c, cudaStreamSynchronize(c->stream));
  bool rows = false;
  for (int s = 0; s < nsys; ++s) rows = rows || so[s + 1] > so[s];
  if (!rows) return fail(c, DCU_ERR_ARG, "empty batch");
  if (cluster_batch<R>(so, nsys)) {
    bool ran = false;
    DCU_TRY(run_batch_clusters<R>(c, nsys, sys_off_d, so, plan, aval, mval, B, X, opt, iters_h, status_h, info, &ran));
    if (ran) return DCU_OK;
  }
  std::vector<int> tsys, trow, toff(nsys + 1, 0);
  for (int s = 0; s < nsys; ++s) {
    toff[s] = (int)tsys.size();
    for (int r0 = so[s]; r0 < so[s + 1]; r0 += BT) {
      tsys.push_back(s);
      trow.push_back(r0);
    }
  }
  toff[nsys] = (int)tsys.size();
  const int ntiles = (int)tsys.size();
  auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
  const size_t vec = al(sizeof(double) * (size_t)n * R);
  const size_t pairs = (size_t)nsys * R;
  const size_t small = al(sizeof(int) * (2 * (size_t)ntiles + nsys + 1)) + al(sizeof(unsigned) * nsys) +
                       al(sizeof(double) * 3 * R * (size_t)ntiles) + al(sizeof(double) * 7 * pairs) +
                       al(sizeof(int) * 3 * pairs) + al(sizeof(int) * (size_t)nsys) + al(sizeof(BGlobal));
  DCU_TRY(ensure(c, B_VEC, 9 * vec + small));
  char* p = bp<char>(c, B_VEC);
  BArgs<R> a;
  std::memset(&a, 0, sizeof(a));  // padding included: the struct keys the graph cache
  a.n = n;
  a.nsys = nsys;
  a.ntiles = ntiles;
  a.sys_off = sys_off_d;
  a.off = plan.off;
  a.kd = plan.kd;
  a.su = plan.su;
  a.ix = plan.idx;
  a.aval = aval;
  a.mval = mval;
  a.b = B;
  a.x = X;
  double* vecs[9];
  for (int i = 0; i < 9; ++i) vecs[i] = reinterpret_cast<double*>(p + i * vec);
  a.r = vecs[0]; a.rs = vecs[1]; a.p0 = vecs[2]; a.p1 = vecs[3]; a.y = vecs[4];
  a.ay = vecs[5]; a.s = vecs[6]; a.z = vecs[7]; a.az = vecs[8];
  char* q = p + 9 * vec;
  int* tiles = reinterpret_cast<int*>(q);
  a.tile_sys = tiles;
  a.tile_row0 = tiles + ntiles;
  a.tile_off = tiles + 2 * ntiles;
  q += al(sizeof(int) * (2 * (size_t)ntiles + nsys + 1));
  a.cnt = reinterpret_cast<unsigned*>(q);
  q += al(sizeof(unsigned) * nsys);
  a.part = reinterpret_cast<double*>(q);
  q += al(sizeof(double) * 3 * R * (size_t)ntiles);
  double* dst = reinterpret_cast<double*>(q);
  a.st.rho = dst; a.st.alpha = dst + pairs; a.st.omega = dst + 2 * pairs; a.st.beta = dst + 3 * pairs;
  a.st.res = dst + 4 * pairs; a.st.thr = dst + 5 * pairs; a.st.bnorm = dst + 6 * pairs;
  q += al(sizeof(double) * 7 * pairs);
  int* ist = reinterpret_cast<int*>(q);
  a.st.active = ist; a.st.conv_it = ist + pairs; a.st.status = ist + 2 * pairs;
  q += al(sizeof(int) * 3 * pairs);
  a.st.sys_live = reinterpret_cast<int*>(q);
  q += al(sizeof(int) * (size_t)nsys);
  a.g = reinterpret_cast<BGlobal*>(q);
  DCU_CUDA(c, cudaMemcpyAsync(tiles, tsys.data(), sizeof(int) * ntiles, cudaMemcpyHostToDevice, c->stream));
  DCU_CUDA(c, cudaMemcpyAsync(tiles + ntiles, trow.data(), sizeof(int) * ntiles, cudaMemcpyHostToDevice, c->stream));
  DCU_CUDA(c, cudaMemcpyAsync(tiles + 2 * ntiles, toff.data(), sizeof(int) * (nsys + 1), cudaMemcpyHostToDevice,
                              c->stream));
  DCU_CUDA(c, cudaMemsetAsync(a.cnt, 0, sizeof(unsigned) * nsys, c->stream));
  const int maxiter = opt->maxiter > 0 ? opt->maxiter : n;
  BGlobal g0{};
  g0.it = 1;
  g0.maxiter = maxiter;
  DCU_CUDA(c, cudaMemcpyAsync(a.g, &g0, sizeof(BGlobal), cudaMemcpyHostToDevice, c->stream));
  DCU_CUDA(c, cudaEventRecord(c->ev[0], c->stream));
  kb_init<R><<<ntiles, BT, 0, c->stream>>>(a, opt->tol, opt->tol_mode);
  DCU_LAUNCHED(c, "kb_init");
  // the first iteration starts with p = r: beta = 0 and p, ay zero-filled
  std::vector<const void*> key = {(const void*)&kb_py<R>, (const void*)(intptr_t)ntiles};
  key_append(key, a);
  GraphSlot* ge = nullptr;
  for (auto& e : c->graphs)
    if (e.key == key) ge = &e;
  if (!ge) {
    cudaGraph_t gr = nullptr;
    DCU_CUDA(c, cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal));
    cudaError_t le = cudaSuccess;
    for (int i = 0; i < BCHUNK && le == cudaSuccess; ++i) {
      le = launch_pdl_b(kb_py<R>, ntiles, BT, c->stream, a);
      if (le == cudaSuccess) le = launch_pdl_b(kb_ay<R>, ntiles, BT, c->stream, a);
      if (le == cudaSuccess) le = launch_pdl_b(kb_sz<R>, ntiles, BT, c->stream, a);
      if (le == cudaSuccess) le = launch_pdl_b(kb_az<R>, ntiles, BT, c->stream, a);
      if (le == cudaSuccess) le = launch_pdl_b(kb_xr<R>, ntiles, BT, c->stream, a);
      if (le == cudaSuccess) le = launch_pdl_b(kb_step<R>, 1, 1, c->stream, a);
    }
    cudaError_t e = cudaStreamEndCapture(c->stream, &gr);
    if (le != cudaSuccess) {
      if (gr) cudaGraphDestroy(gr);
      return cuda_fail(c, le, "cudaLaunchKernelEx (capture)", __FILE__, __LINE__);
    }
    if (e != cudaSuccess) return cuda_fail(c, e, "cudaStreamEndCapture", __FILE__, __LINE__);
    GraphSlot ne;
    ne.key = key;
    ne.nodes = 6 * BCHUNK;
    e = cudaGraphInstantiate(&ne.exec, gr, 0);
    cudaGraphDestroy(gr);
    if (e != cudaSuccess) return cuda_fail(c, e, "cudaGraphInstantiate", __FILE__, __LINE__);
    if (c->graphs.size() >= 8) {
      cudaGraphExecDestroy(c->graphs.front().exec);
      c->graphs.erase(c->graphs.begin());
    }
    c->graphs.push_back(ne);
    ge = &c->graphs.back();
  }
  int* flag = reinterpret_cast<int*>(reinterpret_cast<char*>(c->pinned) + 1024);
  const long long max_chunks = (long long)maxiter / BCHUNK + 4;
  for (long long i = 0;; ++i) {
    if (i > max_chunks) return fail(c, DCU_ERR_CUDA, "batched solver did not terminate");
    DCU_CUDA(c, cudaGraphLaunch(ge->exec, c->stream));
    c->launches += ge->nodes;
    DCU_CUDA(c, cudaMemcpyAsync(flag + (i & 1), &a.g->done, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    DCU_CUDA(c, cudaEventRecord(c->ev[2 + (i & 1)], c->stream));
    if (i > 0) {
      DCU_CUDA(c, cudaEventSynchronize(c->ev[2 + ((i - 1) & 1)]));
      if (flag[(i - 1) & 1]) break;
    }
  }
  DCU_CUDA(c, cudaEventRecord(c->ev[1], c->stream));
  DCU_CUDA(c, cudaMemcpyAsync(iters_h, a.st.conv_it, sizeof(int) * pairs, cudaMemcpyDeviceToHost, c->stream));
  DCU_CUDA(c, cudaMemcpyAsync(status_h, a.st.status, sizeof(int) * pairs, cudaMemcpyDeviceToHost, c->stream));
  BGlobal gh;
  DCU_CUDA(c, cudaMemcpyAsync(&gh, a.g, sizeof(BGlobal), cudaMemcpyDeviceToHost, c->stream));
  DCU_CUDA(c, cudaStreamSynchronize(c->stream));
  int worst = DCU_SOLVE_CONVERGED;
  for (size_t i = 0; i < pairs; ++i) {
    if (status_h[i] < 0) {   // still running when the shared counter hit maxiter
      status_h[i] = DCU_SOLVE_MAXITER;
      iters_h[i] = gh.it;
    }
    worst = std::max(worst, status_h[i]);
  }
  if (info) {
    info->iters = gh.it;
    info->status = worst;
    info->replacements = 0;
    info->res = info->true_res = info->bnorm = 0.0;
    info->a_fp32 = 0;  // the batched kernels read A's FP64 values
    float ms = 0.f;
    cudaEventElapsedTime(&ms, c->ev[0], c->ev[1]);
    info->ms = ms;
  }
  return DCU_OK;
}

}  // namespace

int check_blocks(Ctx* c, int n, const int* ptr, const int* idx, int nsys, const int* sys_off) {
  DCU_TRY(ensure(c, B_STATS, sizeof(int) * 16));
  int* bad = bp<int>(c, B_STATS);
  DCU_CUDA(c, cudaMemsetAsync(bad, 0, sizeof(int), c->stream));
  kb_check_blocks<<<std::min(nsys, 4096), 128, 0, c->stream>>>(ptr, idx, sys_off, nsys, n, bad);
  DCU_LAUNCHED(c, "kb_check_blocks");
  int h = 0;
  DCU_CUDA(c, cudaMemcpyAsync(&h, bad, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
  DCU_CUDA(c, cudaStreamSynchronize(c->stream));
  if (h) return fail(c, DCU_ERR_ARG, "matrix is not block diagonal with respect to the system offsets (%d)", h);
  return DCU_OK;
}

int batch_solve(Ctx* c, int nsys, const int* sys_off, const SellPlan& plan, const double* aval, const double* mval,
                int nrhs, const double* B, double* X, const dcu_options* opt, int* iters, int* status,
                dcu_solve_info* info) {
  kb_own_columns<<<waves_grid(c, plan.n, 256, 8), 256, 0, c->stream>>>(
      sys_off, nsys, plan.n, plan.off, const_cast<int*>(plan.idx), const_cast<int*>(plan.kd), const_cast<int*>(plan.su));
  DCU_LAUNCHED(c, "kb_own_columns");
  switch (nrhs) {
    case 1: return run_batch<1>(c, nsys, sys_off, plan, aval, mval, B, X, opt, iters, status, info);
    case 2: return run_batch<2>(c, nsys, sys_off, plan, aval, mval, B, X, opt, iters, status, info);
    case 4: return run_batch<4>(c, nsys, sys_off, plan, aval, mval, B, X, opt, iters, status, info);
    case 8: return run_batch<8>(c, nsys, sys_off, plan, aval, mval, B, X, opt, iters, status, info);
    default: return fail(c, DCU_ERR_ARG, "nrhs must be 1, 2, 4 or 8 (got %d)", nrhs);
  }
}

}  // namespace dcu
