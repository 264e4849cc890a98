// One-launch BiCGSTAB for operators small enough to stay on the chip.
//
// The recurrences, stopping rules and scalar updates are those of the kernels
// in bicgstab.cu (K0..K6 there); only where the data lives and how the steps
// are separated differ.  Below a few hundred thousand rows an iteration of five
// kernels is bound by its launches and by dependent loads (64 x 64 grid: 17 us an
// iteration, 512 x 512: 40 us, where the data would take 0.1 and 14 us from
// HBM).  Here every block keeps its rows for the whole solve: the entries of A
// and M in shared memory, the row's r*, r, p, Ay, x in registers.  Only the
// vectors that neighbours gather (r and p - omega Ay, Ay, y / z) leave the
// thread, and the steps of an iteration are separated by five block barriers,
// three of which carry the dot products:
//
//   y = M (r + beta q)          q = p - omega Ay, published with r
//   Ay = A y, (r*, Ay)          -> alpha
//   z = M (r - alpha Ay)
//   Az = A z, (Az, s), (Az, Az) -> omega
//   x, r, q, (r*, r), (r, r)    -> rho, beta, ||r||, stop test
//
// Two forms of one kernel:
//   cluster  up to 16 CTAs of one cluster; the gathered vectors are in shared
//            memory and read through distributed shared memory, the barrier is
//            the cluster's hardware barrier, partial sums are written into
//            every CTA's shared memory before it.  Where the columns are
//            scattered the rows are written to every CTA and gathered locally.
//   grid     one block per SM (a cooperative launch); the gathered vectors are
//            in global memory (L2), the barrier is one tagged slot per block
//            that every block polls (arrival and partial sums in one, no
//            atomics), with an iteration limit; the two barriers without sums
//            wait only for the blocks whose rows are gathered.
// Every block sums the same partials in the same order, so all of them take
// the same decisions without a further exchange, and the result does not
// depend on timing.
//
// Measured on one B200 (whole calls, before -> with this kernel): 64 x 64 grid
// 1.17 -> 0.40 ms, 96 x 96 forward and backward 8.4 -> 3.0 ms, the circuit-like
// matrix of 4510 rows 19.2 -> 7.6 ms (its long rows are no longer a serial chain;
// 3.5 with the faster build and analysis), 256 x 256 4.6 -> 2.8 ms, 512 x 512 adjoint 14.9 ->
// 7.8 ms.  An iteration is now bound by its five barriers: about 1.0 us a step in
// the cluster form (hardware barrier 0.45 us, two block-level sums and one
// remote gather the rest), 2.5 to 3.5 us in the grid form (two fences and two
// trips through L2).
//
// Forms with FP32 search vectors are not taken: their iterates follow every
// rounding of the dot products, which are summed in another order here.
#include <algorithm>

#include "internal.cuh"

namespace dcu {
namespace {

constexpr int kPMaxBlocks = kPersistBlocks;  // grid form
constexpr int kPPoll = kPMaxBlocks / 32;     // slots a lane polls
// Grid form: barrier e uses the slots of set e % kPSlotSets.  A block stores
// its tag over the one of barrier e - kPSlotSets, which every block that polls
// for it must have seen: a barrier of all blocks has to lie strictly between
// the two.  Near barriers wait for some blocks only and never follow each
// other, so of two barriers in a row one is of all blocks: three sets suffice
// (with two, a block past a near barrier may overwrite a tag that a distant
// block still polls for), four make the set a mask.
constexpr int kPSlotSets = 4;
constexpr int kPLong = kPersistLong;  // a longer row of a wide slice is summed by a warp
constexpr int kPSlices = 64;        // slices per block, at most (2048 rows)
constexpr unsigned kPollLimit = 1u << 22;  // polls of one barrier before it gives up (seconds)

enum { P_ERR_TIMEOUT = 1, P_ERR_CAPACITY = 2 };
enum { P_GRID = 0, P_PULL = 1, P_PUSH = 2 };  // the grid form; the cluster form, gathering from or writing to the others

// One block's partial sums at one barrier: each FP64 value as two words of
// 32 bits of it and the barrier's number, so that a word that carries the
// number is whole.
struct alignas(128) PSlot {
  ulonglong2 v[2];
};

struct PArgs {
  int n, nslices, spb, blocks;
  const long long* off;
  const int* su;
  const int* kd;
  const int* ix;
  const int* rptr;
  const double* aval;
  const float* aval32;
  const int* a_inexact;
  const void* mval;
  const void* mval8;
  int mkind;              // 0 double, 1 float, 2 bf16
  const double* b;
  double* x;
  double2* rq;            // grid form: r and q of every row
  double* ay;
  double* yz;             // y, then z (and x for the true residual)
  PSlot* slots;           // grid form: [kPSlotSets][kPMaxBlocks]
  SolveOut* out;
  double tol;
  int tol_mode, maxiter, verify;
  int cap_slots, cap_long;
};

__device__ __forceinline__ unsigned p_smem(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned p_mapa(unsigned addr, unsigned rank) {
  unsigned o;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(o) : "r"(addr), "r"(rank));
  return o;
}
// (volatile, so that they stay between the cluster barriers, which are volatile too)
__device__ __forceinline__ double p_ldc(unsigned addr) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ void p_stc(unsigned addr, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" : : "r"(addr), "d"(v) : "memory");
}
__device__ __forceinline__ void p_cluster_barrier() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Views of the block's dynamic shared memory, the same offsets in every block.
template <typename MT>
struct PSmem {
  double* a;         // [cap_slots] A's entries
  double* r;         // cluster forms: r, q, Ay, y / z of the block's rows (pull) or of all rows (push)
  double* q;
  double* ay;        // (push: q's array; q is last read before Ay is written)
  double* yz;
  double* lval;      // [cap_long] sums of the long rows' segments
  MT* m;             // [cap_slots] M's entries
  unsigned* e;       // [cap_slots] column (pull: shared::cluster address of r[column])
  int* lstart;       // [cap_long] a segment's entries
  int* llen;         // [cap_long]
};

template <typename MT, int FORM>
__host__ __device__ inline size_t p_layout(int cap_slots, int cap_long, int rows, int n, PSmem<MT>* s,
                                           unsigned char* base) {
  size_t o = 0;
  auto take = [&](size_t bytes) {
    const size_t at = o;
    o += (bytes + 15) & ~(size_t)15;
    return at;
  };
  const size_t nr = FORM == P_PULL ? (size_t)rows * 8 : FORM == P_PUSH ? (size_t)n * 8 : 0;
  const size_t oa = take((size_t)cap_slots * 8), orr = take(nr), oq = take(nr);
  const size_t oy = FORM == P_PUSH ? oq : take(nr), oz = take(nr);
  const size_t ol = take((size_t)cap_long * 8), om = take((size_t)cap_slots * sizeof(MT));
  const size_t oe = take((size_t)cap_slots * 4), os = take((size_t)cap_long * 4), on = take((size_t)cap_long * 4);
  if (s) {
    s->a = reinterpret_cast<double*>(base + oa);
    s->r = reinterpret_cast<double*>(base + orr);
    s->q = reinterpret_cast<double*>(base + oq);
    s->ay = reinterpret_cast<double*>(base + oy);
    s->yz = reinterpret_cast<double*>(base + oz);
    s->lval = reinterpret_cast<double*>(base + ol);
    s->m = reinterpret_cast<MT*>(base + om);
    s->e = reinterpret_cast<unsigned*>(base + oe);
    s->lstart = reinterpret_cast<int*>(base + os);
    s->llen = reinterpret_cast<int*>(base + on);
  }
  return o;
}

// Rows [32 spb b, 32 spb (b + 1)) belong to block b, row i of them to thread
// i % PT (PT threads, RPT rows each): a warp holds whole slices, entry k of its 32 rows side by side.
template <typename MT, int PT, int RPT, int FORM>
__global__ void __launch_bounds__(PT, 1) k_bi_persist(PArgs a) {
  constexpr int PW = PT / 32;
  constexpr bool CL = FORM != P_GRID, PULL = FORM == P_PULL, PUSH = FORM == P_PUSH;
  extern __shared__ __align__(16) unsigned char p_raw[];
  __shared__ int sbase[kPSlices + 1];
  __shared__ int slong[2];                 // segments of long rows, their entries
  __shared__ int ticket;                   // next segment to sum
  __shared__ unsigned from[kPPoll];        // grid form: the blocks whose rows this one gathers
  __shared__ double red[2][PW];
  __shared__ double sums[2];               // grid form: the totals
  __shared__ double part[2][2][16];        // cluster form: [parity][sum][rank]
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int bid = blockIdx.x;
  const int rows_pb = a.spb * 32;
  PSmem<MT> S;
  p_layout<MT, FORM>(a.cap_slots, a.cap_long, rows_pb, a.n, &S, p_raw);
  const unsigned base_r = p_smem(S.r);
  const unsigned off_q = p_smem(S.q) - base_r, off_ay = p_smem(S.ay) - base_r, off_yz = p_smem(S.yz) - base_r;
  const int s0 = bid * a.spb, ns = max(0, min(a.spb, a.nslices - s0));
  int err = 0;

  // ---- the block's entries into shared memory -----------------------------
  // A slice keeps all its slots, except one that slice_split names (laid out
  // compactly: entries in row order, padding at the end): its rows longer than
  // kPLong go to the long list, a warp to a row, and the others set its width.
  if (tid < 2) slong[tid] = 0;
  if (tid == 0) ticket = 0;
  if (tid < kPPoll) from[tid] = 0u;
  __syncthreads();
  auto slice_len = [&](int s, int w, bool& split) {  // this lane's row length; whether long rows leave the slice
    const int r = s * 32 + lane;
    const int len = r < a.n ? a.rptr[r + 1] - a.rptr[r] : 0;
    split = slice_split(w, len);
    return len;
  };
  for (int t = wid; t < ns; t += PW) {
    const int s = s0 + t;
    const int w = (int)((a.off[s + 1] - a.off[s]) >> 5);
    bool split;
    const int len = slice_len(s, w, split);
    int wt = w;
    if (split) wt = __reduce_max_sync(0xffffffffu, len <= kPLong ? len : 0);
    if (lane == 0) sbase[t + 1] = wt;
  }
  __syncthreads();
  if (tid == 0) {
    int run = 0;
    sbase[0] = 0;
    for (int t = 0; t < ns; ++t) {
      run += sbase[t + 1];
      sbase[t + 1] = run;
    }
  }
  __syncthreads();
  const int lbase = sbase[ns] * 32;  // the long rows' entries follow the slices
  const bool a32 = a.aval32 && *a.a_inexact == 0;
  // entry k of row r (SELL slot q): its column, A's and M's value
  auto fetch = [&](long long q, int r, int k, int f, long long o0, int& c, double& av, MT& mv) {
    c = (f & 1) ? r + (a.kd[(o0 >> 5) + k] >> 1) : a.ix[q];
    av = a32 ? (double)a.aval32[q] : a.aval[q];
    if (a.mkind == 0) {
      mv = (MT) reinterpret_cast<const double*>(a.mval)[q];
    } else {
      const bool nar = (f & 2) && a.mval8;
      const long long j = nar ? (long long)r * kNarrow + k : q;
      const void* src = nar ? a.mval8 : a.mval;
      mv = (MT)(a.mkind == 1 ? reinterpret_cast<const float*>(src)[j]
                             : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(src)[j]));
    }
  };
  auto put = [&](int dst, int c, double av, MT mv) {
    if (dst >= a.cap_slots) {
      err = P_ERR_CAPACITY;
      return;
    }
    S.a[dst] = av;
    S.m[dst] = mv;
    if (!CL) {
      const int o = c / rows_pb;
      if (!(from[o >> 5] >> (o & 31) & 1u)) atomicOr(&from[o >> 5], 1u << (o & 31));
    }
    S.e[dst] = PULL ? p_mapa(base_r + 8u * (unsigned)(c % rows_pb), (unsigned)(c / rows_pb)) : (unsigned)c;
  };
  int li[RPT];  // a long row's first segment in lval and their number << 16, or -1
#pragma unroll
  for (int j = 0; j < RPT; ++j) {
    li[j] = -1;
    const int t = wid + j * PW;
    if (t >= ns) continue;  // whole warps
    const int s = s0 + t, r = s * 32 + lane;
    const long long o0 = a.off[s];
    const int w = (int)((a.off[s + 1] - o0) >> 5), f = a.su[s];
    const int wt = sbase[t + 1] - sbase[t];
    const int dst0 = sbase[t] * 32 + lane;
    bool split;
    const int len = slice_len(s, w, split);
    const int self = r < a.n ? r : s * 32;
    // slots to take: all of the slice's, or a short row's own; the rest add nothing
    const int cnt = r >= a.n ? 0 : (split ? (len <= kPLong ? len : 0) : w);
    for (int k0 = 0; k0 < wt; k0 += 8) {
      int cv[8];
      double av[8];
      MT mv[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        cv[u] = self;
        av[u] = 0.0;
        mv[u] = (MT)0.f;
        if (k0 + u < cnt) fetch(o0 + 32ll * (k0 + u) + lane, r, k0 + u, f, o0, cv[u], av[u], mv[u]);
      }
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (k0 + u < wt) put(dst0 + 32 * (k0 + u), cv[u], av[u], mv[u]);
    }
    unsigned longs = split ? __ballot_sync(0xffffffffu, len > kPLong) : 0u;
    while (longs) {
      const int jl = __ffs(longs) - 1;
      longs &= longs - 1;
      const int L = __shfl_sync(0xffffffffu, len, jl);
      const int nseg = (L + kPersistSeg - 1) / kPersistSeg;
      int l = 0, st = 0;
      if (lane == 0) {
        l = atomicAdd(&slong[0], nseg);
        st = lbase + atomicAdd(&slong[1], L);
      }
      l = __shfl_sync(0xffffffffu, l, 0);
      st = __shfl_sync(0xffffffffu, st, 0);
      if (l + nseg > a.cap_long) {
        err = P_ERR_CAPACITY;
        continue;
      }
      if (lane == jl) li[j] = l | (nseg << 16);
      for (int g = lane; g < nseg; g += 32) {
        S.lstart[l + g] = st + g * kPersistSeg;
        S.llen[l + g] = min(kPersistSeg, L - g * kPersistSeg);
      }
      for (int k = lane; k < L; k += 32) {
        int cv;
        double av;
        MT mv;
        fetch(o0 + 32ll * k + jl, s * 32 + jl, k, f, o0, cv, av, mv);
        put(st + k, cv, av, mv);
      }
    }
  }
  if (err) atomicOr(&a.out->err, err);
  __syncthreads();
  const int nlong = min(slong[0], a.cap_long);

  // ---- gathers ------------------------------------------------------------
  auto g_r = [&](unsigned e) { return PUSH ? S.r[e] : PULL ? p_ldc(e) : a.rq[e].x; };
  auto g_ay = [&](unsigned e) { return PUSH ? S.ay[e] : PULL ? p_ldc(e + off_ay) : a.ay[e]; };
  auto g_yz = [&](unsigned e) { return PUSH ? S.yz[e] : PULL ? p_ldc(e + off_yz) : a.yz[e]; };
  double beta = 0.0, nalpha = 0.0;
  auto x_p = [&](unsigned e) {  // p at a gathered column
    double rv, qv;
    if (PUSH) {
      rv = S.r[e];
      qv = S.q[e];
    } else if (PULL) {
      rv = p_ldc(e);
      qv = p_ldc(e + off_q);
    } else {
      const double2 t = a.rq[e];
      rv = t.x;
      qv = t.y;
    }
    return rv + beta * qv;
  };
  auto x_s = [&](unsigned e) { return g_r(e) + nalpha * g_ay(e); };
  // this thread's row j: sum over its entries, eight gathers in flight
  auto row_dot = [&](int j, auto vals, auto xf) {
    const int t = wid + j * PW;
    const int o = sbase[t], w = sbase[t + 1] - o;
    const int at = o * 32 + lane;
    double acc = 0.0;
    for (int k0 = 0; k0 < w; k0 += 8) {
      double xv[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) xv[u] = (k0 + u < w) ? xf(S.e[at + 32 * (k0 + u)]) : 0.0;
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (k0 + u < w) acc += (double)vals[at + 32 * (k0 + u)] * xv[u];
    }
    return acc;
  };
  const int row0 = s0 * 32;
  auto row_of = [&](int j) { return row0 + tid + j * PT; };
  auto mine = [&](int j) { return tid + j * PT < ns * 32 && row_of(j) < a.n; };
  // The block's rows: each thread its own, then the long rows' segments of
  // kPersistSeg entries, a warp to a segment, by ticket (warps without rows of
  // their own start there at once); a long row adds its segments in order.
  auto rows_dot = [&](auto vals, auto xf, double (&out)[RPT]) {
    if constexpr (RPT == 2) {
      // both rows' gathers in flight together (four rows: spills, slower)
      int at[2], w[2];
      double acc[2] = {0.0, 0.0};
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int t = wid + i * PW;
        const bool in = mine(i) && li[i] < 0;
        const int o = in ? sbase[t] : 0;
        w[i] = in ? sbase[t + 1] - o : 0;
        at[i] = o * 32 + lane;
      }
      const int wm = max(w[0], w[1]);
      for (int k0 = 0; k0 < wm; k0 += 8) {
        double xv[2][8];
#pragma unroll
        for (int u = 0; u < 8; ++u)
#pragma unroll
          for (int i = 0; i < 2; ++i) xv[i][u] = (k0 + u < w[i]) ? xf(S.e[at[i] + 32 * (k0 + u)]) : 0.0;
#pragma unroll
        for (int u = 0; u < 8; ++u)
#pragma unroll
          for (int i = 0; i < 2; ++i)
            if (k0 + u < w[i]) acc[i] += (double)vals[at[i] + 32 * (k0 + u)] * xv[i][u];
      }
      out[0] = acc[0];
      out[1] = acc[1];
    } else {
#pragma unroll
      for (int j = 0; j < RPT; ++j) out[j] = mine(j) && li[j] < 0 ? row_dot(j, vals, xf) : 0.0;
    }
    if (nlong == 0) return;
    __syncwarp();
    for (;;) {
      int l = 0;
      if (lane == 0) l = atomicAdd(&ticket, 1);
      l = __shfl_sync(0xffffffffu, l, 0);
      if (l >= nlong) break;
      const int st = S.lstart[l], L = S.llen[l];
      double xv[kPersistSeg / 32], acc = 0.0;
#pragma unroll
      for (int u = 0; u < kPersistSeg / 32; ++u) xv[u] = (lane + 32 * u < L) ? xf(S.e[st + lane + 32 * u]) : 0.0;
#pragma unroll
      for (int u = 0; u < kPersistSeg / 32; ++u)
        if (lane + 32 * u < L) acc += (double)vals[st + lane + 32 * u] * xv[u];
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
      if (lane == 0) S.lval[l] = acc;
    }
    __syncthreads();
    if (tid == 0) ticket = 0;
#pragma unroll
    for (int j = 0; j < RPT; ++j)
      if (li[j] >= 0) {
        const int l = li[j] & 0xffff, m = li[j] >> 16;
        for (int g = 0; g < m; ++g) out[j] += S.lval[l + g];
      }
  };

  // ---- barrier with up to two sums -----------------------------------------
  // Returns false when the barrier gave up.  All threads' stores before it are
  // visible to all threads of all blocks after it.
  unsigned ep = 0;
  double tot[2] = {0.0, 0.0};
  // near (grid form, nd = 0): wait only for the blocks whose rows this one
  // gathers.  Nothing they write is overwritten before the next barrier of all
  // blocks, and no slot before such a barrier has passed (kPSlotSets): two near
  // ones never follow each other.
  auto sync = [&](int nd, double v0, double v1, bool near = false) -> bool {
    ++ep;
    if (nd > 0) {
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) {
        v0 += __shfl_xor_sync(0xffffffffu, v0, d);
        if (nd > 1) v1 += __shfl_xor_sync(0xffffffffu, v1, d);
      }
      if (lane == 0) {
        red[0][wid] = v0;
        red[1][wid] = v1;
      }
    }
    if constexpr (CL) {
      const unsigned par = ep & 1u;
      if (nd > 0) {
        __syncthreads();
        if (wid == 0) {
          const int d = lane >> 4, rk = lane & 15;
          double s[PW];
#pragma unroll
          for (int w = 0; w < PW; ++w) s[w] = red[d][w];
#pragma unroll
          for (int h = PW / 2; h > 0; h >>= 1)
#pragma unroll
            for (int w = 0; w < h; ++w) s[w] += s[w + h];
          if (d < nd && rk < a.blocks) p_stc(p_mapa(p_smem(&part[par][d][bid]), (unsigned)rk), s[0]);
        }
      }
      p_cluster_barrier();
      if (nd > 0) {
        // lanes 0-15 the first sum's parts, 16-31 the second's
        double t = (lane & 15) < a.blocks ? part[par][lane >> 4][lane & 15] : 0.0;
#pragma unroll
        for (int h = 8; h > 0; h >>= 1) t += __shfl_xor_sync(0xffffffffu, t, h);
        tot[0] = __shfl_sync(0xffffffffu, t, 0);
        tot[1] = __shfl_sync(0xffffffffu, t, 16);
      }
      return true;
    } else {
      // A slot per block, a 128-byte line each (148 blocks polling slots that
      // share lines take 4.5 us a barrier on one B200, 2.2 us on lines of their
      // own; fences and the two trips through L2 are the rest).
      __syncthreads();
      PSlot* const set = a.slots + (ep % kPSlotSets) * kPMaxBlocks;
      const int nsum = max(nd, 1);
      bool lost = false;
      if (wid == 0) {
        if (lane < nsum) {
          // (sixteen at a time: the sum of 32 warps' parts needs no more registers)
          double s0 = 0.0;
#pragma unroll
          for (int w0 = 0; w0 < PW; w0 += 16) {
            double s[16];
#pragma unroll
            for (int w = 0; w < 16; ++w) s[w] = red[lane][w0 + w];
#pragma unroll
            for (int h = 8; h > 0; h >>= 1)
#pragma unroll
              for (int w = 0; w < h; ++w) s[w] += s[w + h];
            s0 += s[0];
          }
          const unsigned long long u = nd > 0 ? (unsigned long long)__double_as_longlong(s0) : 0ull;
          const unsigned long long lo = (u & 0xffffffffull) | ((unsigned long long)ep << 32);
          const unsigned long long hi = (u >> 32) | ((unsigned long long)ep << 32);
          PSlot* dst = set + bid;
          asm volatile("fence.acq_rel.gpu;" ::: "memory");
          asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" : : "l"(&dst->v[lane]), "l"(lo), "l"(hi)
                       : "memory");
        }
        __syncwarp();
        // (a slot already seen is not read again: 2.0 against 2.6 us of polling)
        double t[2] = {0.0, 0.0}, tv[2][kPPoll];
        unsigned got = 0, polls = 0;
#pragma unroll
        for (int m = 0; m < kPPoll; ++m) {
          tv[0][m] = tv[1][m] = 0.0;
          if (lane + 32 * m >= a.blocks || (near && !(from[m] >> lane & 1u))) got |= 1u << m;
        }
        do {
#pragma unroll
          for (int m = 0; m < kPPoll; ++m) {
            if (got >> m & 1u) continue;
            const PSlot* src = set + lane + 32 * m;
            bool seen = true;
#pragma unroll
            for (int d = 0; d < 2; ++d) {
              if (d >= nsum) break;
              unsigned long long lo, hi;
              asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(lo), "=l"(hi) : "l"(&src->v[d])
                           : "memory");
              seen = seen && (unsigned)(lo >> 32) == ep && (unsigned)(hi >> 32) == ep;
              tv[d][m] = __longlong_as_double((long long)((lo & 0xffffffffull) | (hi << 32)));
            }
            if (seen) got |= 1u << m;
          }
          if (++polls > kPollLimit) lost = true;
        } while (!__all_sync(0xffffffffu, got == (1u << kPPoll) - 1u) && !__any_sync(0xffffffffu, lost));
#pragma unroll
        for (int m = 0; m < kPPoll; ++m) {
          t[0] += tv[0][m];
          t[1] += tv[1][m];
        }
        asm volatile("fence.acq_rel.gpu;" ::: "memory");
        if (nd > 0) {
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            t[0] += __shfl_xor_sync(0xffffffffu, t[0], o);
            if (nd > 1) t[1] += __shfl_xor_sync(0xffffffffu, t[1], o);
          }
          if (lane == 0) {
            sums[0] = t[0];
            sums[1] = t[1];
          }
        }
      }
      if (__syncthreads_or(lost)) return false;
      tot[0] = sums[0];
      tot[1] = sums[1];
      return true;
    }
  };

  // ---- the solve ------------------------------------------------------------
  // push: this row's value into every CTA's copy of the vector
  auto push = [&](double* vec, int row, double v) {
    const unsigned at = p_smem(vec + row);
    for (int k = 0; k < a.blocks; ++k) p_stc(p_mapa(at, (unsigned)k), v);
  };
  auto put_rq = [&](int j, double rv, double qv) {
    if (PUSH) {
      push(S.r, row_of(j), rv);
      push(S.q, row_of(j), qv);
    } else if (PULL) {
      S.r[tid + j * PT] = rv;
      S.q[tid + j * PT] = qv;
    } else {
      a.rq[row_of(j)] = make_double2(rv, qv);
    }
  };
  auto put_ay = [&](int j, double v) {
    if (PUSH) push(S.ay, row_of(j), v);
    else if (PULL) S.ay[tid + j * PT] = v;
    else a.ay[row_of(j)] = v;
  };
  auto put_yz = [&](int j, double v) {
    if (PUSH) push(S.yz, row_of(j), v);
    else if (PULL) S.yz[tid + j * PT] = v;
    else a.yz[row_of(j)] = v;
  };
  double r[RPT], p[RPT], ay[RPT], x[RPT], y[RPT], z[RPT];
  double rs[RPT];
  double rho = 0.0, alpha = 0.0, omega = 1.0, res = 0.0, thr = 0.0, bnorm = 0.0, true_res = -1.0;
  int it = 1, status = -1, replacements = 0;
  // Every block has started (its shared memory can be read) and loaded its
  // entries.  (The host sizes the buffers by the rules used here; were they
  // exceeded in one block, every block would stop before the first product.)
  bool ok = sync(0, 0.0, 0.0);
  ok = ok && *(volatile const int*)&a.out->err == 0;
  // v[j] = b - A x with x published in yz; sums (r*, v), (v, v) and (b, b)
  double bb = 0.0;
  auto residual = [&](double (&v)[RPT], bool first) -> bool {
#pragma unroll
    for (int j = 0; j < RPT; ++j)
      if (mine(j)) put_yz(j, x[j]);
    if (!sync(0, 0.0, 0.0, true)) return false;
    rows_dot(S.a, g_yz, v);
    double d0 = 0.0, d1 = 0.0;
    bb = 0.0;
#pragma unroll
    for (int j = 0; j < RPT; ++j) {
      if (!mine(j)) continue;
      const double br = a.b[row_of(j)];
      v[j] = br - v[j];
      if (first) rs[j] = v[j];
      d0 += rs[j] * v[j];
      d1 += v[j] * v[j];
      bb += br * br;
    }
    return sync(2, d0, d1);
  };
#pragma unroll
  for (int j = 0; j < RPT; ++j) {
    x[j] = mine(j) ? a.x[row_of(j)] : 0.0;
    p[j] = ay[j] = y[j] = z[j] = 0.0;
    rs[j] = 0.0;
  }
  ok = ok && residual(r, true);
  if (ok) {
    rho = tot[0];
    res = sqrt(tot[1]);
#pragma unroll
    for (int j = 0; j < RPT; ++j)
      if (mine(j)) put_rq(j, r[j], 0.0);
    ok = sync(1, bb, 0.0);
    bnorm = sqrt(tot[0]);
    thr = a.tol_mode == DCU_TOL_REL ? a.tol * bnorm : a.tol;
    if (res == 0.0) status = DCU_SOLVE_CONVERGED;  // x0 already solves the system
    else if (a.maxiter <= 1) status = DCU_SOLVE_MAXITER;
  }
  while (ok && status < 0) {
    // y = M p
    rows_dot(S.m, x_p, y);
#pragma unroll
    for (int j = 0; j < RPT; ++j) {
      if (!mine(j)) continue;
      const double qv = p[j] - omega * ay[j];
      p[j] = r[j] + beta * qv;
      put_yz(j, y[j]);
    }
    if (!(ok = sync(0, 0.0, 0.0, true))) break;
    // Ay, alpha
    double d0 = 0.0, d1 = 0.0;
    rows_dot(S.a, g_yz, ay);
#pragma unroll
    for (int j = 0; j < RPT; ++j) {
      if (!mine(j)) continue;
      put_ay(j, ay[j]);
      d0 += rs[j] * ay[j];
    }
    if (!(ok = sync(1, d0, 0.0))) break;
    alpha = rho / tot[0];
    if (tot[0] == 0.0 || !isfinite(alpha)) {
      status = DCU_SOLVE_BREAKDOWN;
      break;
    }
    // s = r - alpha Ay (kept in r), z = M s
    nalpha = -1.0 * alpha;
    rows_dot(S.m, x_s, z);
#pragma unroll
    for (int j = 0; j < RPT; ++j) {
      if (!mine(j)) continue;
      r[j] = r[j] + nalpha * ay[j];
      put_yz(j, z[j]);
    }
    if (!(ok = sync(0, 0.0, 0.0, true))) break;
    // Az, omega
    d0 = d1 = 0.0;
    double az[RPT];
    rows_dot(S.a, g_yz, az);
#pragma unroll
    for (int j = 0; j < RPT; ++j) {
      if (!mine(j)) continue;
      d0 += az[j] * r[j];
      d1 += az[j] * az[j];
    }
    if (!(ok = sync(2, d0, d1))) break;
    omega = tot[1] == 0.0 ? 0.0 : tot[0] / tot[1];
    if (!isfinite(omega)) {
      status = DCU_SOLVE_BREAKDOWN;
      break;
    }
    // x, r, q
    const double nomega = -1.0 * omega;
    d0 = d1 = 0.0;
#pragma unroll
    for (int j = 0; j < RPT; ++j) {
      if (!mine(j)) continue;
      x[j] = x[j] + alpha * y[j];
      x[j] = x[j] + omega * z[j];
      const double rn = r[j] + nomega * az[j];
      d0 += rs[j] * rn;
      d1 += rn * rn;
      r[j] = rn;
      put_rq(j, rn, p[j] - omega * ay[j]);
    }
    if (!(ok = sync(2, d0, d1))) break;
    const double rho_new = tot[0];
    beta = (rho_new / rho) * (alpha / omega);
    rho = rho_new;
    res = sqrt(tot[1]);
    if (!isfinite(res)) {
      status = DCU_SOLVE_BREAKDOWN;
    } else if (res < thr) {
      if (!a.verify) {
        status = DCU_SOLVE_CONVERGED;
        break;
      }
      // the true residual: stop, or continue from it (residual replacement)
      if (!(ok = residual(r, false))) break;
      true_res = sqrt(tot[1]);
      if (true_res < thr) {
        status = DCU_SOLVE_CONVERGED;
      } else {
        rho = tot[0];
        res = true_res;
        ++replacements;
        if (++it >= a.maxiter) {
          status = DCU_SOLVE_MAXITER;
        } else {
#pragma unroll
          for (int j = 0; j < RPT; ++j)
            if (mine(j)) put_rq(j, r[j], p[j] - omega * ay[j]);
          if (!(ok = sync(0, 0.0, 0.0))) break;
        }
      }
    } else if (!isfinite(beta) || rho_new == 0.0) {
      status = DCU_SOLVE_BREAKDOWN;
    } else if (++it >= a.maxiter) {
      status = DCU_SOLVE_MAXITER;
    }
  }
  if (ok && true_res < 0.0) {
    ok = residual(z, false);
    true_res = sqrt(tot[1]);
  }
#pragma unroll
  for (int j = 0; j < RPT; ++j)
    if (mine(j)) a.x[row_of(j)] = x[j];
  if (tid == 0) {
    if (!ok) atomicOr(&a.out->err, P_ERR_TIMEOUT);
    if (bid == 0) {
      a.out->res = res;
      a.out->true_res = true_res;
      a.out->bnorm = bnorm;
      a.out->it = it;
      a.out->status = status;
      a.out->replacements = replacements;
      a.out->a32 = a32 ? 1 : 0;
    }
  }
  if constexpr (CL) p_cluster_barrier();  // no CTA leaves while another may still read its shared memory
}

// *ran stays false when the device cannot hold all the blocks at once.
template <typename MT, int PT, int RPT, int FORM>
int p_launch(Ctx* c, PArgs& a, size_t smem, bool* ran) {
  constexpr bool CL = FORM != P_GRID;
  auto kernel = k_bi_persist<MT, PT, RPT, FORM>;
  DCU_CUDA(c, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(a.blocks);
  cfg.blockDim = dim3(PT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = c->stream;
  cudaLaunchAttribute at[1];
  if (CL) {
    if (a.blocks > 8) DCU_CUDA(c, cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = a.blocks;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
  } else {
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
  }
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int fit = 0;
  if (CL) {
    if (cudaOccupancyMaxActiveClusters(&fit, kernel, &cfg) != cudaSuccess) fit = 0;
  } else {
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, kernel, PT, smem) != cudaSuccess) fit = 0;
    fit = (long long)fit * c->sms >= a.blocks ? 1 : 0;
  }
  if (fit < 1) {
    cudaGetLastError();
    return DCU_OK;
  }
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, a);
  if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorLaunchOutOfResources) {
    cudaGetLastError();
    return DCU_OK;
  }
  if (e != cudaSuccess) return cuda_fail(c, e, "k_bi_persist", __FILE__, __LINE__);
  c->launches++;
  *ran = true;
  return DCU_OK;
}

template <typename MT>
int p_dispatch(Ctx* c, PArgs& a, size_t smem, int form, bool* ran) {
  const int rows = a.spb * 32;
  if (form == P_PUSH) return p_launch<MT, 512, 1, P_PUSH>(c, a, smem, ran);
  if (form == P_PULL)
    return rows <= 512 ? p_launch<MT, 512, 1, P_PULL>(c, a, smem, ran) : p_launch<MT, 512, 2, P_PULL>(c, a, smem, ran);
  // (1024 threads hold 64 registers each and spill: 512 x 512 took 11.7 against 10.9 ms)
  if (rows <= 512) return p_launch<MT, 512, 1, P_GRID>(c, a, smem, ran);
  if (rows <= 1024) return p_launch<MT, 512, 2, P_GRID>(c, a, smem, ran);
  return p_launch<MT, 512, 4, P_GRID>(c, a, smem, ran);
}

template <typename MT>
size_t p_bytes(int form, int cap_slots, int cap_long, int rows, int n) {
  return form == P_PUSH   ? p_layout<MT, P_PUSH>(cap_slots, cap_long, rows, n, nullptr, nullptr)
         : form == P_PULL ? p_layout<MT, P_PULL>(cap_slots, cap_long, rows, n, nullptr, nullptr)
                          : p_layout<MT, P_GRID>(cap_slots, cap_long, rows, n, nullptr, nullptr);
}

// Static shared memory of the kernel, rounded up, and the runtime's own.
constexpr size_t kPStatic = 4096;

}  // namespace

PersistShape persist_shape(const Ctx* c, int n, bool second) {
  PersistShape s;
  const int nslices = (n + 31) / 32;
  int k = 1;
  const bool one_cluster = nslices <= 16 * 32;
  // (below 13 blocks of 512 rows the grid form is no faster than the cluster's 16
  // CTAs: circuit-like matrix of 5600 rows, FP64, 5.08 against 4.96 ms; random
  // columns, 7000 rows, 0.62 against 0.70)
  if (second && (!one_cluster || nslices <= 192)) return s;
  // cluster form: up to 16 CTAs of up to 1024 rows; fewer CTAs while 256 rows each
  if (one_cluster && !second) {
    while (k < 16 && (nslices + k - 1) / k > 8) k <<= 1;
    s.cluster = true;
    s.spb = (nslices + k - 1) / k;
  } else {
    const int g = std::min(c->sms, kPMaxBlocks);
    s.cluster = false;
    // 512 rows a block at least: fewer blocks to wait for (256 x 256 grid, 128
    // against 147 blocks: 3.33 -> 3.14 ms; 150 x 150, 44 against 141: 2.01 -> 1.66)
    s.spb = std::max(16, (nslices + g - 1) / g);
  }
  // (a cluster's size stays a power of two: its last blocks may hold no rows)
  s.blocks = s.cluster ? k : (nslices + s.spb - 1) / s.spb;
  if (s.spb > kPSlices) s.blocks = 0;
  return s;
}

int persist_solve(Ctx* c, const SellPlan& plan, const SellA& aval, const void* mval, const void* mval8, int mkind,
                  const double* b, double* x, const dcu_options* opt, bool* ran, SolveOut* out) {
  *ran = false;
  PersistShape sh = persist_shape(c, plan.n);
  if (sh.blocks <= 0 || plan.max_block_slots[0] <= 0) return DCU_OK;
  PArgs a{};
  int rows = 0;
  auto take = [&](int shape) {
    a.cap_slots = plan.max_block_slots[shape];
    a.cap_long = plan.max_block_long[shape];
    rows = sh.spb * 32;
  };
  take(0);
  auto bytes = [&](int form) {
    return kPStatic + (mkind == 0 ? p_bytes<double>(form, a.cap_slots, a.cap_long, rows, plan.n)
                                  : p_bytes<float>(form, a.cap_slots, a.cap_long, rows, plan.n));
  };
  // Scattered columns (fewer than half the slots in slices of one offset a
  // position): a gather of 32 scattered elements through distributed shared
  // memory goes lane by lane, so each row is written to every CTA instead and
  // gathered locally, where the whole vectors fit.  Else, where a third of the
  // entries lie in another CTA's rows (or the cluster does not hold the
  // operator), through L2 in the grid form.  Random columns, 5 a row, BF16 M, whole
  // calls, launches / pull / grid: 10000 rows 1.18 / 0.95 / 0.72 ms, 14000 0.95 /
  // 1.12 / 0.70; columns within 300 rows (12000 rows, a fifth remote) pull / grid
  // 0.51 / 0.56, within 1200 (two thirds) 0.79 / 0.67.
  int form = sh.cluster ? P_PULL : P_GRID;
  if (sh.cluster && 2 * plan.uniform_slots < plan.slots) {
    if (rows <= 512 && bytes(P_PUSH) <= c->smem_optin) {
      form = P_PUSH;
    } else {
      const PersistShape first = sh;
      const bool holds = bytes(P_PULL) <= c->smem_optin;
      if (!holds || 3ll * plan.remote >= plan.nnz) {
        sh = persist_shape(c, plan.n, true);
        take(1);
        form = P_GRID;
        if (bytes(form) > c->smem_optin) {
          sh = first;
          take(0);
          form = P_PULL;
        }
      }
    }
  }
  if (bytes(form) > c->smem_optin) return DCU_OK;
  const size_t smem = bytes(form) - kPStatic;
  auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
  const size_t nslot = form != P_GRID ? 0 : sizeof(PSlot) * kPSlotSets * kPMaxBlocks;
  const size_t vec = al(sizeof(double) * (size_t)plan.n);
  // (without room for its vectors the solve goes to the launches)
  if (!ensure_optional(c, B_PERSIST, al(sizeof(SolveOut)) + nslot + (form == P_GRID ? 4 * vec : 0))) return DCU_OK;
  char* base = bp<char>(c, B_PERSIST);
  a.n = plan.n;
  a.nslices = plan.nslices;
  a.spb = sh.spb;
  a.blocks = sh.blocks;
  a.off = plan.off;
  a.su = plan.su;
  a.kd = plan.kd;
  a.ix = plan.idx;
  a.rptr = plan.rptr;
  a.aval = aval.v64;
  a.aval32 = aval.v32;
  a.a_inexact = aval.inexact;
  a.mval = mval;
  a.mval8 = mval8;
  a.mkind = mkind;
  a.b = b;
  a.x = x;
  a.out = reinterpret_cast<SolveOut*>(base);
  a.slots = reinterpret_cast<PSlot*>(base + al(sizeof(SolveOut)));
  char* v = base + al(sizeof(SolveOut)) + nslot;
  a.rq = reinterpret_cast<double2*>(v);
  a.ay = reinterpret_cast<double*>(v + 2 * vec);
  a.yz = reinterpret_cast<double*>(v + 3 * vec);
  a.tol = opt->tol;
  a.tol_mode = opt->tol_mode;
  a.maxiter = opt->maxiter > 0 ? opt->maxiter : plan.n;
  a.verify = opt->verify;
  DCU_CUDA(c, cudaMemsetAsync(base, 0, al(sizeof(SolveOut)) + nslot, c->stream));
  DCU_TRY(mkind == 0 ? p_dispatch<double>(c, a, smem, form, ran) : p_dispatch<float>(c, a, smem, form, ran));
  if (!*ran) return DCU_OK;
  DCU_CUDA(c, cudaEventRecord(c->ev[1], c->stream));
  DCU_CUDA(c, cudaMemcpyAsync(c->pinned, a.out, sizeof(SolveOut), cudaMemcpyDeviceToHost, c->stream));
  DCU_CUDA(c, cudaStreamSynchronize(c->stream));
  std::memcpy(out, c->pinned, sizeof(SolveOut));
  if (out->err) return fail(c, DCU_ERR_CUDA, "the one-launch solver did not finish (%d)", out->err);
  return DCU_OK;
}

}  // namespace dcu
