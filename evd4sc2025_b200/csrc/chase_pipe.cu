// Stage 2, band -> tridiagonal: the chase as a systolic pipeline over the band.
//
// Same reflectors and the same storage as chase_kernel (bulge_chase.cu; the
// reference's chasing_kernel_one_timeV10, util/inc/bugle_chasingV10.h:21-392),
// with the work cut the other way: a place on the band owns its data and the
// sweeps pass through it, where chase_kernel gives a sweep to a CTA that drags
// its tiles through global memory.
//
// Slot k holds the 32 columns r .. r+31, r = s + 1 + 32 k, of sweep s: the
// diagonal block S and the block N below it (rows r+32 .. r+63).  Its task for
// sweep s, given the reflector u of rows r .. r+31:
//   w = N u,  y = S u                     (old values)
//   x = N(:,0) - w u_0  ->  u' = house(x) (the reflector of rows r+32 .. r+63)
//   N <- H(u') N H(u),  S <- H(u) S H(u)
// u' goes to slot k+1.  The window then slides by one column: the first column
// (S(:,0) and the one nonzero of N(:,0)) goes to slot k-1, one column arrives
// from slot k+1, and N's first row becomes S's new row.  Slot 0's first column
// goes to the head warp, which writes (d, e) of that column and starts the
// next sweep.
//
// What bounds it: the cycle (s, k) -> u' -> (s, k+1) -> column -> (s+1, k), two
// half-tasks and two messages per sweep, n - 2 times.  So a slot is two warps,
// one for N and one for S, a lane per row with the row in registers: w, y and
// x need no other lane, the critical part of a task is 32 products, one warp
// sum and two reciprocal roots, and no barrier stands in it.  (With a slot as
// 128 threads, four to a row, the same cycle took 2.4 us: two CTA-level sums
// through shared memory and a barrier cost more than the longer dot product.)
// The updates of S and N run after the messages have left, while the slot
// waits.  Rows stay in the lane of their number mod 32; columns are shifted by
// one register in the update itself.  Messages carry their flag in every
// 8-byte word (half a double + the sweep number), so one store and one polled
// load pass data with no fence.  Between slots of a CTA they go through shared
// memory, between CTAs of a cluster through distributed shared memory,
// otherwise through global memory and a relay warp of the receiving CTA.
// Measured figures: at launch_chase_pipe, where the form is chosen.
//
// Progress: every slot waits for both neighbours, so all CTAs of a launch must
// be resident together.  One CTA and one cluster (co-scheduled by definition)
// are.  A cooperative launch fits the device, but other kernels may hold the SMs
// of some of its CTAs for any time (a long kernel on another stream, or two such
// launches of different priority, each with a part of the SMs).  So its CTAs
// first count themselves in at a gate; if they are not complete after 2 s the
// gate shuts, all of them leave, and the ticketed kernel behind them, whose
// progress asks for no residency, does the sweeps.  Every wait is bounded.
#include <cooperative_groups.h>

#include <mutex>

#include "common.cuh"

namespace evd {

namespace {

namespace cg = cooperative_groups;

constexpr int kPB = 32;              // band width
constexpr int kPOff = 2 * kPB;       // band-storage rows per column
constexpr int kSlotThreads = 64;     // a warp for N, a warp for S
constexpr int kExtraWarps = 3;       // head, u relay, column relay
constexpr unsigned long long kPipeTimeoutNs = 4000000000ull;  // 4 s
constexpr unsigned long long kGateNs = 2000000000ull;         // 2 s
typedef unsigned long long u64;

struct __align__(16) Word2 {
  u64 lo, hi;  // (flag << 32) | half of the double
};

// Slot k has a task in sweep s while its window's first row r = s + 1 + 32 k is
// a row of the matrix.  Every task waits for the reflector message of its
// sweep, also the last one (r = n - 1), which has nothing to reflect and gets a
// zero: that message is what orders a slot's two warps and its neighbours.
// u(s) to slot k is sent by slot k-1 after it has read c(s-1), which S(k) sent
// after it had read u(s-1) and the row of sweep s-2; so whoever holds u(s) may
// write over everything that was two sweeps old.
__host__ __device__ constexpr int last_sweep(int n, int s1, int k) {
  return s1 - 1 < n - 2 - kPB * k ? s1 - 1 : n - 2 - kPB * k;
}
__host__ __device__ constexpr bool has_next_slot(int n, int r) { return r + kPB <= n - 1; }
// its column r + 31 exists: a column message of the sweep before comes too
__host__ __device__ constexpr bool takes_column(int n, int r) { return r + kPB - 1 <= n - 1; }

// A slot's inbox: reflector and column messages, two sweeps deep (a sender can
// be at most one sweep ahead of the last message its receiver has read).
// Entry 32 of a column is its diagonal element; entry (c mod 32) of column c
// is its element in row c + 32, entry (row mod 32) the ones between.
struct Inbox {
  Word2 u[2][kPB];
  Word2 c[2][kPB + 1];
};

// The messages that cross one CTA boundary of a cooperative launch.
struct Boundary {
  Word2 u[2][kPB];
  Word2 c[2][kPB + 1];
};

struct SlotSmem {
  Inbox in;
  __align__(16) double un[kPB], us[kPB];  // u, first column first, for each warp
  __align__(16) double z[kPB], v[kPB];
  __align__(16) double row[2][kPB];       // N's leaving first row, N warp -> S warp
  int row_flag[2];                        // its sweep + 1
};

__device__ __forceinline__ unsigned smem_u32(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ Word2 pack(double v, unsigned flag) {
  const u64 f = (u64)flag << 32;
  return Word2{f | (unsigned)__double2loint(v), f | (unsigned)__double2hiint(v)};
}
__device__ __forceinline__ double unpack(const Word2& w) {
  return __hiloint2double((int)(unsigned)w.hi, (int)(unsigned)w.lo);
}
__device__ __forceinline__ bool has(const Word2& w, unsigned flag) {
  return (unsigned)(w.lo >> 32) == flag && (unsigned)(w.hi >> 32) == flag;
}
__device__ __forceinline__ Word2 ld_sh(const Word2* p) {
  Word2 w;
  asm volatile("ld.volatile.shared.v2.u64 {%0, %1}, [%2];"
               : "=l"(w.lo), "=l"(w.hi)
               : "r"(smem_u32(p))
               : "memory");
  return w;
}
__device__ __forceinline__ void st_sh(Word2* p, const Word2& w) {
  asm volatile("st.volatile.shared.v2.u64 [%0], {%1, %2};" ::"r"(smem_u32(p)), "l"(w.lo),
               "l"(w.hi)
               : "memory");
}
// generic address: another CTA's shared memory (same cluster) or global memory
__device__ __forceinline__ Word2 ld_any(const Word2* p) {
  Word2 w;
  asm volatile("ld.relaxed.gpu.v2.u64 {%0, %1}, [%2];"
               : "=l"(w.lo), "=l"(w.hi)
               : "l"(p)
               : "memory");
  return w;
}
__device__ __forceinline__ void st_any(Word2* p, const Word2& w) {
  asm volatile("st.relaxed.gpu.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(w.lo), "l"(w.hi)
               : "memory");
}
// Bounded waiting: true once the wait has lasted too long or another CTA has
// raised the error word (called every 256 polls; warp-uniform).
struct Patience {
  u64 t0 = 0;
  __device__ bool over(int* err) {
    int bad = 0;
    if ((threadIdx.x & 31) == 0) {
      u64 t;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
      if (t0 == 0) t0 = t;
      if (*(volatile int*)err != 0) {
        bad = 1;
      } else if (t - t0 > kPipeTimeoutNs) {
        atomicCAS(err, 0, kDevTimeoutChase);
        bad = 1;
      }
    }
    return __shfl_sync(0xffffffffu, bad, 0) != 0;
  }
};

// The one loop that every wait of a warp runs in: all lanes leave it in the same
// turn, as the full-mask shuffle of over() needs.
template <typename Ready>
__device__ __forceinline__ bool wait_warp(int* err, Ready ready) {
  Patience pat;
  for (unsigned it = 1; !__all_sync(0xffffffffu, ready()); ++it)
    if ((it & 255u) == 0 && pat.over(err)) return false;
  return true;
}

// Warp-wide wait for a message of 32 entries (and a 33rd): lane l polls entry l.
template <bool SHARED, bool DIAG>
__device__ __forceinline__ bool wait_msg(const Word2* m, unsigned flag, int* err, Word2& mine,
                                         Word2& diag) {
  const int lane = threadIdx.x & 31;
  return wait_warp(err, [&] {
    mine = SHARED ? ld_sh(m + lane) : ld_any(m + lane);
    bool good = has(mine, flag);
    if (DIAG) {
      diag = SHARED ? ld_sh(m + kPB) : ld_any(m + kPB);
      good = good && has(diag, flag);
    }
    return good;
  });
}

// Both messages of a task in one loop (a wait costs 200 cycles even when the
// message is there): entry l of the reflector, and of the column entry l, or
// its diagonal only.
template <bool DIAG>
__device__ __forceinline__ bool wait_both(const Word2* u, unsigned fu, const Word2* c, unsigned fc,
                                          int* err, Word2& mu, Word2& mc) {
  const int lane = threadIdx.x & 31;
  return wait_warp(err, [&] {
    mu = ld_sh(u + lane);
    mc = ld_sh(DIAG ? c + kPB : c + lane);
    return has(mu, fu) && has(mc, fc);
  });
}

struct PipeArgs {
  int n, s0, s1;  // sweeps [s0, s1), s1 <= n - 2
  double* sub;
  double* U;
  long ldU;
  int* err;
  Boundary* bnd;  // gridDim.x - 1 of them (cooperative launch), or nullptr (cluster)
  int* gate;      // of a cooperative launch
};

// Thread 0 of every CTA of a cooperative launch: true once all have come.  The
// word holds their number; it is shut by a compare-and-swap on an incomplete
// number, so all CTAs get the same answer.
__device__ bool pass_gate(int* gate) {
  atomicAdd(gate, 1);
  u64 t0 = 0, t;
  for (unsigned it = 1;; ++it) {
    const int v = ld_acquire(gate);
    if (v & kGateShut) return false;
    if (v == (int)gridDim.x) return true;
    if ((it & 255u) != 0) continue;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    if (t0 == 0) t0 = t;
    if (t - t0 > kGateNs) atomicCAS(gate, v, v | kGateShut);
  }
}

// The reflector of x (rows at and below the first one): u (this lane's entry),
// its first entry and the element that replaces x_0.  x0 and nrm2 are uniform.
__device__ __forceinline__ double house(double x, bool first, double x0, double nrm2, double& u0,
                                        double& beta) {
  const double rn = rsqrt(nrm2);
  const double a0 = x0 * rn;
  const double sg = (a0 >= 0.0) ? 1.0 : -1.0;
  const double a0n = a0 + sg;
  const double s2 = rsqrt(fabs(a0n));
  u0 = a0n * s2;
  beta = -sg * (nrm2 * rn);
  return first ? u0 : (x * rn) * s2;
}

// Where a slot's messages go: this CTA's shared memory or a generic pointer.
struct Dest {
  Word2* p;
  bool local;
  __device__ __forceinline__ void put(int at, double v, unsigned flag) const {
    const Word2 w = pack(v, flag);
    if (local) st_sh(p + at, w);
    else st_any(p + at, w);
  }
};
template <int SL>
__device__ __forceinline__ Dest dest_u(const PipeArgs& a, SlotSmem* slots, int g, bool cluster) {
  if (g + 1 < SL) return Dest{slots[g + 1].in.u[0], true};
  if (blockIdx.x + 1 >= gridDim.x) return Dest{nullptr, false};
  return Dest{cluster ? cg::this_cluster().map_shared_rank(slots[0].in.u[0], blockIdx.x + 1)
                      : a.bnd[blockIdx.x].u[0],
              false};
}
template <int SL>
__device__ __forceinline__ Dest dest_c(const PipeArgs& a, SlotSmem* slots, Word2* headbox, int g,
                                       bool cluster) {
  if (g > 0) return Dest{slots[g - 1].in.c[0], true};
  if (blockIdx.x == 0) return Dest{headbox, true};
  return Dest{cluster ? cg::this_cluster().map_shared_rank(slots[SL - 1].in.c[0], blockIdx.x - 1)
                      : a.bnd[blockIdx.x - 1].c[0],
              false};
}

// Element j of a 32-long vector in shared memory, read two at a time.
__device__ __forceinline__ double2 pair_of(const double* v, int j) {
  return *reinterpret_cast<const double2*>(v + j);
}

// The N warp of slot k: lane l holds the row of N whose number is l mod 32.
template <int SL>
__device__ __forceinline__ void run_n(const PipeArgs& a, SlotSmem& sm, const Dest du,
                                      const Dest dc, int k) {
  const int lane = threadIdx.x & 31;
  const int n = a.n;
  int r = a.s0 + 1 + kPB * k;
  double N[kPB];  // columns r .. r+31
  {
    const int li = (lane - (a.s0 + 1)) & 31;
#pragma unroll
    for (int j = 0; j < kPB; ++j)
      N[j] = (r + kPB + li < n) ? a.sub[(long)(r + j) * kPOff + (kPB + li - j)] : 0.0;
  }
  const int last = last_sweep(n, a.s1, k);
  for (int s = a.s0; s <= last; ++s, ++r) {
    const int rho = (s + 1) & 31;  // lane of N's first row
    const int li = (lane - rho) & 31;
    const bool next_real = r + kPB <= n - 2;  // a reflector of two rows or more
    const int par = s & 1;
    const unsigned flag = (unsigned)(s + 1);
    Word2 m, dm;
    if (s > a.s0 && takes_column(n, r)) {
      if (!wait_both<false>(sm.in.u[par], flag, sm.in.c[par ^ 1], (unsigned)s, a.err, m, dm))
        return;
      N[kPB - 1] = unpack(dm);
    } else {
      if (s > a.s0) N[kPB - 1] = 0.0;
      if (!wait_msg<true, false>(sm.in.u[par], flag, a.err, m, dm)) return;
    }
    const double u = unpack(m);
    sm.un[li] = u;
    __syncwarp();
    double w0 = 0.0, w1 = 0.0, w2 = 0.0, w3 = 0.0;
#pragma unroll
    for (int j = 0; j < kPB; j += 4) {
      const double2 ua = pair_of(sm.un, j), ub = pair_of(sm.un, j + 2);
      w0 = fma(N[j], ua.x, w0);
      w1 = fma(N[j + 1], ua.y, w1);
      w2 = fma(N[j + 2], ub.x, w2);
      w3 = fma(N[j + 3], ub.y, w3);
    }
    const double w = (w0 + w1) + (w2 + w3);
    const double x = fma(-w, sm.un[0], N[0]);
    const double x0 = __shfl_sync(0xffffffffu, x, rho);
    const double nrm2 = warp_sum_tc(x * x);
    double up = 0.0, up0 = 0.0, beta = x0;
    if (next_real && nrm2 > 0.0) up = house(x, lane == rho, x0, nrm2, up0, beta);
    if (has_next_slot(n, r)) {
      du.put(par * kPB + lane, up, flag);
      const int row = r + kPB + li;
      if (next_real && a.U != nullptr && row < n) a.U[row + (long)s * a.ldU] = up;
    }
    if (s < a.s1 - 1 && lane == rho) dc.put(par * (kPB + 1) + rho, beta, flag);
    // ---- off the critical cycle: N <- N - w u^T, z = N^T u', N <- N - u' z^T,
    // written one column to the left (the first column has left) ----
    double q[16];
#pragma unroll
    for (int j = 0; j < kPB; j += 2) {
      const double2 uj = pair_of(sm.un, j);
      N[j] = fma(-w, uj.x, N[j]);
      N[j + 1] = fma(-w, uj.y, N[j + 1]);
    }
    // z: reduce-scatter over the lanes, lane j ends with z_j
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const double lo = up * N[j], hi = up * N[j + 16];
      const bool up16 = lane & 16;
      q[j] = (up16 ? hi : lo) + __shfl_xor_sync(0xffffffffu, up16 ? lo : hi, 16);
    }
#pragma unroll
    for (int h = 8; h > 0; h >>= 1) {
      const bool b = lane & h;
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (j < h)
          q[j] = (b ? q[j + h] : q[j]) + __shfl_xor_sync(0xffffffffu, b ? q[j] : q[j + h], h);
    }
    sm.z[lane] = q[0];
    __syncwarp();
    {
      double2 zj = pair_of(sm.z, 0);
      N[0] = fma(-up, zj.y, N[1]);
#pragma unroll
      for (int j = 2; j < kPB; j += 2) {
        zj = pair_of(sm.z, j);
        N[j - 1] = fma(-up, zj.x, N[j]);
        N[j] = fma(-up, zj.y, N[j + 1]);
      }
    }
    if (s == a.s1 - 1) {  // this launch's last sweep: back to the band
      if (r + kPB + li < n) {
        double* p = a.sub + (long)r * kPOff + kPB + li;
        p[0] = (li == 0) ? beta : 0.0;
#pragma unroll
        for (int j = 1; j < kPB; ++j) p[(long)j * (kPOff - 1)] = N[j - 1];
      }
    } else if (s < last) {
      // the first row leaves for S; its lane takes the new last row (empty but
      // for the column that the next message brings)
      if (lane == rho) {
        double2* row = reinterpret_cast<double2*>(sm.row[par]);
#pragma unroll
        for (int j = 0; j < kPB; j += 2) row[j / 2] = make_double2(N[j], N[j + 1]);
      }
#pragma unroll
      for (int j = 0; j < kPB - 1; ++j) N[j] = (lane == rho) ? 0.0 : N[j];
      __syncwarp();
      __threadfence_block();
      if (lane == 0) *(volatile int*)&sm.row_flag[par] = (int)flag;
    }
  }
}

// The S warp of slot k: lane l holds the row of S whose number is l mod 32.
template <int SL>
__device__ __forceinline__ void run_s(const PipeArgs& a, SlotSmem& sm, const Dest dc, int k) {
  const int lane = threadIdx.x & 31;
  const int n = a.n;
  int r = a.s0 + 1 + kPB * k;
  double S[kPB];  // columns r .. r+31
  {
    const int li = (lane - (a.s0 + 1)) & 31;
#pragma unroll
    for (int j = 0; j < kPB; ++j) {
      const int hi = max(li, j), lo = min(li, j);
      S[j] = (r + hi < n) ? a.sub[(long)(r + lo) * kPOff + (hi - lo)] : 0.0;
    }
  }
  const int last = last_sweep(n, a.s1, k);
  for (int s = a.s0; s <= last; ++s, ++r) {
    const int rho = (s + 1) & 31;
    const int li = (lane - rho) & 31;
    const int par = s & 1;
    const unsigned flag = (unsigned)(s + 1);
    Word2 m, dm;
    if (s > a.s0) {
      // the row that left N in the last sweep is row and column r + 31 now
      if (!wait_warp(a.err, [&] { return *(volatile int*)&sm.row_flag[par ^ 1] == s; })) return;
      __threadfence_block();
      const double* row = sm.row[par ^ 1];
#pragma unroll
      for (int j = 0; j < kPB - 2; j += 2) {
        const double2 e = pair_of(row, j);
        S[j] = (li == 31) ? e.x : S[j];
        S[j + 1] = (li == 31) ? e.y : S[j + 1];
      }
      S[kPB - 2] = (li == 31) ? row[kPB - 2] : S[kPB - 2];
      S[kPB - 1] = (li == 31) ? 0.0 : row[li];
    }
    if (s > a.s0 && takes_column(n, r)) {
      if (!wait_both<true>(sm.in.u[par], flag, sm.in.c[par ^ 1], (unsigned)s, a.err, m, dm))
        return;
      if (li == 31) S[kPB - 1] = unpack(dm);
    } else {
      if (!wait_msg<true, false>(sm.in.u[par], flag, a.err, m, dm)) return;
    }
    const double u = unpack(m);
    sm.us[li] = u;
    __syncwarp();
    double y0 = 0.0, y1 = 0.0, y2 = 0.0, y3 = 0.0;
#pragma unroll
    for (int j = 0; j < kPB; j += 4) {
      const double2 ua = pair_of(sm.us, j), ub = pair_of(sm.us, j + 2);
      y0 = fma(S[j], ua.x, y0);
      y1 = fma(S[j + 1], ua.y, y1);
      y2 = fma(S[j + 2], ub.x, y2);
      y3 = fma(S[j + 3], ub.y, y3);
    }
    const double y = (y0 + y1) + (y2 + y3);
    const double ht = 0.5 * warp_sum_tc(u * y);
    const double v = fma(-ht, u, y);
    sm.v[li] = v;
    __syncwarp();
    const double first = S[0] - fma(u, sm.v[0], v * sm.us[0]);
    if (s < a.s1 - 1) dc.put(par * (kPB + 1) + (li == 0 ? kPB : lane), first, flag);
#pragma unroll
    for (int j = 0; j < kPB; j += 2) {
      const double2 uj = pair_of(sm.us, j), vj = pair_of(sm.v, j);
      if (j > 0) S[j - 1] = S[j] - fma(u, vj.x, v * uj.x);
      S[j] = S[j + 1] - fma(u, vj.y, v * uj.y);
    }
    if (s == a.s1 - 1 && r + li < n) {
      double* p = a.sub + (long)r * kPOff + li;
      p[0] = first;
#pragma unroll
      for (int j = 1; j < kPB; ++j)
        if (j <= li) p[(long)j * (kPOff - 1)] = S[j - 1];
    }
  }
}

// Column s of every sweep: d and e of that column, the sweep's first reflector.
__device__ void run_head(const PipeArgs& a, SlotSmem* slots, const Word2* headbox) {
  const int lane = threadIdx.x & 31;
  for (int s = a.s0; s < a.s1; ++s) {
    const int first = (s + 1) & 31;
    const int li = (lane - first) & 31;  // row s + 1 + li
    double x, d;
    if (s == a.s0) {
      x = (s + 1 + li < a.n) ? a.sub[(long)s * kPOff + 1 + li] : 0.0;
      d = a.sub[(long)s * kPOff];
    } else {
      Word2 mine, dm;
      const Word2* m = headbox + ((s & 1) ^ 1) * (kPB + 1);
      if (!wait_msg<true, true>(m, (unsigned)s, a.err, mine, dm)) return;
      x = unpack(mine);
      d = unpack(dm);
    }
    const double nrm2 = warp_sum_tc(x * x);
    const double x0 = __shfl_sync(0xffffffffu, x, first);
    double u = 0.0, u0 = 0.0, beta = x0;
    if (nrm2 > 0.0) u = house(x, lane == first, x0, nrm2, u0, beta);
    st_sh(&slots[0].in.u[s & 1][lane], pack(u, (unsigned)(s + 1)));
    const int row = s + 1 + li;
    if (a.U != nullptr && row < a.n) a.U[row + (long)s * a.ldU] = u;
    double2* col = reinterpret_cast<double2*>(a.sub + (long)s * kPOff);
    col[lane] = (lane == 0) ? make_double2(d, beta) : make_double2(0.0, 0.0);
  }
}

// Cooperative launch: messages of the neighbour CTAs, global -> shared memory.
__device__ void run_relay_u(const PipeArgs& a, SlotSmem* slots, int k) {
  const int lane = threadIdx.x & 31;
  const int last = last_sweep(a.n, a.s1, k);
  const Boundary* b = a.bnd + blockIdx.x - 1;
  for (int s = a.s0; s <= last; ++s) {
    Word2 mine, dm;
    if (!wait_msg<false, false>(b->u[s & 1], (unsigned)(s + 1), a.err, mine, dm)) return;
    st_sh(&slots[0].in.u[s & 1][lane], mine);
  }
}
template <int SL>
__device__ void run_relay_c(const PipeArgs& a, SlotSmem* slots, int k) {
  const int lane = threadIdx.x & 31;
  const int last = last_sweep(a.n, a.s1, k);
  const Boundary* b = a.bnd + blockIdx.x;
  for (int s = a.s0 + 1; s <= last && takes_column(a.n, s + 1 + kPB * k); ++s) {
    Word2 mine, dm;
    const int q = (s & 1) ^ 1;
    if (!wait_msg<false, true>(b->c[q], (unsigned)s, a.err, mine, dm)) return;
    st_sh(&slots[SL - 1].in.c[q][lane], mine);
    if (lane == 0) st_sh(&slots[SL - 1].in.c[q][kPB], dm);
  }
}

template <int SL>
__global__ void __launch_bounds__(SL* kSlotThreads + 32 * kExtraWarps, 1)
    chase_pipe_kernel(const PipeArgs a) {
  __shared__ SlotSmem slots[SL];
  __shared__ Word2 headbox[2 * (kPB + 1)];
  const int tid = threadIdx.x;
  const bool cluster = a.bnd == nullptr;
  // no inbox entry may carry a flag of this launch (sweep + 1 >= 1)
  for (int e = tid; e < SL * (int)(sizeof(Inbox) / 16); e += blockDim.x) {
    constexpr int per = (int)(sizeof(Inbox) / 16);
    reinterpret_cast<Word2*>(&slots[e / per].in)[e % per] = Word2{0, 0};
  }
  if (tid < SL * 2) slots[tid >> 1].row_flag[tid & 1] = 0;
  for (int e = tid; e < 2 * (kPB + 1); e += blockDim.x) headbox[e] = Word2{0, 0};
  if (cluster && gridDim.x > 1) cg::this_cluster().sync();
  else __syncthreads();
  if (!cluster && !__syncthreads_and(tid != 0 || pass_gate(a.gate))) return;

  const int nslots = (a.n - 2 - a.s0) / kPB + 1;
  const int k0 = (int)blockIdx.x * SL;
  if (tid < SL * kSlotThreads) {
    const int w = tid >> 5, g = (w < SL) ? w : w - SL;  // N warps, then S warps
    if (k0 + g < nslots) {
      const Dest dc = dest_c<SL>(a, slots, headbox, g, cluster);
      if (w < SL) run_n<SL>(a, slots[g], dest_u<SL>(a, slots, g, cluster), dc, k0 + g);
      else run_s<SL>(a, slots[g], dc, k0 + g);
    }
  } else {
    const int w = (tid - SL * kSlotThreads) >> 5;
    if (w == 0 && blockIdx.x == 0) run_head(a, slots, headbox);
    if (!cluster && w == 1 && blockIdx.x > 0 && k0 < nslots) run_relay_u(a, slots, k0);
    if (!cluster && w == 2 && blockIdx.x + 1 < gridDim.x && k0 + SL - 1 < nslots)
      run_relay_c<SL>(a, slots, k0 + SL - 1);
  }
  // a neighbour may still be writing into this CTA's shared memory
  if (cluster && gridDim.x > 1) cg::this_cluster().sync();
}

// A launch that the device cannot hold at once (fewer SMs than it reports, no
// such cluster) is refused by the runtime: *used turns false.
template <int SL>
int launch(const PipeArgs& a, int ctas, bool coop, cudaStream_t st, bool* used) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(SL * kSlotThreads + 32 * kExtraWarps);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  cfg.attrs = at;
  cfg.numAttrs = 0;
  if (coop) {
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.numAttrs = 1;
  } else if (ctas > 1) {
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ctas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.numAttrs = 1;
  }
  const cudaError_t rc = cudaLaunchKernelEx(&cfg, chase_pipe_kernel<SL>, a);
  if (rc == cudaErrorCooperativeLaunchTooLarge || rc == cudaErrorInvalidClusterSize ||
      rc == cudaErrorInvalidConfiguration || rc == cudaErrorLaunchOutOfResources) {
    (void)cudaGetLastError();
    *used = false;
    return EVD_SUCCESS;
  }
  EVD_CUDA_TRY(rc);
  EVD_LAUNCHED();
  return EVD_SUCCESS;
}

constexpr int kSlA = 4, kSlB = 7;   // slots per CTA
constexpr int kMaxPipeCtas = 160;   // of a cooperative launch
constexpr long kClusterMinN = 1024; // orders up to it fit the portable cluster size

// A cluster of 16 CTAs needs 16 free SMs in one GPC; asked once per device.
bool cluster16_fits() {
  static std::mutex mu;
  static int state[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  std::lock_guard<std::mutex> lock(mu);
  if (state[dev] == 0) {
    const void* fn = (const void*)chase_pipe_kernel<kSlA>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(16);
    cfg.blockDim = dim3(kSlA * kSlotThreads + 32 * kExtraWarps);
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 16;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int count = 0;
    const bool ok =
        cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
            cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&count, fn, &cfg) == cudaSuccess && count > 0;
    (void)cudaGetLastError();
    state[dev] = ok ? 1 : -1;
  }
  return state[dev] > 0;
}

}  // namespace

// Ints of scratch for the boundary messages of a cooperative launch (16-byte
// aligned by the launcher, which needs 3 ints of slack).
long chase_pipe_ints(long n) {
  if (n <= kClusterMinN) return 0;
  const long ctas = std::min<long>((n + kPB * kSlA - 1) / (kPB * kSlA), kMaxPipeCtas);
  return ctas * (long)(sizeof(Boundary) / sizeof(int)) + 4;
}

// Whether the whole chase of order n runs as one pipeline launch on a device
// with `sms` SMs.
bool chase_pipelined(long n, int sms) {
  const long most = std::min(sms, kMaxPipeCtas);
  return n < 3 || (n - 2) / kPB + 1 <= most * kSlB;
}

// Sweeps [s0, s1) by the pipeline; false in *used when no form of it fits (the
// caller then runs chase_kernel), true in *gated when chase_kernel has to follow
// for the case that the gate shuts.  msg: chase_pipe_ints(n) ints, zeroed like
// the gate before the first part of a chase.
// The form, by the number of CTAs of 4 slots: one CTA, a cluster (messages
// through distributed shared memory), or a cooperative launch (through L2 and
// a relay warp), which costs 0.3 us more per message; with 7 slots per CTA
// (96 registers, the rows spill) where 4 would need more CTAs than SMs.
// Measured on B200, ms per chase (chase_kernel -> this kernel) and us per sweep:
//   n = 128: 0.83 -> 0.22 (1.7), 1024: 8.7 -> 1.43 (1.4), 2048: 18.0 -> 2.8 (1.4),
//   4096: 36.5 -> 8.5 (2.1), 16384: 182 -> 34.5 (2.1), 20000: 52 (2.6).
// Inside a cluster the N warp is busy all the time (2750 of 2900 cycles, 600 of
// them the reduce-scatter of z); above, the messages through L2 are the rest.
int launch_chase_pipe(long n, double* sub, double* U, long ldU, int* err, int* msg, int* gate,
                      long s0, long s1, int form, cudaStream_t st, bool* used, bool* gated) {
  *used = true;
  *gated = false;
  PipeArgs a{(int)n, (int)s0, (int)s1, sub, U, ldU, err, nullptr, gate};
  const int slots = (int)((n - 2 - s0) / kPB) + 1;
  const int need = (slots + kSlA - 1) / kSlA;
  if (need <= 8 || (need <= 16 && cluster16_fits())) {
    int c = 1;
    while (c < need) c *= 2;
    return launch<kSlA>(a, c, false, st, used);
  }
  a.bnd = reinterpret_cast<Boundary*>(((uintptr_t)msg + 15) & ~(uintptr_t)15);
  *gated = true;
  if (s0 > 0) EVD_CUDA_TRY(cudaMemsetAsync(gate, 0, sizeof(int), st));  // an earlier part's
  if (form == kChaseShut)  // its highest byte
    EVD_CUDA_TRY(cudaMemsetAsync(reinterpret_cast<char*>(gate) + 3, kGateShut >> 24, 1, st));
  const int most = std::min(device_sm_count(), kMaxPipeCtas);
  if (need <= most) return launch<kSlA>(a, need, true, st, used);
  const int needb = (slots + kSlB - 1) / kSlB;
  if (needb <= most) return launch<kSlB>(a, needb, true, st, used);
  *used = false;
  return EVD_SUCCESS;
}

}  // namespace evd

// The flow of messages as the kernel has it, for the host's check of the order
// it imposes: out = {last sweep of slot k, its task in sweep s waits for a
// reflector, waits for a column, sends a reflector, hands a row from N to S}.
extern "C" void evd_test_chase_flow(int n, int s0, int s1, int k, int s, int out[5]) {
  const int r = s + 1 + evd::kPB * k;
  out[0] = evd::last_sweep(n, s1, k);
  out[1] = 1;
  out[2] = s > s0 && evd::takes_column(n, r);
  out[3] = evd::has_next_slot(n, r);
  out[4] = s < s1 - 1 && s < out[0];
}
