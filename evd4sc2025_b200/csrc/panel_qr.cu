// Panel factorisation for stage 1: tall-skinny QR (m x 32) and the compact
// Householder form Q = I - W Y^T.
//
// Reference: panelQR<double> (api/panelQR.cu:54-108) = hou_tsqr_panel<128,32>
// (api/inc/TallShinnyQR.h:9-133, leaf kernel util/inc/kernelQR.h:215-414),
// then IminusQ, cusolverDnDgetrf without pivoting, getLower and a Dtrsm.
//
// Same numerics, B200 structure:
//  * The TSQR tree has the reference's shape (128-row tiles, R factors
//    stacked 32 rows per child, fan-in 4; api/inc/TallShinnyQR.h:9-133).  The
//    shape is kept on purpose: the signs of R (hence of Y, W and the band)
//    follow from the Householder sign rule applied node by node, so another
//    tree gives R up to row signs, not the reference's R.  It runs as ONE
//    up-sweep kernel, a CTA per tree node, in which the columns of R stream up
//    the tree: a parent works on a group of columns as soon as its children
//    have published theirs, so all levels work at once.  The reference
//    launches one kernel plus batched GEMMs per level.
//  * tsqr_q_kernel forms the explicit thin Q of all nodes at once from their
//    reflectors V (128 x 32, every tau = 1): Q_node = E - V K, E = [I; 0],
//    K = T V_top^T, T^-1 = I + striu(V^T V): a Gram matrix on DMMA, one
//    triangular solve, one DMMA product.
//  * The finishing kernel multiplies 32 x 32 blocks down the tree (right to left
//    as the reference's recursion): a leaf's rows of the thin Q are Q_leaf M.
//    Every CTA also walks to leaf 0 and factors (I - Q)[0:32] = L1 U there
//    (redundantly, no inter-CTA dependency), inverts both factors, and forms
//    Y = (I - Q) U^{-1} and W = (I - Q) L1^{-T} of its 128 rows as one
//    128 x 32 x 64 DMMA product.  This replaces the reference's getrf +
//    getLower + trsm + copy kernels.  Figures: at panel_qr_launch.
//  * In the sy2sb pipeline the finishing kernel writes Y and W straight into
//    dY/dW and the band (R over zeros) into dA (the reference's copyMatrix +
//    getU, api/zy_zy_sy2sb.cu:122-125).
#include "common.cuh"
#include "panel_qr.cuh"

namespace evd {

namespace {

constexpr int kTile = 128;        // rows per TSQR tile (reference: M = 128)
constexpr int kNB = 32;           // panel width (reference: N = 32)
constexpr int kFan = kTile / kNB; // children per tree node (their R factors fill one tile)
constexpr int kThreads = 256;
constexpr int kMaxLevels = 16;
constexpr int kErrWord = 1, kCounters = 2;  // places among the ints of the workspace

struct TsqrPlan {
  int m;
  int nlev;                 // number of levels; level nlev-1 is the root (1 tile)
  int T[kMaxLevels];        // tiles at each level
  int rows[kMaxLevels];     // rows of the matrix factored at each level
  long soff[kMaxLevels];    // offset (doubles) of stack S_L in ws (L >= 1)
  int coff[kMaxLevels];     // offset of the arrival counters of level L (L >= 1)
  long qtop_off;            // 32x32 copy of the top of leaf 0's Q, row-major
  long cnt_off;             // int counters start (in doubles, aligned)
  int ncnt;
  unsigned long long limit; // of a wait, ns
  long total;               // doubles
};

TsqrPlan make_plan(long m) {
  TsqrPlan p{};
  p.m = (int)m;
  int L = 0;
  p.rows[0] = (int)m;
  p.T[0] = ceil_div_i(m, kTile);
  int coff = 0;
  while (p.T[L] > 1 && L + 1 < kMaxLevels) {
    p.rows[L + 1] = kNB * p.T[L];
    p.T[L + 1] = ceil_div_i(p.rows[L + 1], kTile);
    p.coff[L + 1] = coff;
    coff += p.T[L + 1];
    ++L;
  }
  p.nlev = L + 1;
  // the ticket, the error word, a counter per inner node and column group
  p.ncnt = kCounters + kNB / 8 * coff;
  p.limit = 4000000000ull;
  // Arrival counters come first, at a fixed offset: a workspace sized (and
  // zeroed) for the largest panel then serves every smaller panel, whose
  // counters are a prefix of the same region (the kernels reset each counter
  // after use).
  p.cnt_off = 0;
  long off = (p.ncnt + 1) / 2 + 2;  // ints packed two per double
  off = (off + 1) / 2 * 2;        // keep the stacks 16-byte aligned
  for (int l = 1; l < p.nlev; ++l) {
    p.soff[l] = off;
    off += (long)p.rows[l] * kNB;
  }
  p.qtop_off = off;
  off += kNB * kNB;
  p.total = off;
  return p;
}

// ---- 32-wide products on the FP64 tensor pipe ----
// mma.m8n8k4: lane (g, t) = (lane / 4, lane % 4) holds A[g][t], B[t][g] and
// D[g][2t], D[g][2t+1].  32 x 32 matrices are row-major with kLd doubles per
// row, 128-row tiles column-major with kVLd per column: both strides are 32
// bytes mod 128, which makes every fragment read conflict-free.
constexpr int kLd = 36, kVLd = kTile + 4;

__device__ __forceinline__ void mma8(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}
// rows 8 mi .. 8 mi + 7 of A B, all 32 columns of B (both 32 x 32)
__device__ __forceinline__ void row_block(const double* A, const double* B, int mi,
                                          double (&d)[4][2]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int ni = 0; ni < 4; ++ni) d[ni][0] = d[ni][1] = 0.0;
#pragma unroll
  for (int kk = 0; kk < 8; ++kk) {
    const double af = A[(8 * mi + g) * kLd + 4 * kk + t];
#pragma unroll
    for (int ni = 0; ni < 4; ++ni) mma8(d[ni], af, B[(4 * kk + t) * kLd + 8 * ni + g]);
  }
}

// ---- up-sweep: all tree nodes at once, columns streamed up the tree ----
// One CTA per node (128 x 32 tile: rows of the panel, or the stacked R factors
// of four children).  A column of R is final as soon as its reflector is, and a
// parent needs of its children only the columns up to the one it works on, so
// a node takes its columns in four groups of eight, each as soon as all children
// have published theirs: load, apply the node's earlier reflectors as one
// compact-WY update on DMMA (A -= V T^T V^T A), factor the eight columns, publish
// their part of R, extend T.  All levels work at the same time, one group
// behind each other.  Same steps per column as my_hou_kernel<128,32>
// (util/inc/kernelQR.h:215-414): u = x/||x||, u0 += sign(u0), u scaled to
// ||u||^2 = 2; diag(R) = -sign(x0) ||x||.
//
// What bounds it: the chain of 32 columns, about 600 cycles each, once, plus
// eight columns per further level; factoring a level after the other took 21 us
// per level.  In the eight columns a warp owns one column, a lane four rows;
// x^T a and ||x||^2 are reduced together from the bare column x, and u^T a
// follows from the norm.
//
// Progress: CTAs take nodes from a ticket, leaves first, and wait only for
// children, which earlier tickets own.  When a wait runs out (4 s), the node
// fills its R with NaN and sets the workspace's error word, which the solvers
// report; the nodes and panels that follow wait no more (their counters may
// hold late arrivals) and have NaN too.
constexpr int kGrp = 8, kGroups = kNB / kGrp;
constexpr int kWLd = kGrp + 4;  // row stride of 8-wide matrices (conflict-free fragments)

struct UpSmem {
  double V[kNB * kVLd];
  double A[kGrp * kVLd];
  double T[kNB * kLd];
  double W[2][kNB * kWLd], W2[kNB * kWLd];
  double x[2][kTile];  // column j below row j (zero elsewhere)
  double x0[2];        // its row j
  double RR[kNB];
  int node, ok;
};

// D (8 x 8 tile) += A B over k-steps [k0, k1) in two chains; a(kk), b(kk) give
// this lane's fragment elements.
template <typename FA, typename FB>
__device__ __forceinline__ void tile_mma(double (&d)[2], int k0, int k1, FA a, FB b) {
  double e[2] = {0.0, 0.0};
  for (int kk = k0; kk < k1; kk += 2) {
    mma8(d, a(kk), b(kk));
    mma8(e, a(kk + 1), b(kk + 1));
  }
  d[0] += e[0];
  d[1] += e[1];
}

__global__ void __launch_bounds__(kThreads, 2)
    tsqr_up_kernel(const TsqrPlan plan, double* A, long lda, double* ws, double* Rout, long ldr) {
  pdl_entry();
  extern __shared__ __align__(16) double up_smem[];
  UpSmem& sm = *reinterpret_cast<UpSmem*>(up_smem);
  int* ticket = reinterpret_cast<int*>(ws + plan.cnt_off);
  int* err = ticket + kErrWord;
  int* cnt = ticket + kCounters;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  if (tid == 0) {
    sm.node = atomicAdd(ticket, 1);
    sm.ok = *(volatile int*)err == 0;
  }
  for (int e = tid; e < kNB * kLd; e += kThreads) sm.T[e] = 0.0;
  __syncthreads();
  int idx = sm.node, level = 0;
  while (idx >= plan.T[level]) idx -= plan.T[level++];
  const bool root = plan.T[level] == 1;
  double* src = (level == 0) ? A + (long)idx * kTile : ws + plan.soff[level] + (long)idx * kTile;
  const long ld = (level == 0) ? lda : plan.rows[level];
  const int mm = min(kTile, plan.rows[level] - idx * kTile);
  double* Rdst = root ? Rout : ws + plan.soff[level + 1] + (long)idx * kNB;
  const long ldR = root ? ldr : plan.rows[level + 1];
  const int nch = level ? min(kFan, plan.T[level - 1] - kFan * idx) : 0;
  int* arrived = level ? cnt + (plan.coff[level] + idx) * kGroups : nullptr;
  int* up = root ? nullptr : cnt + (plan.coff[level + 1] + idx / kFan) * kGroups;

  // element e of a thread's share of a group: row tid % 128, columns tid / 128 + 2 e
  const int lr = tid & (kTile - 1), lc = tid >> 7;
  double nxt[4];
  auto fetch = [&](int G) {
#pragma unroll
    for (int e = 0; e < 4; ++e)
      nxt[e] = (lr < mm) ? __ldcg(src + lr + (long)(kGrp * G + lc + 2 * e) * ld) : 0.0;
  };
  if (level == 0) fetch(0);

#pragma unroll 1
  for (int G = 0; G < kGroups; ++G) {
    if (level > 0) {
      if (tid == 0) {
        int* f = arrived + G;
        unsigned long long t0 = 0, now;
        for (unsigned it = 1; sm.ok && ld_acquire(f) < nch; ++it) {
          if ((it & 1023u) != 0) continue;
          asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
          if (t0 == 0) t0 = now;
          if (now - t0 > plan.limit) {
            atomicCAS(err, 0, kDevTimeoutTree);
            sm.ok = 0;
          }
        }
        if (sm.ok) *f = 0;  // ready for the next panel
      }
      __syncthreads();
      fetch(G);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e)
      sm.A[(lc + 2 * e) * kVLd + lr] = sm.ok ? nxt[e] : __longlong_as_double(0x7ff8000000000000ll);
    if (level == 0 && G + 1 < kGroups) fetch(G + 1);
    __syncthreads();
    if (G > 0) {
      // W = V^T A: tile warp / 2, half of K per warp
      if (warp < 2 * G) {
        const int mi = warp >> 1, h = warp & 1;
        double d[2] = {0.0, 0.0};
        const double* va = sm.V + (8 * mi + g) * kVLd + t;
        const double* ab = sm.A + g * kVLd + t;
        tile_mma(d, 16 * h, 16 * h + 16, [&](int kk) { return va[4 * kk]; },
                 [&](int kk) { return ab[4 * kk]; });
        sm.W[h][(8 * mi + g) * kWLd + 2 * t] = d[0];
        sm.W[h][(8 * mi + g) * kWLd + 2 * t + 1] = d[1];
      }
      __syncthreads();
      if (warp < G) {  // W2 = T^T W
        double d[2] = {0.0, 0.0};
        tile_mma(d, 0, 2 * G, [&](int kk) { return sm.T[(4 * kk + t) * kLd + 8 * warp + g]; },
                 [&](int kk) {
                   return sm.W[0][(4 * kk + t) * kWLd + g] + sm.W[1][(4 * kk + t) * kWLd + g];
                 });
        sm.W2[(8 * warp + g) * kWLd + 2 * t] = d[0];
        sm.W2[(8 * warp + g) * kWLd + 2 * t + 1] = d[1];
      }
      __syncthreads();
#pragma unroll
      for (int q = 0; q < 2; ++q) {  // A -= V W2
        const int row = 8 * (2 * warp + q) + g;
        double d[2] = {0.0, 0.0};
        tile_mma(d, 0, 2 * G, [&](int kk) { return sm.V[(4 * kk + t) * kVLd + row]; },
                 [&](int kk) { return sm.W2[(4 * kk + t) * kWLd + g]; });
        sm.A[(2 * t) * kVLd + row] -= d[0];
        sm.A[(2 * t + 1) * kVLd + row] -= d[1];
      }
      __syncthreads();
    }
    // ---- the eight columns: warp w has column 8 G + w, lane l rows 4 l .. 4 l + 3
    const int col = kGrp * G + warp;
    double a[4];
    {
      const double2 p = *reinterpret_cast<const double2*>(sm.A + warp * kVLd + 4 * lane);
      const double2 q = *reinterpret_cast<const double2*>(sm.A + warp * kVLd + 4 * lane + 2);
      a[0] = p.x;
      a[1] = p.y;
      a[2] = q.x;
      a[3] = q.y;
    }
    auto publish = [&](int j) {  // this warp's column j to shared memory
      double2* x = reinterpret_cast<double2*>(sm.x[j & 1] + 4 * lane);
      const int r = 4 * lane;
      x[0] = make_double2(r > j ? a[0] : 0.0, r + 1 > j ? a[1] : 0.0);
      x[1] = make_double2(r + 2 > j ? a[2] : 0.0, r + 3 > j ? a[3] : 0.0);
      if (lane == (j >> 2)) {
        const double lo = (j & 1) ? a[1] : a[0], hi = (j & 1) ? a[3] : a[2];
        sm.x0[j & 1] = (j & 2) ? hi : lo;
      }
    };
    if (warp == 0) publish(kGrp * G);
    __syncthreads();
#pragma unroll 1
    for (int w = 0; w < kGrp; ++w) {
      const int j = kGrp * G + w;
      const double x0 = sm.x0[j & 1];
      const double2 p = *reinterpret_cast<const double2*>(sm.x[j & 1] + 4 * lane);
      const double2 q = *reinterpret_cast<const double2*>(sm.x[j & 1] + 4 * lane + 2);
      double nrm2 = fma(p.x, p.x, p.y * p.y) + fma(q.x, q.x, q.y * q.y);
      double dot = fma(p.x, a[0], p.y * a[1]) + fma(q.x, a[2], q.y * a[3]);
      const double lo = (j & 1) ? a[1] : a[0], hi = (j & 1) ? a[3] : a[2];
      const double aj = __shfl_sync(0xffffffffu, (j & 2) ? hi : lo, j >> 2);
#pragma unroll
      for (int m = 16; m > 0; m >>= 1) {
        const double u = __shfl_xor_sync(0xffffffffu, nrm2, m);
        const double v = __shfl_xor_sync(0xffffffffu, dot, m);
        nrm2 += u;
        dot += v;
      }
      nrm2 = fma(x0, x0, nrm2);
      // A zero column (nothing to annihilate) gets u = sqrt(2) e_j rather than
      // u = 0: H = I - u u^T then only flips row j, R_jj = 0, every reflector
      // keeps ||u||^2 = 2, and I - Q stays nonsingular for the Householder
      // reconstruction (u = 0 would give a zero pivot there).
      const bool live = nrm2 > 0.0;
      const double rn = live ? rsqrt(nrm2) : 0.0;  // 1 / ||x||
      const double c0 = x0 * rn;
      const double sg = (c0 >= 0.0) ? 1.0 : -1.0;
      const double c0n = c0 + sg;
      const double s2 = rsqrt(fabs(c0n));
      const double sc = rn * s2;                               // u = sc x below row j
      const double u0 = live ? c0n * s2 : 1.4142135623730951;  // u in row j
      const bool at = lane == (j >> 2);
      if (warp > w) {
        const double d = fma(sc, dot, u0 * aj);  // u^T a
        const double f = -d * sc, fj = -d * u0;
        a[0] = fma(f, p.x, a[0]) + ((at && (j & 3) == 0) ? fj : 0.0);
        a[1] = fma(f, p.y, a[1]) + ((at && (j & 3) == 1) ? fj : 0.0);
        a[2] = fma(f, q.x, a[2]) + ((at && (j & 3) == 2) ? fj : 0.0);
        a[3] = fma(f, q.y, a[3]) + ((at && (j & 3) == 3) ? fj : 0.0);
        if (warp == w + 1) publish(j + 1);
      } else if (warp == w) {
        const double x[4] = {p.x, p.y, q.x, q.y};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          a[i] = (4 * lane + i > j) ? sc * x[i] : a[i];
          a[i] = (at && (j & 3) == i) ? u0 : a[i];
        }
        if (lane == 0) sm.RR[j] = -sg * (nrm2 * rn);
      }
      __syncthreads();
    }
    // ---- R of these columns to the parent, reflectors to V and the tile
    if (lane < kNB / 4) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int row = 4 * lane + i;
        Rdst[row + (long)col * ldR] = (row < col) ? a[i] : ((row == col) ? sm.RR[col] : 0.0);
      }
    }
    if (up != nullptr) {
      __syncthreads();
      if (tid == 0) {
        __threadfence();
        atomicAdd(up + G, 1);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = 4 * lane + i;
      const double v = (row >= col) ? a[i] : 0.0;
      sm.V[col * kVLd + row] = v;
      if (row < mm) src[row + (long)col * ld] = v;
    }
    if (G + 1 == kGroups) break;
    __syncthreads();
    // ---- T: its new columns are T22 = (I + striu(V2^T V2))^-1 and
    // T12 = -T11 (V1^T V2) T22
    if (warp < 2 * (G + 1)) {
      const int mi = warp >> 1, h = warp & 1;
      double d[2] = {0.0, 0.0};
      const double* va = sm.V + (8 * mi + g) * kVLd + t;
      const double* vb = sm.V + (8 * G + g) * kVLd + t;
      tile_mma(d, 16 * h, 16 * h + 16, [&](int kk) { return va[4 * kk]; },
               [&](int kk) { return vb[4 * kk]; });
      sm.W[h][(8 * mi + g) * kWLd + 2 * t] = d[0];
      sm.W[h][(8 * mi + g) * kWLd + 2 * t + 1] = d[1];
    }
    __syncthreads();
    if (warp == 0 && lane < kGrp) {  // column `lane` of T22, from its bottom
      double c[kGrp];
#pragma unroll
      for (int i = kGrp - 1; i >= 0; --i) {
        double acc = 0.0;
#pragma unroll
        for (int k = i + 1; k < kGrp; ++k)
          acc = fma(sm.W[0][(8 * G + i) * kWLd + k] + sm.W[1][(8 * G + i) * kWLd + k], c[k], acc);
        c[i] = (i < lane) ? -acc : (i == lane ? 1.0 : 0.0);
        sm.T[(8 * G + i) * kLd + 8 * G + lane] = c[i];
      }
    }
    __syncthreads();
    if (warp < G) {  // P = (V1^T V2) T22
      double d[2] = {0.0, 0.0};
      tile_mma(d, 0, 2,
               [&](int kk) {
                 const int at = (8 * warp + g) * kWLd + 4 * kk + t;
                 return sm.W[0][at] + sm.W[1][at];
               },
               [&](int kk) { return sm.T[(8 * G + 4 * kk + t) * kLd + 8 * G + g]; });
      sm.W2[(8 * warp + g) * kWLd + 2 * t] = d[0];
      sm.W2[(8 * warp + g) * kWLd + 2 * t + 1] = d[1];
    }
    __syncthreads();
    if (warp < G) {  // T12 = -T11 P
      double d[2] = {0.0, 0.0};
      tile_mma(d, 0, 2 * G, [&](int kk) { return sm.T[(8 * warp + g) * kLd + 4 * kk + t]; },
               [&](int kk) { return sm.W2[(4 * kk + t) * kWLd + g]; });
      sm.T[(8 * warp + g) * kLd + 8 * G + 2 * t] = -d[0];
      sm.T[(8 * warp + g) * kLd + 8 * G + 2 * t + 1] = -d[1];
    }
    // T and V are next read after the barriers of the next group's load
  }
  if (root && tid == 0) *ticket = 0;  // every node has been taken: ready for the next panel
}

struct QSmem {
  double V[kNB * kVLd];
  double G[kNB * kLd];  // G[j * kLd + i] = (V^T V)_ij, i < j
  double K[kNB * kLd];
};

// x[i] -= row[i] * f, i < j, the row read two at a time before the products.
template <int J>
__device__ __forceinline__ void eliminate(double (&x)[kNB], const double* row, double f) {
  double2 t[(J + 1) / 2 + 1];
#pragma unroll
  for (int i = 0; i < (J + 1) / 2; ++i) t[i] = *reinterpret_cast<const double2*>(row + 2 * i);
#pragma unroll
  for (int i = 0; i < J; ++i) x[i] = fma(-((i & 1) ? t[i / 2].y : t[i / 2].x), f, x[i]);
}
// Back substitution, lane = right-hand side: B x = rhs, B upper triangular with
// B_ij at Bt[j * kLd + i] (i < j) and diagonal 1 / rd (unit when rd is null).
template <int J = kNB - 1>
__device__ __forceinline__ void back_solve(double (&x)[kNB], const double* Bt, const double* rd) {
  if (rd) x[J] *= rd[J];
  if constexpr (J > 0) {
    eliminate<J>(x, Bt + J * kLd, x[J]);
    back_solve<J - 1>(x, Bt, rd);
  }
}

// Explicit Q of every tree node, all levels at once (the up-sweep left the
// reflectors in each node's tile): one CTA per node, Q = E - V K.
__global__ void __launch_bounds__(kThreads, 1)
    tsqr_q_kernel(const TsqrPlan plan, double* A, long lda, double* ws) {
  pdl_entry();
  extern __shared__ __align__(16) double q_smem[];
  QSmem& sm = *reinterpret_cast<QSmem*>(q_smem);
  int idx = blockIdx.x, level = 0;
  while (level < plan.nlev && idx >= plan.T[level]) {
    idx -= plan.T[level];
    ++level;
  }
  if (level >= plan.nlev) return;
  double* src = (level == 0) ? A + (long)idx * kTile : ws + plan.soff[level] + (long)idx * kTile;
  const long ld = (level == 0) ? lda : plan.rows[level];
  const int mm = min(kTile, plan.rows[level] - idx * kTile);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int e = threadIdx.x; e < kNB * kTile; e += kThreads) {
    const int j = e / kTile, row = e % kTile;
    sm.V[j * kVLd + row] = (row < mm) ? __ldcg(src + row + (long)j * ld) : 0.0;
  }
  __syncthreads();
  // the ten upper 8 x 8 tiles of V^T V
  for (int q = warp; q < 10; q += kThreads / 32) {
    const int nj = (q < 1) ? 0 : (q < 3) ? 1 : (q < 6) ? 2 : 3;
    const int mi = q - nj * (nj + 1) / 2;
    double d[2] = {0.0, 0.0}, f[2] = {0.0, 0.0};
    const double* va = sm.V + (8 * mi + g) * kVLd + t;
    const double* vb = sm.V + (8 * nj + g) * kVLd + t;
#pragma unroll 8
    for (int kk = 0; kk < kTile / 8; ++kk) {
      mma8(d, va[8 * kk], vb[8 * kk]);
      mma8(f, va[8 * kk + 4], vb[8 * kk + 4]);
    }
    sm.G[(8 * nj + 2 * t) * kLd + 8 * mi + g] = d[0] + f[0];
    sm.G[(8 * nj + 2 * t + 1) * kLd + 8 * mi + g] = d[1] + f[1];
  }
  __syncthreads();
  if (warp == 0) {
    // (I + striu(G)) K = V_top^T, column `lane` of K
    double k[kNB];
#pragma unroll
    for (int i = 0; i < kNB; ++i) k[i] = sm.V[i * kVLd + lane];
    back_solve(k, sm.G, nullptr);
#pragma unroll
    for (int i = 0; i < kNB; ++i) sm.K[i * kLd + lane] = k[i];
  }
  __syncthreads();
  for (int mi = warp; mi < kTile / 8; mi += kThreads / 32) {
    double d[4][2];
#pragma unroll
    for (int ni = 0; ni < 4; ++ni) d[ni][0] = d[ni][1] = 0.0;
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) {
      const double af = sm.V[(4 * kk + t) * kVLd + 8 * mi + g];
#pragma unroll
      for (int ni = 0; ni < 4; ++ni) mma8(d[ni], af, sm.K[(4 * kk + t) * kLd + 8 * ni + g]);
    }
    const int row = 8 * mi + g;
    if (row >= mm) continue;
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = 8 * ni + 2 * t + h;
        const double v = ((row == c) ? 1.0 : 0.0) - d[ni][h];
        src[row + (long)c * ld] = v;
        // leaf 0's tile is overwritten by the finishing kernel's CTA 0
        if (blockIdx.x == 0 && row < kNB) ws[plan.qtop_off + row * kNB + c] = v;
      }
  }
}

constexpr int kHalf = kThreads / 2;  // threads of a group of the finishing kernel

struct FinishSmem {
  double Q[kNB * kVLd];  // this CTA's rows of its leaf's Q
  // per group (0: this CTA's leaf, 1: leaf 0): the current block, two products
  double B[2][kNB * kLd], M[2][2][kNB * kLd];
  double Ui[kNB * kLd];  // U^{-1}
  double Li[kNB * kLd];  // L1^{-T}
  double L[kNB * kLd];   // L1, row-major: L1^T by columns
  double Ut[kNB * kLd];  // U by columns
  double rd[kNB];        // 1 / U_jj
  double A0[kNB * kLd];  // (I - Q)[0:32]
};

// 1 / x of a normal number to about an ulp: the hardware's approximation and two
// Newton steps, without the branches of a division.
__device__ __forceinline__ double reciprocal(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  r = fma(r, fma(-x, r, 1.0), r);
  return fma(r, fma(-x, r, 1.0), r);
}

__global__ void reciprocal_kernel(long n, const double* x, double* y) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i < n) y[i] = reciprocal(x[i]);
}

__device__ __forceinline__ void group_bar(int grp) {
  asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "n"(kHalf) : "memory");
}
// Out = s * A B + (ident ? I : 0), all 32 x 32, by a group of four warps.
__device__ __forceinline__ void group_mul(const double* A, const double* B, double* Out, double s,
                                          bool ident) {
  const int w = (threadIdx.x & (kHalf - 1)) >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, q = lane & 3;
  double d[4][2];
  row_block(A, B, w, d);
#pragma unroll
  for (int ni = 0; ni < 4; ++ni)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = 8 * w + g, c = 8 * ni + 2 * q + h;
      Out[r * kLd + c] = fma(s, d[ni][h], (ident && r == c) ? 1.0 : 0.0);
    }
}

// Path product down the tree to leaf t, M = B_1 (B_2 (... B_top)) with B_L the
// rows of level L's Q that belong to the child on the path; returns M.
__device__ const double* walk(const TsqrPlan& plan, const double* __restrict__ ws, int t, int grp,
                              FinishSmem& sm) {
  const int tid = threadIdx.x & (kHalf - 1);
  constexpr int kPer = kNB * kNB / kHalf;  // elements per thread of a 32 x 32 block
  double br[kPer];
  auto fetch = [&](int level) {  // level >= 1
    const double* b = ws + plan.soff[level] + (long)kNB * (t >> (2 * (level - 1)));
#pragma unroll
    for (int e = 0; e < kPer; ++e) {
      const int at = tid + e * kHalf;
      br[e] = __ldcg(b + (at & 31) + (long)(at >> 5) * plan.rows[level]);
    }
  };
  auto put = [&](double* dst) {
#pragma unroll
    for (int e = 0; e < kPer; ++e) {
      const int at = tid + e * kHalf;
      dst[(at & 31) * kLd + (at >> 5)] = br[e];
    }
  };
  int level = plan.nlev - 1, cur = 0;
  if (level == 0) {
#pragma unroll
    for (int e = 0; e < kPer; ++e) {
      const int at = tid + e * kHalf;
      sm.M[grp][0][(at >> 5) * kLd + (at & 31)] = ((at >> 5) == (at & 31)) ? 1.0 : 0.0;
    }
    group_bar(grp);
    return sm.M[grp][0];
  }
  fetch(level);
  put(sm.M[grp][0]);
  while (--level > 0) {
    fetch(level);
    put(sm.B[grp]);
    group_bar(grp);
    group_mul(sm.B[grp], sm.M[grp][cur], sm.M[grp][cur ^ 1], 1.0, false);
    cur ^= 1;
    group_bar(grp);
  }
  group_bar(grp);
  return sm.M[grp][cur];
}
static_assert(kFan == 4, "walk() shifts the child index by two bits per level");

// mode 0: write the explicit thin Q into A (evd_tsqr).
// mode 1: write Y (into Yout), W (into Wout), and optionally the band panel
//         (R over zeros) into Aband (sy2sb).
__global__ void __launch_bounds__(kThreads, 1)
    tsqr_finish_kernel(const TsqrPlan plan, const double* ws, double* A, long lda, int mode,
                       double* Yout, long ldy, double* Wout, long ldw, const double* Rin,
                       long ldr, double* Aband, long ldband) {
  pdl_entry();
  extern __shared__ __align__(16) double dsm[];
  FinishSmem& sm = *reinterpret_cast<FinishSmem*>(dsm);
  const int t = blockIdx.x;
  const int r0 = t * kTile;
  const int mm = min(kTile, plan.m - r0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const int grp = threadIdx.x / kHalf;
  const double* M = nullptr;
  if (grp == 0) {
#pragma unroll 16
    for (int e = threadIdx.x; e < kNB * kTile; e += kHalf) {
      const int j = e / kTile, row = e % kTile;
      sm.Q[j * kVLd + row] = (row < mm) ? __ldcg(A + (long)(r0 + row) + (long)j * lda) : 0.0;
    }
    walk(plan, ws, t, 0, sm);
  } else if (mode == 1) {
    M = walk(plan, ws, 0, 1, sm);
    for (int at = threadIdx.x - kHalf; at < kNB * kNB; at += kHalf)
      sm.B[1][(at >> 5) * kLd + (at & 31)] = __ldcg(ws + plan.qtop_off + at);
    group_bar(1);
    group_mul(sm.B[1], M, sm.A0, -1.0, true);
    group_bar(1);
    const int w1 = warp - kHalf / 32;
    if (w1 == 0) {
      // unpivoted LU by one warp (lane = row, the row in registers; row k is
      // broadcast by shuffles, all issued before the pivot's reciprocal is
      // needed): 14k cycles; a rolled loop, rows through shared memory and four
      // warps with a barrier per step took 16k to 29k
      double lu[kNB];
#pragma unroll
      for (int c = 0; c < kNB; ++c) lu[c] = sm.A0[lane * kLd + c];
#pragma unroll
      for (int k = 0; k < kNB; ++k) {
        double row[kNB];
#pragma unroll
        for (int c = k; c < kNB; ++c) row[c] = __shfl_sync(0xffffffffu, lu[c], k);
        const double rp = reciprocal(row[k]);
        if (lane == 0) sm.rd[k] = rp;
        const double l = (lane > k) ? lu[k] * rp : 0.0;
        if (lane > k) lu[k] = l;
#pragma unroll
        for (int c = k + 1; c < kNB; ++c) lu[c] = fma(-l, row[c], lu[c]);
      }
#pragma unroll
      for (int c = 0; c < kNB; ++c) {
        sm.L[lane * kLd + c] = (c < lane) ? lu[c] : ((c == lane) ? 1.0 : 0.0);
        sm.Ut[c * kLd + lane] = (c >= lane) ? lu[c] : 0.0;
      }
    }
    group_bar(1);
    // both inverses, lane = column
    if (w1 < 2) {
      double x[kNB];
#pragma unroll
      for (int i = 0; i < kNB; ++i) x[i] = (i == lane) ? 1.0 : 0.0;
      if (w1 == 0) back_solve(x, sm.Ut, sm.rd);
      else back_solve(x, sm.L, nullptr);
      double* dst = (w1 == 0) ? sm.Ui : sm.Li;
#pragma unroll
      for (int i = 0; i < kNB; ++i) dst[i * kLd + lane] = x[i];
    }
  }
  __syncthreads();
  M = sm.M[0][max(plan.nlev - 2, 0) & 1];  // where walk() left this leaf's product

  if (mode == 0) {
    for (int mi = warp; mi < kTile / 8; mi += kThreads / 32) {
      double d[4][2];
#pragma unroll
      for (int ni = 0; ni < 4; ++ni) d[ni][0] = d[ni][1] = 0.0;
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) {
        const double af = sm.Q[(4 * kk + q) * kVLd + 8 * mi + g];
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) mma8(d[ni], af, M[(4 * kk + q) * kLd + 8 * ni + g]);
      }
      const int row = 8 * mi + g;
      if (row >= mm) continue;
#pragma unroll
      for (int ni = 0; ni < 4; ++ni)
#pragma unroll
        for (int h = 0; h < 2; ++h) A[(long)(r0 + row) + (long)(8 * ni + 2 * q + h) * lda] = d[ni][h];
    }
    return;
  }

  // rows >= 32: I - Q = -Q_leaf M, so Y = -Q_leaf (M U^{-1}), W = -Q_leaf (M L1^{-T});
  // the products (negated) go to B[0] and B[1]
  group_mul(M, grp ? sm.Li : sm.Ui, sm.B[grp], -1.0, false);
  __syncthreads();
  for (int mi = warp; mi < kTile / 8; mi += kThreads / 32) {
    const bool head = t == 0 && mi < kNB / 8;
    const double* by = head ? sm.Ui : sm.B[0];
    const double* bw = head ? sm.Li : sm.B[1];
    double y[4][2], z[4][2];
#pragma unroll
    for (int ni = 0; ni < 4; ++ni) y[ni][0] = y[ni][1] = z[ni][0] = z[ni][1] = 0.0;
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) {
      const double af = head ? sm.A0[(8 * mi + g) * kLd + 4 * kk + q]
                             : sm.Q[(4 * kk + q) * kVLd + 8 * mi + g];
#pragma unroll
      for (int ni = 0; ni < 4; ++ni) {
        mma8(y[ni], af, by[(4 * kk + q) * kLd + 8 * ni + g]);
        mma8(z[ni], af, bw[(4 * kk + q) * kLd + 8 * ni + g]);
      }
    }
    const int row = 8 * mi + g;
    if (row >= mm) continue;
    const long gr = r0 + row;
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = 8 * ni + 2 * q + h;
        Yout[gr + (long)c * ldy] = head ? sm.L[row * kLd + c] : y[ni][h];
        Wout[gr + (long)c * ldw] = z[ni][h];
        if (Aband)
          Aband[gr + (long)c * ldband] =
              (gr < kNB && c >= gr) ? __ldcg(Rin + gr + (long)c * ldr) : 0.0;
      }
  }
}

int finish_attr() {
  EVD_TRY(smem_attr_once((const void*)tsqr_finish_kernel, (int)sizeof(FinishSmem)));
  EVD_TRY(smem_attr_once((const void*)tsqr_up_kernel, (int)sizeof(UpSmem)));
  EVD_TRY(smem_attr_once((const void*)tsqr_q_kernel, (int)sizeof(QSmem)));
  return EVD_SUCCESS;
}

}  // namespace

long panel_qr_ws_doubles(long m) { return make_plan(m).total; }

const int* panel_error_word(const double* ws) {
  return reinterpret_cast<const int*>(ws) + kErrWord;  // cnt_off is 0 for every m
}

int panel_qr_check(long m, long n, long lda) {
  if (n != kNB || m < kNB || (m % kNB) != 0 || lda < m) return EVD_ERR_INVALID_ARG;
  if (m > (1L << 30)) return EVD_ERR_INVALID_ARG;
  return EVD_SUCCESS;
}

int panel_counters_reset(long m, double* ws, cudaStream_t st) {
  TsqrPlan plan = make_plan(m);
  if (plan.ncnt > 0)
    EVD_CUDA_TRY(cudaMemsetAsync(ws + plan.cnt_off, 0, sizeof(int) * plan.ncnt, st));
  return EVD_SUCCESS;
}

// Three launches.  Measured on B200, us per panel, with a tree level after the
// other, explicit node Q's by 32 rank-1 updates and row-by-row solves -> now:
// m = 128 89 -> 48, 992 178 -> 65, 4096 235 -> 72, 16384 226 -> 95.  What is left:
// the 32 dependent columns, 5 us per further tree level, 6 us for the node Q's
// and 16 us to finish, half of it the 32 steps of the LU.
int panel_qr_launch(long m, double* A, long lda, double* ws, int mode, double* Yout, long ldy,
                    double* Wout, long ldw, double* R, long ldr, double* Aband, long ldband,
                    cudaStream_t st) {
  TsqrPlan plan = make_plan(m);
  if (plan.nlev >= kMaxLevels) return EVD_ERR_INVALID_ARG;
  EVD_TRY(finish_attr());
  int nodes = 0;
  for (int l = 0; l < plan.nlev; ++l) nodes += plan.T[l];
  EVD_TRY(launch_pdl(tsqr_up_kernel, nodes, kThreads, sizeof(UpSmem), st, plan, A, lda, ws, R,
                     ldr));
  EVD_TRY(launch_pdl(tsqr_q_kernel, nodes, kThreads, sizeof(QSmem), st, plan, A, lda,
                     ws));
  EVD_TRY(launch_pdl(tsqr_finish_kernel, plan.T[0], kThreads, sizeof(FinishSmem), st,
                     plan, ws, A, lda, mode, Yout, ldy, Wout, ldw, R, ldr, Aband, ldband));
  return EVD_SUCCESS;
}

}  // namespace evd

extern "C" long evd_panel_qr_work_size(long m, long n) {
  if (evd::panel_qr_check(m, n, m) != EVD_SUCCESS) return 0;
  return evd::panel_qr_ws_doubles(m);
}

extern "C" int evd_tsqr(long m, long n, double* A, long lda, double* R, long ldr, double* work,
                        long lwork, cudaStream_t stream) {
  EVD_TRY(evd::panel_qr_check(m, n, lda));
  if (!A || !R || !work || ldr < n) return EVD_ERR_INVALID_ARG;
  if (lwork < evd::panel_qr_ws_doubles(m)) return EVD_ERR_WORKSPACE;
  EVD_TRY(evd::panel_counters_reset(m, work, stream));
  return evd::panel_qr_launch(m, A, lda, work, 0, nullptr, 0, nullptr, 0, R, ldr, nullptr, 0,
                              stream);
}

extern "C" int evd_panel_qr(long m, long n, double* A, long lda, double* W, long ldw, double* R,
                            long ldr, double* work, long lwork, cudaStream_t stream) {
  EVD_TRY(evd::panel_qr_check(m, n, lda));
  if (!A || !W || !R || !work || ldr < n || ldw < m) return EVD_ERR_INVALID_ARG;
  if (lwork < evd::panel_qr_ws_doubles(m)) return EVD_ERR_WORKSPACE;
  EVD_TRY(evd::panel_counters_reset(m, work, stream));
  return evd::panel_qr_launch(m, A, lda, work, 1, A, lda, W, ldw, R, ldr, nullptr, 0, stream);
}

// For the tests: the up-sweep without its first leaf and with waits of `limit`
// ns (at most 1 s), on a workspace as the last call left it or (fresh) reset;
// returns the status that a solver would.
extern "C" int evd_test_tsqr_timeout(long m, double* A, long lda, double* R, double* work,
                                     int fresh, long limit, cudaStream_t stream) {
  using namespace evd;
  EVD_TRY(panel_qr_check(m, kNB, lda));
  TsqrPlan plan = make_plan(m);
  if (plan.nlev < 2 || limit > 1000000000) return EVD_ERR_INVALID_ARG;
  EVD_TRY(finish_attr());
  if (fresh) EVD_TRY(panel_counters_reset(m, work, stream));
  const int one = 1;
  EVD_CUDA_TRY(cudaMemcpyAsync(work, &one, sizeof(int), cudaMemcpyHostToDevice, stream));
  int nodes = -1;
  for (int l = 0; l < plan.nlev; ++l) nodes += plan.T[l];
  plan.limit = (unsigned long long)limit;
  EVD_TRY(launch_pdl(tsqr_up_kernel, nodes, kThreads, sizeof(UpSmem), stream, plan, A, lda, work,
                     R, (long)kNB));
  return read_device_error(panel_error_word(work), stream);
}

// For the tests: y = reciprocal(x) of the panel's LU, elementwise.
extern "C" int evd_test_reciprocal(long n, const double* x, double* y, cudaStream_t stream) {
  if (n <= 0) return EVD_SUCCESS;
  evd::reciprocal_kernel<<<evd::ceil_div_i(n, 256), 256, 0, stream>>>(n, x, y);
  EVD_LAUNCHED();
  return EVD_SUCCESS;
}
