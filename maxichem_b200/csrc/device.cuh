// Device arithmetic of the per-call chemistry solve: rates, right-hand side, Jacobian, dense LU and solves,
// Rodas3 stages, step control and the guard. One CTA steps one cell at a time; its W warps share the cell's arrays in
// shared memory. Every sum that reaches the state has a fixed order (ascending index, or the 32-lane butterfly), so
// a cell's result does not depend on the batch, its order, or the launch shape.
//
// Arithmetic follows imalsky/maxichem maxichem/kernels/common.cuh, call.cuh, guard.cuh and recover.cuh (cited per
// function). The library is built with -fmad=false: every fused multiply-add is an explicit fma().
#pragma once
#include <cstdint>

#include "../../include/maxichem_b200.h"

namespace mx {

constexpr unsigned FULL = 0xffffffffu;
constexpr double GAMMA = 0.5;            // Rodas3's diagonal coefficient (Sandu et al. 1997)
constexpr double RODAS_C21 = 4.0;        // stage coupling C_21
constexpr double RODAS_C43 = 8.0 / 3.0;  // stage coupling, -C_43
constexpr double TROE_C0 = 0.4, TROE_C1 = 0.67, TROE_N0 = 0.75, TROE_N1 = 1.27, TROE_D = 0.14;  // Venot et al. 2012
constexpr int FL_FALLOFF = 1, FL_SECOND_K0 = 2, FL_THREE_BODY = 4, FL_TROE = 64, FL_EFF = 128, FL_VM11 = 512;
constexpr int GUARD_NONFINITE = 4, GUARD_UNFINISHED = 8, GUARD_DRIFT = 16;

// A network's tables on the device, and the per-CTA shared-memory layout (offsets in doubles).
struct Net {
  int ns, nr, nrt, nj, nel, n_entries;
  const int* perm;
  const uint64_t* rx8;  // 8 bytes per reaction: reactants 0-2, products 3-5, padding
  const double* rc;
  const int* rf;
  const double* nasa;
  const double* atoms;
  const int* sv_ptr;
  const uint32_t* sv_term;
  const int* jac_ptr;
  const uint32_t* jac_entry;
  const uint32_t* jac_term;
  double etot, drift;
  // per-thread streams of the S v and Jacobian sums for the CTA (group 0) and its last 96 threads (group 1)
  int st_threads[2], sv_rounds[2], jac_rounds, n_pieces;
  const int* sv_row_ptr;
  // four words of a thread together, group q of thread t at q * threads + t, a spare group at the end
  const uint4* sv[2];  // S v: reaction | coefficient code << 11 | end of a piece << 13 | the piece << 16
  const uint4* jt;     // the Jacobian's terms, for the CTA
  const uint2* jd;     // per term 16 bits: where its entry goes when the term ends it
  // shared-memory layout (offsets in doubles); a_doubles: the matrix region's size in doubles. The mixed-precision
  // layout adds the row scales (oS), the Jacobian's diagonal (oDg), n at the try's state (onN), w (oW), the
  // residual (oR) and a stage's right side (oB); the plain layout leaves them 0.
  int ld, oA, oK, oV, on, oN, oY, oF, oU, oK1, oK2, oK3, oK4, oD, oRed, oInts, oPart, oG, doubles, a_doubles;
  int oS, oDg, onN, oW, oR, oB;
  unsigned sms;  // of the device
};

struct CallArgs {
  const double *x, *T, *P, *dt, *h_in, *J;
  int B;
  double rtol, atol;
  int max_steps;
  double *x_out, *h_out;
  int* done;
  double* steps;
  int *flag, *status, *count, *list;
  unsigned long long* tries;  // nullable: [0] tries, [1] tries after a rejection, [2] recovery tries
  const int* in_list;  // list-mode kernels: the cells to step, in_count[0] of them (in_count[1]: their queue)
  int* in_count;
  int* sel;        // the mixed kernel's hand-backs for the plain kernel, sel_count[0] of them
  int* sel_count;
};

// Pointers into one CTA's shared memory.
struct Cell {
  double *A, *kf, *kr, *v, *n, *N, *Y, *F, *U, *K1, *K2, *K3, *K4, *dinv, *red, *part, *G;
  int* ints;
};

__device__ __forceinline__ Cell cell_arrays(const Net& net, double* smem) {
  Cell c;
  c.A = smem + net.oA;
  c.kf = smem + net.oK;
  c.kr = c.kf + net.nr;
  c.v = smem + net.oV;
  c.n = smem + net.on;
  c.N = smem + net.oN;
  c.Y = smem + net.oY;
  c.F = smem + net.oF;
  c.U = smem + net.oU;
  c.K1 = smem + net.oK1;
  c.K2 = smem + net.oK2;
  c.K3 = smem + net.oK3;
  c.K4 = smem + net.oK4;
  c.dinv = smem + net.oD;
  c.red = smem + net.oRed;
  c.ints = (int*)(smem + net.oInts);
  c.part = smem + net.oPart;
  c.G = smem + net.oG;
  return c;
}

// The thread's index, with a 2-warp CTA's warps exchanged in every other pair of CTAs of an SM. Warp 0 runs the triangular
// solves, so the warps 0 of an SM's CTAs should sit on different schedulers. The device gives 4-warp CTAs' warps slots
// that do (measured: 0 1 2 3, 5 6 7 4, 10 11 8 9, 15 12 13 14; rotating them here put all four on one scheduler, 98
// against 84 ms for 65,536 cells of 69 species), 2-warp CTAs' ones slots 0 1, 2 3, 4 5, ..., two schedulers of four
// (a settled call of 40,000 cells of 41 species: 9.77 ms without the exchange, 9.31 with it; 1,000 cells 0.48 and 0.47).
// It takes CTA b for the (b / SMs)-th of its SM, the order in which a grid's first CTAs were dealt out here; where a
// device deals them out otherwise, results are the same and the exchange may gain nothing.
template <int W>
__device__ __forceinline__ int spread_tid(unsigned sms) {
  if (W != 2) return (int)threadIdx.x;
  const int turn = (int)(blockIdx.x / sms) / 2;
  return (int)((threadIdx.x + 32 * turn) % (32 * W));
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
  return v;
}

__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(FULL, v, o));
  return v;
}

// sum of y[0..n) as a warp forms it: lane l adds y[l], y[l + 32], ... then the butterfly (every lane returns it). Four
// loads at a time; past the end it adds 0.
__device__ __forceinline__ double lane_sum(const double* y, int n, int lane) {
  double p = 0.0;
#pragma unroll 1
  for (int i = lane; i < n; i += 128) {
    double v[4];
#pragma unroll
    for (int q = 0; q < 4; q++) v[q] = i + 32 * q < n ? y[i + 32 * q] : 0.0;
#pragma unroll
    for (int q = 0; q < 4; q++) p += v[q];
  }
  return warp_sum(p);
}

// +1, -1, +2, -2 for the codes 0-3 in c's lowest bits, put together as a double's upper half
__device__ __forceinline__ double code_coefficient(unsigned c) {
  return __hiloint2double((int)((0x3ff00000u + ((c & 2u) << 19)) | (c << 31)), 0);
}

// ---- rates (common.cuh:136-242) ----

__device__ __forceinline__ double law(const double* __restrict__ q, int fl, double Tc, double lT, double iT,
                                      double nd) {
  double k = exp(q[0] + q[1] * lT - q[2] * iT);
  if (fl & FL_SECOND_K0) k += exp(q[3] + q[4] * lT - q[5] * iT);
  if (fl & FL_FALLOFF) {
    const double pr = k * nd / exp(q[6] + q[7] * lT - q[8] * iT);
    k = k > 0.0 ? k / (1.0 + pr) : 0.0;
    if ((fl & FL_TROE) && k > 0.0) {
      const double fc = log10((1.0 - q[9]) * exp(-Tc / q[10]) + q[9] * exp(-Tc / q[11]) + exp(-q[12] / Tc));
      const double x = (fl & FL_VM11) ? log10(pr) : log10(pr) - TROE_C0 - TROE_C1 * fc;
      // at Pr = 0 the standard ratio tends to -1 / d, so F to Fc^(d^2 / (1 + d^2)); the VM11 one to -inf, F to 1
      const double y = (fl & FL_VM11) ? x / (TROE_N0 - TROE_N1 * fc)
                                      : (isfinite(x) ? x / (TROE_N0 - TROE_N1 * fc - TROE_D * x) : -1.0 / TROE_D);
      k *= exp10(fc / (1.0 + y * y));
    }
  }
  if (fl & FL_EFF) k *= q[13];
  return k;
}

__device__ __forceinline__ double bimolecular_rate(int molecules, bool three_body, double k, double nd) {
  return molecules >= 2 ? k * (molecules == 3 ? nd : 1.0) : (three_body ? k / nd : 0.0);
}

__device__ __forceinline__ double gibbs_rt(const double* __restrict__ a, double Tc, double lT, double iT) {
  const double T2 = Tc * Tc, T3 = T2 * Tc, T4 = T3 * Tc;
  const double h = -a[0] * iT * iT + a[1] * lT * iT + a[2] + a[3] * Tc / 2 + a[4] * T2 / 3 + a[5] * T3 / 4 +
                   a[6] * T4 / 5 + a[7] * iT;
  const double s = -a[0] * iT * iT / 2 - a[1] * iT + a[2] * lT + a[3] * Tc + a[4] * T2 / 2 + a[5] * T3 / 3 +
                   a[6] * T4 / 4 + a[8];
  return h - s;
}

// kf, kr of one cell (cell_rates, common.cuh:222-242); g (ns + 1 doubles) is scratch. Two barriers.
__device__ __forceinline__ void cell_rates(const Net& net, const Cell& c, double Tc, double nd, const double* __restrict__ Jc,
                           int tid, int nt) {
  const double lT = log(Tc), iT = 1.0 / Tc, lKT = log(MX_KB * Tc / MX_P0);
  double* g = c.v;
  const double* cf = net.nasa + (Tc < MX_NASA_SPLIT_T ? 0 : net.ns * 9);
#pragma unroll 1
  for (int i = tid; i < net.ns; i += nt) g[i] = gibbs_rt(cf + 9 * i, Tc, lT, iT);
  if (tid == 0) g[net.ns] = 0.0;
  __syncthreads();
#pragma unroll 1
  for (int r = tid; r < net.nr; r += nt) {
    if (r >= net.nrt) {
      c.kf[r] = Jc[r - net.nrt];
      c.kr[r] = 0.0;
      continue;
    }
    const int fl = __ldg(net.rf + r);
    const uint64_t w = __ldg(net.rx8 + r);
    const int x0 = w & 255, x1 = (w >> 8) & 255, x2 = (w >> 16) & 255;
    const int x3 = (w >> 24) & 255, x4 = (w >> 32) & 255, x5 = (w >> 40) & 255;
    const double k = law(net.rc + 14 * r, fl, Tc, lT, iT, nd);
    const double dg = g[x3] + g[x4] + g[x5] - g[x0] - g[x1] - g[x2];
    const double c3 = (fl & FL_THREE_BODY) ? nd : 1.0;
    const double dmu = (double)(((fl >> 3) & 7) - 4);
    double kf = k * c3, kr = (k * exp(dg + dmu * lKT)) * c3;
    const int mf = (fl >> 10) & 3, mr = (fl >> 12) & 3;
    const bool tb = (fl & FL_THREE_BODY) != 0;
    const double q = fmax(bimolecular_rate(mf, tb, kf, nd), bimolecular_rate(mr, tb, kr, nd));
    if (q > MX_K_COLL) {
      const double cc = MX_K_COLL / q;
      kf *= cc;
      kr *= cc;
    }
    c.kf[r] = kf;
    c.kr[r] = kr;
  }
  if (tid == 0) c.kf[2 * net.nr] = 0.0;  // the zero rate of the Jacobian stream's padding
  __syncthreads();
}

// ---- right-hand side (rhs, common.cuh:282-353) ----

// A barrier over the threads of a group: named barrier id (0 is __syncthreads' own) over n threads.
__device__ __forceinline__ void group_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }

// S v's pieces into part: each thread of the group its pieces (ascending reactions) from its coalesced word stream, four
// words a load and the next four on their way; v[nr] = 0 pads. The four values are read before the first piece is
// written, which the compiler could not do by itself (a store between them may alias). Row i of S v is then
// part[sv_row_ptr[i]] + ... in order. What bounds it is the latency of the chain table word, v, fma, store: 69 species,
// one cell an SM, a right-hand side took 7,450 cycles and takes 4,430.
__device__ __forceinline__ void sv_pieces_of(const Net& net, const Cell& c, const double* v, int gtid, int gnt) {
  const int g = gnt == net.st_threads[0] ? 0 : 1;
  const uint4* __restrict__ sw = net.sv[g] + gtid;
  double s = 0.0;
  uint4 next = __ldg(sw);
#pragma unroll 1
  for (int q = net.sv_rounds[g]; q > 0; q -= 4) {
    const unsigned w[4] = {next.x, next.y, next.z, next.w};
    sw += gnt;
    next = __ldg(sw);
    double x[4];
#pragma unroll
    for (int k = 0; k < 4; k++) x[k] = v[w[k] & 0x7ffu];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      s = fma(code_coefficient(w[k] >> 11), x[k], s);
      if (w[k] & 0x2000u) {
        c.part[w[k] >> 16] = s;
        s = 0.0;
      }
    }
  }
}

// Row i of S v from its pieces, added in order.
__device__ __forceinline__ double sv_row(const Cell& c, int p0, int p1) {
  double r = c.part[p0];
#pragma unroll 1
  for (int p = p0 + 1; p < p1; p++) r += c.part[p];
  return r;
}
__device__ __forceinline__ double sv_row(const Net& net, const Cell& c, int i) {
  return sv_row(c, __ldg(net.sv_row_ptr + i), __ldg(net.sv_row_ptr + i + 1));
}

// F = (ntot / nd) S v(n) at Y, u0 = S v / nd into U when u0; n = nd Y / ntot. Returns ntot. Run by a group of whole
// warps (gtid its thread index, gnt its size, synchronised by named barrier bar); three barriers.
__device__ __forceinline__ double rhs(const Net& net, const Cell& c, const double* Y, bool u0, double nd, int gtid, int gnt, int bar) {
  const int lane = gtid & 31, ns = net.ns, nr = net.nr;
  // what this thread will read from the tables, on its way while the sum is formed
  const int p0 = gtid < ns ? __ldg(net.sv_row_ptr + gtid) : 0, p1 = gtid < ns ? __ldg(net.sv_row_ptr + gtid + 1) : 0;
  uint64_t w0 = gtid < nr ? __ldg(net.rx8 + gtid) : 0, w1 = gtid + gnt < nr ? __ldg(net.rx8 + gtid + gnt) : 0;
  const double ntot = lane_sum(Y, ns, lane), xf = nd / ntot, ixf = ntot / nd;
#pragma unroll 1
  for (int i = gtid; i < ns; i += gnt) c.n[i] = Y[i] * xf;
  if (gtid == 0) {
    c.n[ns] = 1.0;
    c.v[nr] = 0.0;
  }
  group_sync(bar, gnt);
  const double* n = c.n;
#pragma unroll 1
  for (int r = gtid; r < nr; r += 2 * gnt) {  // two reactions at a time, their values read before either is written
    const uint64_t u = w0, w = w1;
    const int r1 = r + gnt < nr ? r + gnt : r, r2 = r + 2 * gnt;
    if (r2 < nr) w0 = __ldg(net.rx8 + r2);
    if (r2 + gnt < nr) w1 = __ldg(net.rx8 + r2 + gnt);
    const double a0 = c.kf[r] * n[u & 255] * n[(u >> 8) & 255] * n[(u >> 16) & 255];
    const double b0 = c.kr[r] * n[(u >> 24) & 255] * n[(u >> 32) & 255] * n[(u >> 40) & 255];
    const double a1 = c.kf[r1] * n[w & 255] * n[(w >> 8) & 255] * n[(w >> 16) & 255];
    const double b1 = c.kr[r1] * n[(w >> 24) & 255] * n[(w >> 32) & 255] * n[(w >> 40) & 255];
    c.v[r] = a0 - b0;
    if (r1 > r) c.v[r1] = a1 - b1;
  }
  group_sync(bar, gnt);
  sv_pieces_of(net, c, c.v, gtid, gnt);
  group_sync(bar, gnt);
  // each row: its pieces added in order
#pragma unroll 1
  for (int i = gtid; i < ns; i += gnt) {
    const double r = i == gtid ? sv_row(c, p0, p1) : sv_row(net, c, i);
    c.F[i] = r * ixf;
    if (u0) c.U[i] = r / nd;
  }
  group_sync(bar, gnt);
  return ntot;
}

__device__ __forceinline__ double rhs(const Net& net, const Cell& c, const double* Y, bool u0, double nd, int tid,
                                      int nt) {
  return rhs(net, c, Y, u0, nd, tid, nt, 0);
}

// A = -Jn (dense, row stride ld), then U = u0 + (-Jn N) / ntot (call.cuh:61-79, jacobian_times_x). Three barriers.
__device__ __forceinline__ void jacobian_w(const Net& net, const Cell& c, double ntot, int tid, int nt) {
  const int ns = net.ns, ld = net.ld;
  double2* zero = (double2*)c.A;  // to the even count that the layout rounds the matrix to
#pragma unroll 4
  for (int i = tid; i < (ns * ld + 1) / 2; i += nt) zero[i] = make_double2(0.0, 0.0);
  __syncthreads();
  {  // each thread its entries from its coalesced word stream, four terms a load (the padding words use the zero rate
     // kf[2 nr]); the four products are formed before the first entry is written. A term at a time, each waiting for
     // the store before it, the Jacobian and w of 69 species took 14,800 cycles on one cell an SM; 6,800 so.
    const uint4* __restrict__ jw = net.jt + tid;
    const uint2* __restrict__ jd = net.jd + tid;
    double acc = 0.0;
    uint4 next = __ldg(jw);
    uint2 next_to = __ldg(jd);
#pragma unroll 1
    for (int q = net.jac_rounds; q > 0; q -= 4) {
      const unsigned w[4] = {next.x, next.y, next.z, next.w};
      const unsigned to[4] = {next_to.x & 0xffffu, next_to.x >> 16, next_to.y & 0xffffu, next_to.y >> 16};
      jw += nt;
      jd += nt;
      next = __ldg(jw);
      next_to = __ldg(jd);
      double pr[4];
#pragma unroll
      for (int k = 0; k < 4; k++) pr[k] = c.kf[w[k] & 0xfffu] * c.n[(w[k] >> 16) & 255u] * c.n[w[k] >> 24];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        acc = fma(code_coefficient(w[k] >> 12), pr[k], acc);
        if (w[k] & 0x4000u) {
          c.A[to[k]] = -acc;
          acc = 0.0;
        }
      }
    }
  }
  __syncthreads();
#pragma unroll 1
  for (int i = tid; i < ns; i += nt) {
    const double* a = c.A + i * ld;
    double acc = 0.0;
#pragma unroll 8
    for (int j = 0; j < ns; j++) acc = fma(a[j], c.N[j], acc);
    c.U[i] = c.U[i] + acc / ntot;
  }
  __syncthreads();
}

// ---- the LU without exchanges, on the matrix pipe ----
// Every entry receives its updates A_ij <- fma(-l_ik, A_kj, A_ij) in ascending k, l_ik = A_ik / A_kk taken as
// A_ik * (1 / A_kk): the order and the operations of the right-looking LU, so the bits of the sparse factorisation
// on the fill pattern (call.cuh:81-112) for finite data. Blocked by 8, with the trailing update as FP64 matrix
// instructions. mma.m8n8k4 adds its four products to an entry one after the other in ascending k, each a correctly
// rounded fma: measured equal to the fma chain on 786,432 random entries over 24 binary orders of magnitude, at the
// FP64 pipe's full rate (36.8 TFLOP/s). One instruction does the work of 8 warp-wide fma's, and an 8 x 8 tile needs 8
// shared accesses a lane for 512 fma's.
// Per block: the rows below it (L) on half of the warps and the columns right of it (U) on the other half, one lane
// each, in registers; then warp 0 updates and factors the next diagonal block while the other warps update the rest.
// What bounds it is the chain of the diagonal blocks (69 pivots of a reciprocal, a product, an fma and a shuffle) and
// shared-memory bandwidth: 69 species, 26,300 cycles with one cell an SM, 39,900 with four that all factor at once (a
// factorisation in 4 x 4 register tiles 60,000 and 76,500). The loops are kept rolled where they can be: the whole try
// is 60 KB of code, and unrolled forms that are faster alone (the diagonal block's pivots, 8-pivot solves) made the
// call 13 % slower with four cells an SM, by instruction fetch.

// c (8 x 8: lane 4 g + t holds row g, columns 2 t and 2 t + 1) += a (8 x 4: row g, column t) b (4 x 8: row t, column g)
__device__ __forceinline__ void mma_f64(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};" : "+d"(c0), "+d"(c1) : "d"(a), "d"(b));
}

__device__ __forceinline__ void pair_from(const double* p, double& a, double& b) {
  a = p[0];
  b = p[1];
}
__device__ __forceinline__ void pair_to(double* p, double a, double b) {
  p[0] = a;
  p[1] = b;
}

// The LU of an 8 x 8 block (its first nb rows and columns) held as mma_f64 holds c, on one warp; 1 / pivot to dinv.
// The chain from pivot to pivot is a reciprocal, a product and an fma: every lane forms the next pivot alike from
// values gathered while the reciprocal is under way. An entry that takes no update uses a multiplier or a pivot row's
// entry of 0, and fma(-0, u, x) = x for finite u.
__device__ __forceinline__ void lu_diagonal(double& x0, double& x1, double* dinv, int nb, int lane) {
  const int g = lane >> 2, t = lane & 3;
  double piv = __shfl_sync(FULL, x0, 0);
  // one pivot k, in column 2 q + S: a the entries of its column's parity, b of the next column's (in lanes t == n)
  auto pivot = [&](int k, int q, int n, double& a, double& b, bool odd) {
    const double below = __shfl_sync(FULL, a, 4 * k + 4 + q), right = __shfl_sync(FULL, b, 4 * k + n);
    const double next = __shfl_sync(FULL, b, 4 * k + 4 + n), col = __shfl_sync(FULL, a, 4 * g + q);
    const double u0 = __shfl_sync(FULL, x0, 4 * k + t), u1 = __shfl_sync(FULL, x1, 4 * k + t);
    const double d = __drcp_rn(piv);
    piv = fma(-(below * d), right, next);
    const double l = col * d, m = g > k ? l : 0.0;
    x0 = fma(-m, t > q ? u0 : 0.0, x0);
    x1 = fma(-m, t > q || (t == q && !odd) ? u1 : 0.0, x1);
    if (t == q && g > k) a = l;
    if (lane == 0) dinv[k] = d;
  };
#pragma unroll 1
  for (int q = 0; 2 * q < nb; q++) {
    pivot(2 * q, q, q, x0, x1, false);
    if (2 * q + 1 < nb) pivot(2 * q + 1, q, q + 1, x1, x0, true);
  }
}

// The block kb .. kb + 7 of L and U applied to the trailing tiles of tile rows first, first + step, ... (without_first:
// all but the first tile of tile row 0) on one warp.
__device__ __forceinline__ void trailing_tiles(double* A, int ld, int kb, int ns, int first, int step,
                                               bool without_first, int lane) {
  const int ke = kb + 8, m = (ns - ke + 7) >> 3, g = lane >> 2, t = lane & 3;
#pragma unroll 1
  for (int ti = first; ti < m; ti += step) {
    const int r0 = ke + 8 * ti + g;
    const double* la = A + r0 * ld + kb + t;
    const double a0 = -la[0], a1 = -la[4];
    const double* ub = A + (kb + t) * ld + ke + g;
    double* cp = A + r0 * ld + ke + 2 * t;
    int left = ns - ke - 2 * t;  // columns from the lane's first one on
    if (r0 >= ns) left = 0;
    int tj = 0;
    if (without_first && ti == 0) {
      tj = 1;
      ub += 8;
      cp += 8;
      left -= 8;
    }
#pragma unroll 1
    for (; tj < m; tj += 2) {
      double c0, c1, e0, e1;
      pair_from(cp, c0, c1);
      pair_from(cp + 8, e0, e1);
      const double b0 = ub[0], f0 = ub[8], b1 = ub[4 * ld], f1 = ub[4 * ld + 8];
      mma_f64(c0, c1, a0, b0);
      mma_f64(e0, e1, a0, f0);
      mma_f64(c0, c1, a1, b1);
      mma_f64(e0, e1, a1, f1);
      if (left > 1) pair_to(cp, c0, c1);
      else if (left > 0) cp[0] = c0;
      if (left > 9) pair_to(cp + 8, e0, e1);
      else if (left > 8) cp[8] = e0;
      ub += 16;
      cp += 16;
      left -= 16;
    }
  }
}

// Reads past the matrix's last row or column (a tile's rest) stay inside the cell's shared memory, whose layout keeps
// (ns + 8) ld + 16 doubles from oA on; such rows and columns of a tile are not written.
template <int W>
__device__ __noinline__ void lu_mma(int ns, int ld, int oA, int oD, int tid) {
  extern __shared__ double smem[];
  double* A = smem + oA;
  double* dinv = smem + oD;
  const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
#pragma unroll 1
  for (int kb = -8; kb + 8 < ns; kb += 8) {  // the first round only factors the first diagonal block
    const int ke = kb + 8;
    const double* D = A + kb * ld + kb;
    if (kb < 0) {
    } else if (warp < W / 2) {  // L: row i of the block's columns times U^-1
#pragma unroll 1
      for (int i = ke + tid; i < ns; i += 16 * W) {
        double* r = A + i * ld + kb;
        double x[8];
#pragma unroll
        for (int j = 0; j < 8; j += 2) pair_from(r + j, x[j], x[j + 1]);
#pragma unroll
        for (int k = 0; k < 8; k++) {
          x[k] *= dinv[kb + k];
          double u[8];
#pragma unroll
          for (int j = (k + 1) & ~1; j < 8; j += 2) pair_from(D + k * ld + j, u[j], u[j + 1]);
#pragma unroll
          for (int j = k + 1; j < 8; j++) x[j] = fma(-x[k], u[j], x[j]);
        }
#pragma unroll
        for (int j = 0; j < 8; j += 2) pair_to(r + j, x[j], x[j + 1]);
      }
    } else {  // U: column j of the block's rows, L^-1 times it
#pragma unroll 1
      for (int j = ke + tid - 16 * W; j < ns; j += 16 * W) {
        double* cj = A + kb * ld + j;
        double x[8];
#pragma unroll
        for (int s = 0; s < 8; s++) x[s] = cj[s * ld];
#pragma unroll
        for (int s = 1; s < 8; s++) {
          double l[8];
#pragma unroll
          for (int k = 0; k < s; k += 2) pair_from(D + s * ld + k, l[k], l[k + 1]);
#pragma unroll
          for (int k = 0; k < s; k++) x[s] = fma(-l[k], x[k], x[s]);
          cj[s * ld] = x[s];
        }
      }
    }
    __syncthreads();
    // the trailing tiles: warp 0 the first one (the next diagonal block), the other warps the rest by tile rows
    if (warp == 0) {
      double* cp = A + (ke + g) * ld + ke + 2 * t;
      double c0, c1;
      pair_from(cp, c0, c1);
      if (kb >= 0) {
        const double* la = A + (ke + g) * ld + kb + t;
        const double* ub = A + (kb + t) * ld + ke + g;
        mma_f64(c0, c1, -la[0], ub[0]);
        mma_f64(c0, c1, -la[4], ub[4 * ld]);
      }
      const int nb = min(8, ns - ke);
      lu_diagonal(c0, c1, dinv + ke, nb, lane);
      if (g < nb && 2 * t < nb) cp[0] = c0;
      if (g < nb && 2 * t + 1 < nb) cp[1] = c1;
    } else if (kb >= 0) {
      trailing_tiles(A, ld, kb, ns, warp - 1, W - 1, true, lane);
    }
    __syncthreads();
  }
}

// the LU of A into A and dinv by the cell's W warps
template <int W>
__device__ __forceinline__ void lu(const Net& net, double* A, double* dinv, int tid) {
  extern __shared__ double smem[];
  lu_mma<W>(net.ns, net.ld, (int)(A - smem), (int)(dinv - smem), tid);
}

// value a[p] for p = idx (R known at compile time: no local memory)
template <int R>
__device__ __forceinline__ double pick(const double (&a)[R], int idx) {
  double v = a[0];
#pragma unroll
  for (int p = 1; p < R; p++)
    if (idx == p) v = a[p];
  return v;
}

// y <- M0^-1 y on one warp with the factors of the LU: lane l holds rows l + 32 p. Forward unit
// L in ascending k, U in descending k with x_k = a_k / U_kk (msolve, common.cuh:504-522). Each entry receives the
// one-pivot sweep's fma's in its order, four pivots at a time: their four values are gathered from their lanes, every
// lane solves the 4 x 4 block alike (its entries are broadcast reads) and applies the four to its rows, so four
// pivots cost one shuffle latency instead of four; the matrix's last rows past a multiple of four go one by one. One
// warp issues it, so its instructions and their latencies are the time: 8,600 cycles at 69 species, one pivot at a time
// 10,700.
// Not inlined: the call kernel solves at four places, and one copy of the code keeps the instruction cache warm; the
// vector and the matrix are offsets into shared memory, so that its accesses stay shared ones.
// With oU >= 0 the Sherman-Morrison correction of W = M0 - w 1^T follows (sherman's operations).
template <int R>
__device__ __noinline__ void lu_solve_at(int ns, int ld, int oA, int oD, int oY, int oU, double c0, int lane) {
  extern __shared__ double smem[];
  const double* A = smem + oA;
  const double* dinv = smem + oD;
  double* y = smem + oY;
  const int last = ns - 1, tail = ns & ~3;  // pivots tail .. last one by one
  double a[R], d[R];
  const double* row[R];
#pragma unroll
  for (int p = 0; p < R; p++) {
    const int i = min(lane + 32 * p, last);
    row[p] = A + i * ld;
    d[p] = dinv[i];
    a[p] = y[i];
  }
  const double* dg = A;  // the block's diagonal
#pragma unroll
  for (int c = 0; c < R; c++) {  // forward: rows 32 c .. 32 c + 31
    const int nb = min(32, tail - 32 * c);
#pragma unroll 1
    for (int b = 0; b < nb; b += 4) {
      const int k = 32 * c + b;
      const double *d1 = dg + ld, *d2 = d1 + ld, *d3 = d2 + ld;
      const double l10 = d1[0], l20 = d2[0], l21 = d2[1], l30 = d3[0], l31 = d3[1], l32 = d3[2];
      double l[R][4], g[4];
#pragma unroll
      for (int s = 0; s < 4; s++) g[s] = __shfl_sync(FULL, a[c], b + s);
#pragma unroll
      for (int p = c; p < R; p++)
#pragma unroll
        for (int s = 0; s < 4; s++) l[p][s] = row[p][k + s];
      g[1] = fma(-l10, g[0], g[1]);
      g[2] = fma(-l20, g[0], g[2]);
      g[3] = fma(-l30, g[0], g[3]);
      g[2] = fma(-l21, g[1], g[2]);
      g[3] = fma(-l31, g[1], g[3]);
      g[3] = fma(-l32, g[2], g[3]);
#pragma unroll
      for (int s = 0; s < 4; s++)
#pragma unroll
        for (int p = c; p < R; p++)
          if (p > c || lane > b + s) a[p] = fma(-l[p][s], g[s], a[p]);
      dg = d3 + ld + 4;
    }
    if (R <= 4 ? c == R - 1 : c == last >> 5) {
#pragma unroll 1
      for (int k = tail; k < last; k++) {
        const double yk = __shfl_sync(FULL, a[c], k & 31);
        if (lane > (k & 31)) a[c] = fma(-row[c][k], yk, a[c]);
      }
    }
  }
#pragma unroll
  for (int c = R - 1; c >= 0; c--) {  // backward: rows 32 c + 31 .. 32 c
    if (R <= 4 ? c == R - 1 : c == last >> 5) {
#pragma unroll 1
      for (int k = last; k >= tail; k--) {
        const double z = __shfl_sync(FULL, a[c] * d[c], k & 31);
#pragma unroll
        for (int p = 0; p <= c; p++)
          if (p < c || lane < (k & 31)) a[p] = fma(-row[p][k], z, a[p]);
      }
    }
    const int nb = min(32, tail - 32 * c);
#pragma unroll 1
    for (int q = 4; q <= nb; q += 4) {
      const int b = nb - q, k = 32 * c + b;
      dg -= 4 * ld + 4;
      const double *e1 = dg + ld, *e2 = e1 + ld;
      const double u01 = dg[1], u02 = dg[2], u03 = dg[3], u12 = e1[2], u13 = e1[3], u23 = e2[3];
      const double d0 = dinv[k], d1 = dinv[k + 1], d2 = dinv[k + 2], d3 = dinv[k + 3];
      double u[R][4], g[4];
#pragma unroll
      for (int s = 0; s < 4; s++) g[s] = __shfl_sync(FULL, a[c], b + s);
#pragma unroll
      for (int p = 0; p <= c; p++)
#pragma unroll
        for (int s = 0; s < 4; s++) u[p][s] = row[p][k + s];
      double z[4];
      z[3] = g[3] * d3;
      z[2] = fma(-u23, z[3], g[2]) * d2;
      z[1] = fma(-u12, z[2], fma(-u13, z[3], g[1])) * d1;
      z[0] = fma(-u01, z[1], fma(-u02, z[2], fma(-u03, z[3], g[0]))) * d0;
#pragma unroll
      for (int s = 3; s >= 0; s--)
#pragma unroll
        for (int p = 0; p <= c; p++)
          if (p < c || lane < b + s) a[p] = fma(-u[p][s], z[s], a[p]);
    }
  }
#pragma unroll
  for (int p = 0; p < R; p++) a[p] *= d[p];
  if (oU >= 0) {
    const double* u = smem + oU;
    double s = 0.0;
#pragma unroll
    for (int p = 0; p < R; p++)
      if (lane + 32 * p < ns) s += a[p];
    s = warp_sum(s) * c0;
#pragma unroll
    for (int p = 0; p < R; p++) a[p] = fma(s, u[min(lane + 32 * p, last)], a[p]);
  }
  __syncwarp();
#pragma unroll
  for (int p = 0; p < R; p++)
    if (lane + 32 * p < ns) y[lane + 32 * p] = a[p];
  __syncwarp();
}

template <int R>
__device__ __forceinline__ void lu_solve(const Net& net, const double* A, const double* dinv, double* y, int lane) {
  extern __shared__ double smem[];
  lu_solve_at<R>(net.ns, net.ld, (int)(A - smem), (int)(dinv - smem), (int)(y - smem), -1, 0.0, lane);
}

// y <- W^-1 y on one warp: the solve and the Sherman-Morrison correction with u = M0^-1 w and c0 = 1 / (1 - sum u)
template <int R>
__device__ __forceinline__ void w_solve(const Net& net, const double* A, const double* dinv, double* y, const double* u,
                                        double c0, int lane) {
  extern __shared__ double smem[];
  lu_solve_at<R>(net.ns, net.ld, (int)(A - smem), (int)(dinv - smem), (int)(y - smem), (int)(u - smem), c0, lane);
}

// y <- y + c0 (sum y) u on one warp (sherman_morrison_update, common.cuh:542-557)
__device__ __forceinline__ void sherman(const Net& net, double* y, const double* u, double c0, int lane) {
  const double s = lane_sum(y, net.ns, lane) * c0;
#pragma unroll 1
  for (int i = lane; i < net.ns; i += 32) y[i] = fma(s, u[i], y[i]);
  __syncwarp();
}

// ---- the recovery's dense LU with threshold partial pivoting (recover.cuh:7-82) ----

// On one warp, for more rows a lane than the blocked form's registers hold.
__device__ __forceinline__ void dense_lu_pivot(const Net& net, double* A, double* dinv, int* pr, int lane) {
  const int ns = net.ns, ld = net.ld;
#pragma unroll 1
  for (int i = lane; i < ns; i += 32) pr[i] = i;
  __syncwarp();
  for (int k = 0; k < ns; k++) {
    double best = -1.0;
    int bi = ns;
#pragma unroll 1
    for (int i = k + lane; i < ns; i += 32) {
      const double a = fabs(A[i * ld + k]);
      if (a > best) {
        best = a;
        bi = i;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double ob = __shfl_xor_sync(FULL, best, o);
      const int oi = __shfl_xor_sync(FULL, bi, o);
      if (ob > best || (ob == best && oi < bi)) {
        best = ob;
        bi = oi;
      }
    }
    const bool exchange = bi != ns && bi != k && !(fabs(A[k * ld + k]) >= MX_PIVTAU * best);
    __syncwarp();
    if (exchange) {
#pragma unroll 1
      for (int j = lane; j < ns; j += 32) {
        const double a = A[k * ld + j];
        A[k * ld + j] = A[bi * ld + j];
        A[bi * ld + j] = a;
      }
      if (lane == 0) {
        const int t = pr[k];
        pr[k] = pr[bi];
        pr[bi] = t;
      }
    }
    __syncwarp();
    const double dk = 1.0 / A[k * ld + k];
    if (lane == 0) dinv[k] = dk;
#pragma unroll 1
    for (int i = k + 1 + lane; i < ns; i += 32) {
      const double l = A[i * ld + k] * dk;
      A[i * ld + k] = l;
      for (int j = k + 1; j < ns; j++) A[i * ld + j] = fma(-l, A[k * ld + j], A[i * ld + j]);
    }
    __syncwarp();
  }
}

// The same factorisation (its exchanges, its operations in its order, so its bits) by the cell's W warps, 8 columns at a
// time: warp 0 factors the 8 columns in registers (lane l holds rows l + 32 p, the pivot's column in x[.][0]; they move
// down by one per pivot), the other columns take its exchanges and their rows of U, one lane each, and the trailing
// tiles run on the matrix instructions as lu_mma's. A recovery is a chain of thousands of tries of a few cells, so its
// latency is what the call waits for: 1,000 cells of 41 species over 1e10 s, 19 of them recovered, took 116 ms with one
// warp eliminating an element at a time, 80 ms so.
template <int W, int R>
__device__ __noinline__ void dense_lu_at(int ns, int ld, int oA, int oD, int oP, int oX, int tid) {
  extern __shared__ double smem[];
  double* A = smem + oA;
  double* dinv = smem + oD;
  int* pr = (int*)smem + oP;
  int* from = (int*)(smem + oX);  // the row that each pivot of the block came from [8]
  const int lane = tid & 31, warp = tid >> 5;
#pragma unroll 1
  for (int i = tid; i < ns; i += 32 * W) pr[i] = i;
  __syncthreads();
#pragma unroll 1
  for (int kb = 0; kb < ns; kb += 8) {
    const int nb = min(8, ns - kb), ke = kb + nb;
    if (warp == 0) {
      double x[R][8];
#pragma unroll
      for (int p = 0; p < R; p++) {
        const int i = lane + 32 * p;
#pragma unroll
        for (int j = 0; j < 8; j++) x[p][j] = i >= kb && i < ns && j < nb ? A[i * ld + kb + j] : 0.0;
      }
#pragma unroll 1
      for (int k = 0; k < nb; k++) {
        const int row = kb + k;
        double best = -1.0, own[R], u[8], w[8];
        int bi = ns;
#pragma unroll
        for (int p = 0; p < R; p++) {
          const int i = lane + 32 * p;
          const double v = fabs(x[p][0]);
          if (i >= row && i < ns && v > best) {
            best = v;
            bi = i;
          }
          own[p] = x[p][0];
        }
        {  // the largest magnitude over the warp, ties to the lower row; a NaN is never taken
          const unsigned long long bits = bi < ns ? __double_as_longlong(best) : 0ull;
          const unsigned hi = (unsigned)(bits >> 32), lo = (unsigned)bits;
          const unsigned mh = __reduce_max_sync(FULL, hi);
          const unsigned ml = __reduce_max_sync(FULL, hi == mh ? lo : 0u);
          bi = __reduce_min_sync(FULL, bi < ns && hi == mh && lo == ml ? bi : ns);
          best = bi < ns ? __longlong_as_double((long long)((unsigned long long)mh << 32 | ml)) : -1.0;
        }
        const double akk = __shfl_sync(FULL, pick<R>(own, row >> 5), row & 31);
        const bool exchange = bi != ns && bi != row && !(fabs(akk) >= MX_PIVTAU * best);
        const int src = exchange ? bi : row;
#pragma unroll
        for (int j = 0; j < 8; j++) {
          double c[R];
#pragma unroll
          for (int p = 0; p < R; p++) c[p] = x[p][j];
          u[j] = __shfl_sync(FULL, pick<R>(c, src >> 5), src & 31);
          if (exchange) w[j] = __shfl_sync(FULL, pick<R>(c, row >> 5), row & 31);
        }
        if (exchange) {
#pragma unroll
          for (int p = 0; p < R; p++)
#pragma unroll
            for (int j = 0; j < 8; j++) {
              if (lane + 32 * p == row) x[p][j] = u[j];
              if (lane + 32 * p == bi) x[p][j] = w[j];
            }
          if (lane < k) {  // the block's finished columns
            double *a0 = A + row * ld + kb + lane, *a1 = A + bi * ld + kb + lane;
            const double a = *a0;
            *a0 = *a1;
            *a1 = a;
          }
          if (lane == 8) {
            const int q = pr[row];
            pr[row] = pr[bi];
            pr[bi] = q;
          }
          __syncwarp();
        }
        const double d = __drcp_rn(u[0]);
#pragma unroll
        for (int p = 0; p < R; p++) {
          const int i = lane + 32 * p;
          const double l = x[p][0] * d;
          if (i >= kb && i < ns) A[i * ld + row] = i > row ? l : x[p][0];
#pragma unroll
          for (int j = 1; j < 8; j++) x[p][j - 1] = i > row ? fma(-l, u[j], x[p][j]) : x[p][j];
          x[p][7] = 0.0;
        }
        if (lane == 0) {
          dinv[row] = d;
          from[k] = src;
        }
        __syncwarp();
      }
    }
    __syncthreads();
#pragma unroll 1
    for (int q = tid; q < ns - nb; q += 32 * W) {  // the other columns: the exchanges, and right of the block U's rows
      const int j = q < kb ? q : q + nb;
      double* cj = A + j;
#pragma unroll 1
      for (int k = 0; k < nb; k++) {
        const int s = from[k];
        if (s != kb + k) {
          const double a = cj[(kb + k) * ld];
          cj[(kb + k) * ld] = cj[s * ld];
          cj[s * ld] = a;
        }
      }
      if (j >= ke) {
        const double* D = A + kb * ld + kb;
        double x[8];
#pragma unroll
        for (int s = 0; s < 8; s++) x[s] = cj[(kb + s) * ld];
#pragma unroll
        for (int s = 1; s < 8; s++) {
#pragma unroll
          for (int k = 0; k < s; k++) x[s] = fma(-D[s * ld + k], x[k], x[s]);
          cj[(kb + s) * ld] = x[s];
        }
      }
    }
    __syncthreads();
    if (ke < ns) trailing_tiles(A, ld, kb, ns, warp, W, false, lane);
    __syncthreads();
  }
}

// P A = L U of the dense W by the cell's W warps: A, dinv (1 / U_kk) and pr; c.red is scratch
template <int W, int R>
__device__ __forceinline__ void dense_lu(const Net& net, const Cell& c, int* pr, int tid) {
  if constexpr (R <= 4) {
    extern __shared__ double smem[];
    dense_lu_at<W, R>(net.ns, net.ld, (int)(c.A - smem), (int)(c.dinv - smem), (int)(pr - (int*)smem),
                      (int)(c.red - smem), tid);
  } else {
    if (tid < 32) dense_lu_pivot(net, c.A, c.dinv, pr, tid);
    __syncthreads();
  }
}

// y <- W^-1 y with the factors of dense_lu on one warp: its rows in the exchanges' order, then lu_solve's sweeps
template <int R>
__device__ __forceinline__ void dense_solve(const Net& net, const double* A, const double* dinv, const int* pr, double* y,
                                            int lane) {
  double a[R];
#pragma unroll
  for (int p = 0; p < R; p++) a[p] = lane + 32 * p < net.ns ? y[pr[lane + 32 * p]] : 0.0;
  __syncwarp();
#pragma unroll
  for (int p = 0; p < R; p++)
    if (lane + 32 * p < net.ns) y[lane + 32 * p] = a[p];
  __syncwarp();
  lu_solve<R>(net, A, dinv, y, lane);
}

// ---- step control (common.cuh:90-133) ----

struct StepState {
  double h, t, nok, pen, pha;
  bool prej;
};

__device__ __forceinline__ double step_factor(double en, bool ok, bool prej, double pen, double pha, double ha) {
  const bool efin = isfinite(en);
  double fac = efin ? MX_STEP_SAFETY / cbrt(fmax(en, MX_ERR_FLOOR)) : MX_FAC_NONFINITE;
  fac = fmin(fmax(fac, ok ? MX_FACACC : MX_FACREJ), MX_FACMAX);
  if (!ok && efin && prej && en > 1.0 && pen > 1.0 && pha > ha) {
    const double pe = log(pen / en) / log(pha / ha);
    fac = pe > MX_SECANT_MIN_ORDER
              ? fmax(pow(MX_SECANT_TARGET / en, 1.0 / fmin(pe, MX_SECANT_MAX_ORDER)), MX_SECMIN)
              : MX_SECMIN;
  }
  if (!ok) fac = fmin(fac, MX_FAC_AFTER_REJECT);
  return fac;
}

// err of a try on warp 0 (try_error, common.cuh:570-590): Y = N + 2 K1 + K3 + K4; writes en and ok to red[0..1].
// Lane l takes rows l, l + 32, ..., R of them at most, whose divisions then run side by side.
template <int R>
__device__ __forceinline__ void try_error(const Net& net, const Cell& c, bool first, double rtol, double atol, int lane) {
  double q[R], e2 = 0.0, em = 0.0;
  bool nn = true;
#pragma unroll
  for (int p = 0; p < R; p++) {
    const int i = min(lane + 32 * p, net.ns - 1);
    const bool in = lane + 32 * p < net.ns;
    const double y = c.N[i] + 2.0 * c.K1[i] + c.K3[i] + c.K4[i];
    if (in) c.Y[i] = y;
    const double sc = fma(rtol, fmax(fabs(c.N[i]), fabs(y)), atol);
    q[p] = in ? c.K4[i] / sc : 0.0;
    nn = nn && (!in || y >= -atol);
  }
#pragma unroll
  for (int p = 0; p < R; p++) {
    e2 = fma(q[p], q[p], e2);
    em = fmax(em, fabs(q[p]));
  }
  const double er = sqrt(warp_sum(e2) / net.ns), emx = warp_max(em);
  const double en = (first && isfinite(er)) ? fmax(er, emx) : er;
  const bool ok = (en <= 1.0) && __all_sync(FULL, nn) && isfinite(en);
  if (lane == 0) {
    c.red[0] = en;
    c.red[1] = ok ? 1.0 : 0.0;
  }
}

// ---- the guard's test (guard.cuh:13-108), on one warp ----
// Sums over species are formed as a warp forms them: lane l adds species l, l + 32, ... in order, then the butterfly.
// The small element system (at most MX_MAX_ELEMENTS) is factored by every lane alike from the butterflied sums.

// Doubles of shared scratch the guard needs (guard_scratch): e0 and e1, the element matrix, its first diagonal, the
// right side, lambda, the sum, and g per species.
__host__ __device__ constexpr int guard_scratch(int ns) {
  return 2 * MX_MAX_ELEMENTS + MX_MAX_ELEMENTS * MX_MAX_ELEMENTS + 3 * MX_MAX_ELEMENTS + 2 + ns;
}

// The guard's test of a stepped cell's result xo (network species order) against its input x0, on one warp: the bits
// GUARD_NONFINITE, GUARD_UNFINISHED, GUARD_DRIFT, 0 when it passed (guard.cuh:63-108). A passing result has its element
// shares put back in place (element_multipliers, guard.cuh:24-57): x' = x (1 + sum_e lambda_e a_ie), clamped,
// renormalised. Every sum runs over the species in network order, one lane per sum, as the reference's one thread
// per cell adds them, so each sum has the reference's bits. at: atoms [ns][nel]; scr: guard_scratch(ns) doubles of
// shared memory, free during the guard.
static __device__ __noinline__ int check_cell(const Net& net, const double* x0, double* xo, int done, double nok,
                                       double atol, int lane, const double* at, double* scr) {
  constexpr int ME = MX_MAX_ELEMENTS;
  const int ns = net.ns, nel = net.nel;
  double* se = scr;            // [2 ME]: e0, then e1 at ME
  double* m = se + 2 * ME;     // [ME][ME], upper triangle
  double* m0 = m + ME * ME;    // [ME]
  double* y = m0 + ME;         // [ME]
  double* lam = y + ME;        // [ME]
  double* sum_at = lam + ME;   // [2]
  double* g = sum_at + 2;      // [ns]
  if (lane < 2 * nel) {        // e0[e] on lanes 0..nel-1, e1[e] on lanes nel..2 nel-1 (guard.cuh:70-77)
    const int e = lane < nel ? lane : lane - nel;
    const double* xs = lane < nel ? x0 : xo;
    double acc = 0.0;
    for (int i = 0; i < ns; i++) acc = fma(at[i * nel + e], xs[i], acc);
    se[lane < nel ? e : ME + e] = acc;
  }
  bool fin = true;
#pragma unroll 1
  for (int i = lane; i < ns; i += 32) fin = fin && isfinite(xo[i]);
  const bool xfin = __all_sync(FULL, fin);
  __syncwarp();
  double s0 = 0.0, s1 = 0.0;
  for (int e = 0; e < nel; e++) {
    s0 += se[e];
    s1 += se[ME + e];
  }
  bool drift = false;  // shares_drifted (guard.cuh:13-21)
  for (int e = 0; e < nel; e++)
    drift = drift || fabs(se[ME + e] / s1 - se[e] / s0) > net.drift * se[e] / s0 + 2.0 * atol * nok * net.etot / s0;
  const int c = (xfin ? 0 : GUARD_NONFINITE) | (done ? 0 : GUARD_UNFINISHED) | (drift ? GUARD_DRIFT : 0);
  if (c) return c;
  // (A X A^T)[e][f], f >= e: over species with a_ie and a_if both nonzero (guard.cuh:29-37)
#pragma unroll 1
  for (int q = lane; q < nel * nel; q += 32) {
    const int e = q / nel, f = q - e * nel;
    if (f >= e) {
      double acc = 0.0;
      for (int i = 0; i < ns; i++) {
        const double ae = at[i * nel + e], af = at[i * nel + f];
        if (ae != 0.0 && af != 0.0) acc = fma(ae * af, xo[i], acc);
      }
      m[e * ME + f] = acc;
    }
  }
  __syncwarp();
  if (lane == 0) {  // LDL^T and the back substitution; an element whose pivot vanishes is left out (guard.cuh:38-56)
    const double r = s1 / s0;
    for (int e = 0; e < nel; e++) {
      m0[e] = m[e * ME + e];
      y[e] = fma(se[e], r, -se[ME + e]);
    }
    for (int k = 0; k < nel; k++) {
      if (!(m[k * ME + k] > MX_ELEMENT_PIVOT_MIN * m0[k])) continue;
      for (int j = k + 1; j < nel; j++) {
        const double l = m[k * ME + j] / m[k * ME + k];
        for (int f = j; f < nel; f++) m[j * ME + f] = fma(-l, m[k * ME + f], m[j * ME + f]);
        y[j] = fma(-l, y[k], y[j]);
      }
    }
    for (int k = nel - 1; k >= 0; k--) {
      lam[k] = 0.0;
      if (!(m[k * ME + k] > MX_ELEMENT_PIVOT_MIN * m0[k])) continue;
      double b = y[k];
      for (int f = k + 1; f < nel; f++) b = fma(-m[k * ME + f], lam[f], b);
      lam[k] = b / m[k * ME + k];
    }
  }
  __syncwarp();
#pragma unroll 1
  for (int i = lane; i < ns; i += 32) {  // g per species (guard.cuh:94-99)
    double gi = 1.0;
    for (int e = 0; e < nel; e++) {
      const double a = at[i * nel + e];
      if (a != 0.0) gi = fma(lam[e], a, gi);
    }
    g[i] = fmin(fmax(gi, 1.0 - MX_GMAX), 1.0 + MX_GMAX);
  }
  __syncwarp();
  if (lane == 0) {  // the sum of x g in network order (guard.cuh:100)
    double sum = 0.0;
    for (int i = 0; i < ns; i++) sum = fma(xo[i], g[i], sum);
    sum_at[0] = sum;
  }
  __syncwarp();
  const double sum = sum_at[0];
#pragma unroll 1
  for (int i = lane; i < ns; i += 32) xo[i] *= g[i];
  __syncwarp();
  if (!(isfinite(sum) && sum > 0.0)) return GUARD_NONFINITE;
  const double is = 1.0 / sum;
#pragma unroll 1
  for (int i = lane; i < ns; i += 32) xo[i] *= is;
  __syncwarp();
  return 0;
}

// The guard's inputs into the matrix's space, free once the steps are done: atoms [ns][nel] and the cell's input row,
// so the guard's species sums read shared memory. Falls back to global memory when they do not fit.
__device__ __forceinline__ void stage_guard_inputs(const Net& net, const Cell& c, const double* x0, int tid, int nt,
                                                   const double** at, const double** xin) {
  const int ns = net.ns, na = ns * net.nel;
  if (na + ns > net.a_doubles) return;
#pragma unroll 1
  for (int e = tid; e < na; e += nt) c.A[e] = __ldg(net.atoms + e);
#pragma unroll 1
  for (int i = tid; i < ns; i += nt) c.A[na + i] = x0[i];
  *at = c.A;
  *xin = c.A + na;
}

}  // namespace mx
