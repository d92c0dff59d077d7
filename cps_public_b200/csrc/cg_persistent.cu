// cg_persistent.cu -- every iteration of an FP64 CG solve on a small lattice in
// one cooperative kernel.
//
// On lattices where one CG iteration is a few microseconds of device work (the
// Wilson 8^4 workload has 2048 sites per checkerboard), the launch-per-step
// loop of solver.cu is bound by launch and scheduling latency, not bandwidth.
// Here a single cooperative launch runs the iterations of DiracOp::InvCg
// (cps_pp/src/util/dirac_op/d_op_base/comsrc/inv_cg.C:293-364) until every
// right-hand side halts: the four hops of MatPcDagMatPc (the residual update
// r -= alpha A p, |r|^2 and x += alpha p fused into the last one, as in the
// launch-per-step loop), then p = r + beta p, separated by grid barriers.
// Every block keeps its own copy of the recurrence scalars (CgState) in shared
// memory and sums the per-block partials of each reduction in the same order, so
// all blocks hold identical scalars and take the same branches; block 0
// writes the state back when the loop ends.  Fields written inside the launch
// are read through L2 (ld.global.cg), never through the read-only cache.
//
// Two forms.  On fields of at most PCG_DP_SITES entries (all right-hand sides)
// the hops run with eight lanes per entry and the direction update rides on the
// next iteration's first two hops, so an iteration is four hops and four grid
// barriers; it beats the device-side graph loop of solver.cu there and is the default
// (figures at PCG_AUTO_SITES, host.h).  Larger fields run the column hop of
// hop_kernel plus a p-update phase (five barriers), slower than the graph loop
// (Wilson 8^2x10x16: 4.0 against 2.7 ms per solve), only when asked for.
//
// Grid barriers spin on an arrival counter with a time limit: a wait that
// runs out sets the error flag, every other block leaves at its next wait, and
// the host reports the error.  The cooperative launch keeps all blocks
// resident, so the barriers complete in normal operation.
#include <string.h>

#include "host.h"
#include "hop.cuh"

namespace cpsb {

// Threads per block: 128, or 32 for single-slice columns (Wilson), so that a
// unit is 32 columns whose link table fits shared memory and a small lattice
// still spreads over many SMs.
constexpr int PCG_NT_MAX = 128;
// Fields (all right-hand sides) of at most this many entries use the
// direction-parallel hop phases (the largest bound of the automatic mode).
constexpr long PCG_DP_SITES = PCG_AUTO_SITES;
// Longest barrier wait before it gives up (ns of the global timer): far above a
// phase of any lattice the loop takes, and above kernels of other streams that
// may hold SMs while the launch's blocks become resident.
constexpr unsigned long long PCG_WAIT_NS = 5000000000ull;

__device__ __forceinline__ unsigned long long pcg_now() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

struct PcgArgs {
  // the four hops of one iteration (in, out, x, cb, dag, a set per phase):
  // [0] t1 = D p, [1] t2 = p - kappa^2 D t1 with |t2|^2, [2] t1 = D^dag t2,
  // [3] A p = t2 - kappa^2 D^dag t1 consumed by the residual update
  DslashArgs ph[4];
  SpinorPtr r, p, x;
  CgState *S;
  double *partial;  // [nrhs][gridDim.x] block partials
  unsigned *bar;    // [0] arrivals, counted up over the whole launch
  int *err;         // set when a barrier wait ran out
};

// Grid barrier with a bounded wait; false (in every thread) when this block's
// wait ran out or another block has already reported one.  One counter that only
// grows: a block adds one and waits until all blocks of its `epoch`-th barrier have
// (a wrap-around of the counter is harmless, the difference is compared).  Two
// trips to L2 -- the add, and the poll that sees the last one -- where a
// generation word read before and written after the count makes it five.
__device__ __forceinline__ bool pcg_sync(const PcgArgs &P, unsigned &epoch) {
  __shared__ int ok;
  epoch++;
  __syncthreads();
  if (threadIdx.x == 0) {
    ok = 1;
    const unsigned want = epoch * gridDim.x;
    __threadfence();
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(P.bar) : "memory");
    unsigned seen;
    unsigned long long t0 = 0;
    for (unsigned n = 0;; n++) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(P.bar) : "memory");
      if ((int)(seen - want) >= 0) break;
      if ((n & 63u) == 63u) {  // the limit and the error flag, off the common path
        const unsigned long long now = pcg_now();
        if (!t0) t0 = now;
        if (*(volatile int *)P.err || now - t0 > PCG_WAIT_NS) {
          atomicExch(P.err, 1);
          ok = 0;
          break;
        }
      }
    }
    __threadfence();
  }
  __syncthreads();
  return ok != 0;
}

// One hop over every unit of the lattice (the FP64 branch of hop_kernel with one
// right-hand side per thread at a time).  MODE 0: out = D in; 1: out = x + a D in
// with |out|^2 into nrm; 2: A p = x + a D in, then r -= alpha A p, x_sol += alpha p
// and |r|^2 into nrm.
template <int NT, bool LC, bool DAG, int MODE>
__device__ __forceinline__ void pcg_hop(const DslashArgs &A, const PcgArgs &P, unsigned char *dsh, double *nrm,
                                        const int *skip, const double *alpha) {
  const Geom &g = A.g;
  const int C0 = g.cs[0];
  const int TX = NT / C0;
  const HopShm L = hop_shm(TX, NT, g.nrhs, true, LC);
  const int sp = threadIdx.x % C0;
  const int xl = threadIdx.x / C0;
  const int ntiles = (g.n4cb + TX - 1) / TX;
  const int nunits = ntiles * g.ncls;
  const unsigned per = (unsigned)g.n4cb * (unsigned)g.ls;
  for (int unit = blockIdx.x; unit < nunits; unit += gridDim.x) {
    const int k = unit % g.ncls, tile = unit / g.ncls;
    const int par_out = A.five_d ? ((1 - A.cb + k) & 1) : 1 - A.cb;
    __syncthreads();  // the previous unit is done with the tables
    load_unit<P64, LC>(A, tile, k, par_out, TX, NT, dsh);
    __syncthreads();
    const int xs = tile * TX + xl;
    const int C = g.cs[k];
    if (xl >= TX || xs >= g.n4cb || sp >= C) continue;
    HopCtx hc;
    entry_ctx<P64, LC>(hc, A, dsh, L, xl, xs, k, sp, par_out);
    const unsigned own = (k ? (unsigned)g.kb1 : 0u) + (unsigned)xs * (unsigned)C + (unsigned)sp;
    for (int q = 0; q < g.nrhs; q++) {
      if (skip[q]) continue;
      const unsigned rb = (unsigned)q * per;
      const unsigned i = rb + own;
      Spinor<double> acc = hop_entry_64<P64, LC, DAG, 1, true>(A, hc, rb);
      if (MODE == 0) {
        store_spinor<P64>(A.out, i, acc);
        continue;
      }
      const double a = A.a;
      const Spinor<double> xv = unpack64(load_raw64_l2(A.x, i));
#pragma unroll
      for (int s2 = 0; s2 < 4; s2++)
#pragma unroll
        for (int r = 0; r < 3; r++) acc.c[s2][r] = xv.c[s2][r] + cscale(a, acc.c[s2][r]);
      if (MODE == 1) {
        store_spinor<P64>(A.out, i, acc);
        nrm[q * NT + threadIdx.x] += norm2(acc);
        continue;
      }
      const double al = alpha[q];
      Spinor<double> rv = unpack64(load_raw64_l2(P.r, i));
      const Spinor<double> pv = unpack64(load_raw64_l2(P.p, i));
      Spinor<double> sv = unpack64(load_raw64_l2(P.x, i));
#pragma unroll
      for (int s2 = 0; s2 < 4; s2++)
#pragma unroll
        for (int r = 0; r < 3; r++) sv.c[s2][r] = cscale(al, pv.c[s2][r]) + sv.c[s2][r];
      store_spinor<P64>(P.x, i, sv);
#pragma unroll
      for (int s2 = 0; s2 < 4; s2++)
#pragma unroll
        for (int r = 0; r < 3; r++) rv.c[s2][r] = rv.c[s2][r] - cscale(al, acc.c[s2][r]);
      store_spinor<P64>(P.r, i, rv);
      nrm[q * NT + threadIdx.x] += norm2(rv);
    }
  }
}

// The same phase with eight lanes per entry: lane d loads neighbour d and its
// link, multiplies, and leaves the half spinor U h in the shared-memory slots gsh
// (6 x NT double2); then lanes 0-3 each take one spin of the entry, sum the eight
// directions in order, add the 5th-direction term and run the epilogue on their
// three chunks.  All field loads through L2.  A phase is a chain of latencies, so
// nothing on it depends on the lane's direction by a branch (the eight directions
// differ in which chunks and link elements are loaded and in signs, chosen by
// address or select), the epilogue's operands are loaded before the neighbours, and
// the lattice indexes of a thread's first entry are made once per launch.
// Wilson 8^4, mass 0.1, to 1e-10 from host arrays: 2.43 -> 1.53 ms a solve against one
// branch per direction, lane 0 alone after the products and a generation barrier.
// PUPD folds the direction update p = r + beta p of the previous iteration in:
// MODE 0 forms each neighbour's r + beta p from r and the old p as it loads
// them, and MODE 1 forms its own entry's, stores it as the new p and uses it as
// the xpay input (one fused multiply-add per real in both, so the two agree).
struct Pcg8Idx {
  bool valid;
  unsigned own;   // entry within a right-hand side
  unsigned ni;    // neighbour entry of the lane's direction
  long lk;        // element 0 of the lane's link
  unsigned e5;    // lanes 0-3: entry of the 5th-direction neighbour at dag 0 / 1 of the lane's spin
  unsigned e5d;
  double f5, f5d;
};

__device__ __forceinline__ Pcg8Idx pcg8_index(const DslashArgs &A, int cb, long e, int d) {
  const Geom &g = A.g;
  Pcg8Idx r;
  r.valid = e < (long)g.n4cb * g.ls;
  r.own = r.valid ? (unsigned)e : 0u;  // lanes beyond the field work on entry 0 and drop it
  const int k = (g.ncls == 2 && r.own >= (unsigned)g.kb1) ? 1 : 0;
  const int C = g.cs[k];
  const unsigned rem = r.own - (k ? (unsigned)g.kb1 : 0u);
  const int x = (int)(rem / (unsigned)C);
  const int sp = (int)(rem - (unsigned)x * (unsigned)C);
  const int s = g.ncls == 2 ? k + 2 * sp : sp;
  const int par_out = A.five_d ? ((1 - cb + k) & 1) : 1 - cb;
  const int mu = d & 3;
  Coord c = decode(g, x, par_out);
  const int n = mu == 0 ? g.lx : mu == 1 ? g.ly : mu == 2 ? g.lz : g.lt;
  int v = mu == 0 ? c.x : mu == 1 ? c.y : mu == 2 ? c.z : c.t;
  v = d < 4 ? (v + 1 == n ? 0 : v + 1) : (v == 0 ? n - 1 : v - 1);
  const int xn = cbindex(g, mu == 0 ? v : c.x, mu == 1 ? v : c.y, mu == 2 ? v : c.z, mu == 3 ? v : c.t);
  r.ni = (k ? (unsigned)g.kb1 : 0u) + (unsigned)xn * (unsigned)C + (unsigned)sp;
  r.lk = (long)(((d < 4 ? par_out : 1 - par_out) * 4 + mu) * 9) * A.U.n4cb + (d < 4 ? x : xn);
  // dwf_dslash_5_plus: upper (lower) chirality from s-1 (s+1) at dag 0, swapped at dag 1
  const unsigned em = site_entry(g, s == 0 ? g.ls - 1 : s - 1, x), ep = site_entry(g, s == g.ls - 1 ? 0 : s + 1, x);
  const double fm = s == 0 ? A.hop5_wall : A.hop5_fact, fp = s == g.ls - 1 ? A.hop5_wall : A.hop5_fact;
  const bool upper = d < 2;
  r.e5 = upper ? em : ep;
  r.e5d = upper ? ep : em;
  r.f5 = upper ? fm : fp;
  r.f5d = upper ? fp : fm;
  return r;
}

__device__ __forceinline__ double2 fma2d(double a, double2 x, double2 y) {
  return make_double2(__fma_rn(a, x.x, y.x), __fma_rn(a, x.y, y.y));
}

template <int NT, bool DAG, int MODE, bool PUPD>
__device__ __forceinline__ void pcg8_hop(const DslashArgs &A, const PcgArgs &P, const Pcg8Idx &first, double2 *gsh,
                                         double *nrm, const int *skip, const double *alpha, const double *beta) {
  const Geom &g = A.g;
  constexpr double sdag = DAG ? -1.0 : 1.0;
  const int d = threadIdx.x & 7, mu = d & 3;
  const double sg = d < 4 ? -sdag : sdag;
  const int base = threadIdx.x & ~7;
  const unsigned per = (unsigned)g.n4cb * (unsigned)g.ls;
  const long wstride = (long)gridDim.x * (NT / 8);
  const long e_first = (long)blockIdx.x * (NT / 8) + threadIdx.x / 8;
  // lanes 4-7 take no part after the products
  const bool owner = d < 4;
  for (int q = 0; q < g.nrhs; q++) {
    if (skip[q]) continue;
    const unsigned rb = (unsigned)q * per;
    const double b = PUPD ? beta[q] : 0.0;
    for (long e = e_first; e - (threadIdx.x / 8) % 4 < (long)per; e += wstride) {  // all four entries of a warp together
      Pcg8Idx ix = first;
      // a second round only where fewer than PCG_DP_SITES / 16 blocks are resident
      if (e != e_first) ix = pcg8_index(A, A.cb, e, d);
      const unsigned i = rb + ix.own;
      const bool mine = owner && ix.valid;
      // the epilogue's operands and the 5th-direction term of the lane's spin (chunks 3 d + c)
      double2 xo[3], ro[3], po[3], so[3], v5[3];
      if (mine) {
        if (MODE != 0) {
          const double2 *bx = entry_ptr<12, const double2>(A.x.data, i) + 24 * d;
#pragma unroll
          for (int c = 0; c < 3; c++) xo[c] = __ldcg(bx + 8 * c);
        }
        if (MODE == 2 || (MODE == 1 && PUPD)) {
          const double2 *br = entry_ptr<12, const double2>(P.r.data, i) + 24 * d;
#pragma unroll
          for (int c = 0; c < 3; c++) ro[c] = __ldcg(br + 8 * c);
        }
        if (MODE == 2) {
          const double2 *bp = entry_ptr<12, const double2>(P.p.data, i) + 24 * d;
          const double2 *bs = entry_ptr<12, const double2>(P.x.data, i) + 24 * d;
#pragma unroll
          for (int c = 0; c < 3; c++) {
            po[c] = __ldcg(bp + 8 * c);
            so[c] = __ldcg(bs + 8 * c);
          }
        }
        if (A.hop5) {
          const unsigned i5 = rb + (DAG ? ix.e5d : ix.e5);
          const double2 *b5 = entry_ptr<12, const double2>(A.in.data, i5) + 24 * d;
#pragma unroll
          for (int c = 0; c < 3; c++) v5[c] = __ldcg(b5 + 8 * c);
          if (PUPD && MODE == 0) {
            const double2 *br = entry_ptr<12, const double2>(P.r.data, i5) + 24 * d;
#pragma unroll
            for (int c = 0; c < 3; c++) v5[c] = fma2d(b, v5[c], __ldcg(br + 8 * c));
          }
        }
      }
      {
        // h0 = psi0 + s0 [i] X0, h1 = psi1 + s1 [i] X1 with X0, X1 = psi3, psi2 (x, y) or psi2, psi3 (z, t)
        const double2 *bn = entry_ptr<12, const double2>(A.in.data, rb + ix.ni);
        const double2 *br = entry_ptr<12, const double2>(P.r.data, rb + ix.ni);
        const int x0 = mu < 2 ? 9 : 6, x1 = mu < 2 ? 6 : 9;
        double2 u[6], x[6];
#pragma unroll
        for (int c = 0; c < 3; c++) {
          u[c] = __ldcg(bn + 8 * c);
          u[3 + c] = __ldcg(bn + 8 * (3 + c));
          x[c] = __ldcg(bn + 8 * (x0 + c));
          x[3 + c] = __ldcg(bn + 8 * (x1 + c));
        }
        if (PUPD && MODE == 0) {
#pragma unroll
          for (int c = 0; c < 3; c++) {
            u[c] = fma2d(b, u[c], __ldcg(br + 8 * c));
            u[3 + c] = fma2d(b, u[3 + c], __ldcg(br + 8 * (3 + c)));
            x[c] = fma2d(b, x[c], __ldcg(br + 8 * (x0 + c)));
            x[3 + c] = fma2d(b, x[3 + c], __ldcg(br + 8 * (x1 + c)));
          }
        }
        // U (forward) or U^dag (backward): row r, column k of it is element lr + lc of the stored link
        const double2 *lp = (const double2 *)A.U.data + ix.lk;
        const double cj = d < 4 ? 1.0 : -1.0;
        double2 l[9];
#pragma unroll
        for (int r = 0; r < 3; r++)
#pragma unroll
          for (int k = 0; k < 3; k++) {
            l[3 * r + k] = __ldg(lp + (long)(d < 4 ? 3 * r + k : 3 * k + r) * A.U.n4cb);
            l[3 * r + k].y *= cj;
          }
        const bool rot = (mu & 1) == 0;
        const double s0 = mu == 1 ? -sg : sg, s1 = mu == 2 ? -sg : sg;
        cplx<double> h[2][3];
#pragma unroll
        for (int c = 0; c < 3; c++) {
          const double2 a0 = rot ? make_double2(-x[c].y, x[c].x) : x[c];
          const double2 a1 = rot ? make_double2(-x[3 + c].y, x[3 + c].x) : x[3 + c];
          const double2 h0 = fma2d(s0, a0, u[c]), h1 = fma2d(s1, a1, u[3 + c]);
          h[0][c] = mk(h0.x, h0.y);
          h[1][c] = mk(h1.x, h1.y);
        }
#pragma unroll
        for (int a = 0; a < 2; a++)
#pragma unroll
          for (int r = 0; r < 3; r++) {
            const cplx<double> o = cmul(mk(l[3 * r].x, l[3 * r].y), h[a][0]) +
                                   cmul(mk(l[3 * r + 1].x, l[3 * r + 1].y), h[a][1]) +
                                   cmul(mk(l[3 * r + 2].x, l[3 * r + 2].y), h[a][2]);
            gsh[(3 * a + r) * NT + threadIdx.x] = make_double2(o.re, o.im);
          }
      }
      __syncwarp();
      if (mine) {
        // spin d of the sum over directions: U h itself for the upper spins, and for the
        // lower ones the multiples of h0, h1 of accum_reconstruct (cpsb_device.cuh)
        double2 acc[3];
#pragma unroll
        for (int c = 0; c < 3; c++) acc[c] = make_double2(0.0, 0.0);
        const bool lower = d >= 2;
#pragma unroll
        for (int j = 0; j < 8; j++) {
          const int m = j & 3;
          const double sj = j < 4 ? -sdag : sdag;
          const int hs = !lower ? d : m < 2 ? 3 - d : d - 2;
          const double low = m == 0 ? -sj : m == 1 ? (d == 2 ? sj : -sj) : m == 2 ? (d == 2 ? -sj : sj) : sj;
          const double cf = lower ? low : 1.0;
#pragma unroll
          for (int c = 0; c < 3; c++) {
            const double2 v = gsh[(3 * hs + c) * NT + base + j];
            acc[c] = fma2d(cf, lower && (m & 1) == 0 ? make_double2(-v.y, v.x) : v, acc[c]);
          }
        }
        if (A.hop5) {
          const double f5 = DAG ? ix.f5d : ix.f5;
#pragma unroll
          for (int c = 0; c < 3; c++) acc[c] = fma2d(f5, v5[c], acc[c]);
        }
        if (MODE == 0) {
          double2 *bo = entry_ptr<12, double2>(A.out.data, i) + 24 * d;
#pragma unroll
          for (int c = 0; c < 3; c++) bo[8 * c] = acc[c];
        } else {
          if (PUPD && MODE == 1) {
            // the new direction p = r + beta p at this entry: stored, and the xpay input
            double2 *bx = entry_ptr<12, double2>(A.x.data, i) + 24 * d;
#pragma unroll
            for (int c = 0; c < 3; c++) {
              xo[c] = fma2d(b, xo[c], ro[c]);
              bx[8 * c] = xo[c];
            }
          }
#pragma unroll
          for (int c = 0; c < 3; c++) acc[c] = fma2d(A.a, acc[c], xo[c]);
          double n2 = 0.0;
          if (MODE == 1) {
            double2 *bo = entry_ptr<12, double2>(A.out.data, i) + 24 * d;
#pragma unroll
            for (int c = 0; c < 3; c++) {
              bo[8 * c] = acc[c];
              n2 += acc[c].x * acc[c].x + acc[c].y * acc[c].y;
            }
          } else {
            const double al = alpha[q];
            double2 *bs = entry_ptr<12, double2>(P.x.data, i) + 24 * d;
            double2 *br = entry_ptr<12, double2>(P.r.data, i) + 24 * d;
#pragma unroll
            for (int c = 0; c < 3; c++) {
              bs[8 * c] = fma2d(al, po[c], so[c]);
              const double2 rn = fma2d(-al, acc[c], ro[c]);
              br[8 * c] = rn;
              n2 += rn.x * rn.x + rn.y * rn.y;
            }
          }
          nrm[q * NT + threadIdx.x] += n2;
        }
      }
      __syncwarp();  // the slots are written again in the next round
    }
  }
}

// Per-right-hand-side sums of nrm over the grid, left in out[] of every block: the
// first warp of each block adds the block partials, a lane every 32nd and then the
// lanes pairwise, so all blocks get the same bits without a further exchange.
template <int NT>
__device__ __forceinline__ bool pcg_reduce(const PcgArgs &P, int nrhs, double *nrm, double *red, double *out,
                                           unsigned &epoch) {
  for (int q = 0; q < nrhs; q++) {
    const double bs = block_sum<NT>(nrm[q * NT + threadIdx.x], red);
    nrm[q * NT + threadIdx.x] = 0;
    if (threadIdx.x == 0) P.partial[q * gridDim.x + blockIdx.x] = bs;
  }
  if (!pcg_sync(P, epoch)) return false;
  if (threadIdx.x < 32) {
    for (int q = 0; q < nrhs; q++) {
      double v = 0;
      for (int k = threadIdx.x; k < (int)gridDim.x; k += 32) v += __ldcg(P.partial + q * gridDim.x + k);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (threadIdx.x == 0) out[q] = v;
    }
  }
  __syncthreads();
  return true;
}

// DP: the hop phases with eight lanes per entry (pcg8_hop), for the smallest lattices.
template <int NT, bool LC, bool DP>
__global__ void __launch_bounds__(NT, 1) pcg_kernel(PcgArgs P) {
  extern __shared__ __align__(16) unsigned char dsh[];
  __shared__ CgState S;
  __shared__ double red[NT / 32];
  __shared__ double sums[MAX_RHS], alpha[MAX_RHS], beta[MAX_RHS];
  __shared__ int skip[MAX_RHS];
  const Geom &g = P.ph[0].g;
  const int nrhs = g.nrhs;
  const int C0 = g.cs[0];
  const HopShm L = hop_shm(NT / C0, NT, nrhs, true, LC);
  double2 *gsh = (double2 *)dsh;  // DP: 6 x NT half-spinor slots
  double *nrm = (double *)(dsh + (DP ? (size_t)6 * NT * sizeof(double2) : L.norm));
  unsigned epoch = 0;
  Pcg8Idx ix[2];  // DP: of the thread's first entry, input checkerboard 0 and 1
  if constexpr (DP)
#pragma unroll
    for (int cb = 0; cb < 2; cb++)
      ix[cb] = pcg8_index(P.ph[0], cb, (long)blockIdx.x * (NT / 8) + threadIdx.x / 8, threadIdx.x & 7);
  if (threadIdx.x == 0) S = *P.S;
  for (int q = 0; q < nrhs; q++) nrm[q * NT + threadIdx.x] = 0;
  __syncthreads();
  const long per = (long)g.n4cb * g.ls;
  for (int guard = 0; guard <= S.max_iter + 1; guard++) {
    bool all = true;
    for (int q = 0; q < nrhs; q++) all = all && S.halt_done[q];
    if (all) break;
    if (threadIdx.x < nrhs) {
      skip[threadIdx.x] = S.halt[threadIdx.x];
      // DP: the direction update of the previous iteration rides on this one's
      // first two hops (p = r on entry: beta 0 in the first iteration)
      beta[threadIdx.x] = guard == 0 ? 0.0 : S.beta[threadIdx.x];
    }
    __syncthreads();
    // t1 = D p
    if constexpr (DP) pcg8_hop<NT, false, 0, true>(P.ph[0], P, ix[1], gsh, nrm, skip, alpha, beta);
    else pcg_hop<NT, LC, false, 0>(P.ph[0], P, dsh, nrm, skip, alpha);
    if (!pcg_sync(P, epoch)) break;
    // t2 = MatPc p, d = |t2|^2
    if constexpr (DP) pcg8_hop<NT, false, 1, true>(P.ph[1], P, ix[0], gsh, nrm, skip, alpha, beta);
    else pcg_hop<NT, LC, false, 1>(P.ph[1], P, dsh, nrm, skip, alpha);
    if (!pcg_reduce<NT>(P, nrhs, nrm, red, sums, epoch)) break;
    if (threadIdx.x < nrhs && !skip[threadIdx.x]) S.d[threadIdx.x] = sums[threadIdx.x];
    __syncthreads();
    // t1 = D^dag t2
    if constexpr (DP) pcg8_hop<NT, true, 0, false>(P.ph[2], P, ix[1], gsh, nrm, skip, alpha, beta);
    else pcg_hop<NT, LC, true, 0>(P.ph[2], P, dsh, nrm, skip, alpha);
    if (!pcg_sync(P, epoch)) break;
    // A p = MatPcDag t2: r -= alpha A p, x += alpha p, |r|^2
    if (threadIdx.x < nrhs) {
      const int q = threadIdx.x;
      alpha[q] = S.rr[q] / (S.d[q] + S.shift * S.pp[q]);
    }
    __syncthreads();
    if constexpr (DP) pcg8_hop<NT, true, 2, false>(P.ph[3], P, ix[0], gsh, nrm, skip, alpha, beta);
    else pcg_hop<NT, LC, true, 2>(P.ph[3], P, dsh, nrm, skip, alpha);
    if (!pcg_reduce<NT>(P, nrhs, nrm, red, sums, epoch)) break;
    if (threadIdx.x == 0)
      for (int q = 0; q < nrhs; q++)
        if (!skip[q]) cg_advance(&S, q, sums[q]);
    __syncthreads();
    if constexpr (DP) {
      // p is updated by the next iteration's first two hops; a right-hand side
      // that halted here is skipped from then on
      if (threadIdx.x == 0)
        for (int q = 0; q < nrhs; q++) S.halt_done[q] = S.halt[q];
      __syncthreads();
      continue;
    }
    // p = r + beta p for the right-hand sides still iterating (cg_xp_update, blas.cu)
    for (int q = 0; q < nrhs; q++) {
      if (S.halt_done[q] || S.halt[q]) continue;
      const double b = S.beta[q];
      for (long j = (long)blockIdx.x * NT + threadIdx.x; j < per; j += (long)gridDim.x * NT) {
        const unsigned i = (unsigned)(q * per + j);
        Spinor<double> pv = unpack64(load_raw64_l2(P.p, i));
        const Spinor<double> rv = unpack64(load_raw64_l2(P.r, i));
#pragma unroll
        for (int s2 = 0; s2 < 4; s2++)
#pragma unroll
          for (int r = 0; r < 3; r++) pv.c[s2][r] = cscale(b, pv.c[s2][r]) + rv.c[s2][r];
        store_spinor<P64>(P.p, i, pv);
      }
    }
    __syncthreads();
    if (threadIdx.x == 0)
      for (int q = 0; q < nrhs; q++) S.halt_done[q] = S.halt[q];
    if (!pcg_sync(P, epoch)) break;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *P.S = S;
}

// Largest grid of a persistent solve on this device: all blocks resident.
static int pcg_max_blocks(const void *fn, int nt, size_t shm) {
  int dev = 0, nsm = 0, per_sm = 0, coop = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop ||
      cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, nt, shm) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return nsm * per_sm;
}

int persistent_cg_mode() {
  const char *e = getenv("CPSB_PERSISTENT_CG");
  return e ? atoi(e) : 1;
}

// Runs the iterations of an FP64 CG solve whose state (r, p, x, CgState) the
// caller has set up.  Returns cudaErrorNotSupported, launching nothing, where
// the persistent form does not apply (the caller then runs its own loop).
cudaError_t launch_persistent_cg(const DslashArgs &base, double mkappa2, SpinorPtr t1, SpinorPtr t2, SpinorPtr r,
                                 SpinorPtr p, SpinorPtr x, CgState *S, double *partial, size_t partial_slots,
                                 unsigned *bar_err, cudaStream_t st) {
  const Geom &g = base.g;
  const int C0 = g.cs[0];
  if (C0 < 1 || C0 > PCG_NT_MAX) return cudaErrorNotSupported;
  const long per = (long)g.n4cb * g.ls;
  const bool dp = per * g.nrhs <= PCG_DP_SITES;
  const int nt = dp ? PCG_NT_MAX : C0 == 1 ? 32 : PCG_NT_MAX;
  const int TX = nt / C0;
  const bool lc = TX <= 32;
  const size_t shm = dp ? (size_t)6 * nt * sizeof(double2) + (size_t)nt * g.nrhs * sizeof(double)
                        : hop_shm(TX, nt, g.nrhs, true, lc).total;
  if (shm > 48 * 1024) return cudaErrorNotSupported;
  const void *fn = dp ? (const void *)pcg_kernel<PCG_NT_MAX, false, true>
                      : nt == 32 ? (const void *)pcg_kernel<32, true, false>
                      : lc ? (const void *)pcg_kernel<PCG_NT_MAX, true, false>
                           : (const void *)pcg_kernel<PCG_NT_MAX, false, false>;
  const long units = dp ? (per + nt / 8 - 1) / (nt / 8) : (long)((g.n4cb + TX - 1) / TX) * g.ncls;
  const int grid = (int)std::min(units, (long)pcg_max_blocks(fn, nt, shm));
  if (grid < 1 || (size_t)grid * g.nrhs > partial_slots) return cudaErrorNotSupported;
  PcgArgs P;
  memset(&P, 0, sizeof(P));
  for (int k = 0; k < 4; k++) {
    P.ph[k] = base;
    P.ph[k].torder = 0;
    P.ph[k].skip = nullptr;
    memset(&P.ph[k].red, 0, sizeof(Reduce));
    P.ph[k].cg = nullptr;
  }
  P.ph[0].in = p, P.ph[0].out = t1, P.ph[0].cb = 1, P.ph[0].dag = 0, P.ph[0].a = 1.0;
  P.ph[1].in = t1, P.ph[1].out = t2, P.ph[1].x = p, P.ph[1].cb = 0, P.ph[1].dag = 0, P.ph[1].a = mkappa2;
  P.ph[2].in = t2, P.ph[2].out = t1, P.ph[2].cb = 1, P.ph[2].dag = 1, P.ph[2].a = 1.0;
  P.ph[3].in = t1, P.ph[3].x = t2, P.ph[3].cb = 0, P.ph[3].dag = 1, P.ph[3].a = mkappa2;
  P.r = r;
  P.p = p;
  P.x = x;
  P.S = S;
  P.partial = partial;
  P.bar = bar_err;
  P.err = (int *)(bar_err + 2);
  cudaError_t e = cudaMemsetAsync(bar_err, 0, 4 * sizeof(unsigned), st);
  if (e != cudaSuccess) return e;
  void *args[] = {&P};
  e = cudaLaunchCooperativeKernel(fn, dim3((unsigned)grid), dim3(nt), args, shm, st);
  count_launch();
  return e;
}

}  // namespace cpsb
