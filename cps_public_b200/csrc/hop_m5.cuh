// hop_m5.cuh -- the Mobius 4-D hop with the M5 column operations of its output
// fused in: one pass over memory where the operator otherwise runs the hop,
// stores its output, and reads it back in a separate M5 kernel.
//
//   dag 0:  out = a * mix(M5^-1 (D in))                  (zmobius_m-sym2.h: the
//           M5^-1 that follows the first kappa_b D4 of MatPc, dag 0)
//   dag 1:  out = [x +] a * M5^-dag(mix^dag(D^dag in))  [, |out|^2]
//           (zmobius_mdag-sym2.h: the M5^-dag after each D4^dag of MatPcDag), or
//           with A.cg the CG update on it as in hop_kernel: out = A p is not stored
//           but consumed by r -= alpha (A p + shift p), x += alpha p and |r|^2
//
// With 4-D checkerboarding (DWF_4D_EOPREC_EE) every slice of a site has the
// same parity, so the column of a site holds all Ls slices and the block that
// computes a tile's hop owns whole columns: the Ls hop outputs of a column are
// written to a shared-memory tile, one thread per (column, complex component)
// runs the sweeps of m5_sweep.cuh over its Ls values in registers, and every
// thread reads its own entry back for the epilogue and the store.  The hop
// itself is hop.cuh's (links of the unit in shared memory, neighbour tables).
#pragma once
#include "hop.cuh"
#include "m5_sweep.cuh"

namespace cpsb {

// Dynamic shared memory: hop.cuh's tables, then the sweep tile.
template <int P, int LS>
__host__ __device__ inline size_t hop_m5_tile_off(int TX, int NT, int nrhs, bool norm) {
  return (hop_shm(TX, NT, nrhs, norm, true).total + 15) & ~(size_t)15;
}
template <int P, int LS>
__host__ __device__ inline size_t hop_m5_shm(int TX, int NT, int nrhs, bool norm) {
  return hop_m5_tile_off<P, LS>(TX, NT, nrhs, norm) + sweep_tile_bytes<P, LS>(TX);
}

// Thread t owns slice t % LS of tile column t / LS for every right-hand side
// in turn; the skip mask is read per right-hand side, uniformly over the block,
// so every thread reaches every barrier.
template <int P, int NT, int MINB, bool DAG, bool XPAY, bool NORM, int CGR, int LS, int DEPTH>
__global__ void __launch_bounds__(NT, MINB) hop_m5_kernel(DslashArgs A, M5Coef cf) {
  typedef typename SweepT<P>::T BT;
  constexpr int TX = NT / LS;
  constexpr int CST = LS + 1;
  const Geom &g = A.g;
  extern __shared__ __align__(16) unsigned char dsh[];
  __shared__ double red[NT / 32];
  __shared__ double cg_alpha[MAX_RHS];  // as in hop_kernel
  const HopShm L = hop_shm(TX, NT, g.nrhs, NORM || CGR, true);
  BT *tile_buf = (BT *)(dsh + hop_m5_tile_off<P, LS>(TX, NT, g.nrhs, NORM || CGR));
  double *nrm_sh = (double *)(dsh + L.norm);
  if (NORM || CGR)
    for (int q = 0; q < g.nrhs; q++) nrm_sh[q * NT + threadIdx.x] = 0;
  const int sp = threadIdx.x % LS;
  const int xl = threadIdx.x / LS;
  const int ntiles = (g.n4cb + TX - 1) / TX;
  const unsigned per = (unsigned)g.n4cb * (unsigned)LS;
  const int par_out = 1 - A.cb;
  if ((int)blockIdx.x < ntiles) load_unit<P, true>(A, blockIdx.x, 0, par_out, TX, NT, dsh);
  if (CGR && threadIdx.x < g.nrhs) {
    const CgState *S = A.cg;
    cg_alpha[threadIdx.x] = S->rr[threadIdx.x] / (S->d[threadIdx.x] + S->shift * S->pp[threadIdx.x]);
  }
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    if (tile != (int)blockIdx.x) {
      __syncthreads();  // the previous tile is done with the tables and the sweep tile
      load_unit<P, true>(A, tile, 0, par_out, TX, NT, dsh);
    }
    __syncthreads();
    const int x = tile * TX + xl;
    const bool act = xl < TX && x < g.n4cb;
    const int nx = min(TX, g.n4cb - tile * TX);
    HopCtx hc;
    if (act) entry_ctx<P, true>(hc, A, dsh, L, xl, x, 0, sp, par_out);
    const unsigned own = (unsigned)x * (unsigned)LS + (unsigned)sp;
    BT *mine = tile_buf + (size_t)xl * 12 * CST + sp;  // component q of this entry at mine[q * CST]
    for (int rhs = 0; rhs < g.nrhs; rhs++) {
      if (A.skip && A.skip[rhs]) continue;
      const unsigned rb = (unsigned)rhs * per;
      const unsigned i = rb + own;
      // 1. the hop of this thread's entry into the sweep tile (FP64: component
      // q = 3 spin + colour as (re, im); FP32 / 16-bit: q = 2 (3 p + colour) +
      // (0 re, 1 im) as the lanes (spin 2p, spin 2p + 1))
      if (act) {
        if constexpr (P == P64) {
          const Spinor<double> o = hop_entry_64<P, true, DAG, DEPTH>(A, hc, rb);
#pragma unroll
          for (int q = 0; q < 12; q++) mine[q * CST] = make_double2(o.c[q / 3][q % 3].re, o.c[q / 3][q % 3].im);
        } else {
          const SpX2 o = hop_entry_x2<P, true, DAG, DEPTH>(A, hc, rb);
#pragma unroll
          for (int q = 0; q < 6; q++) {
            mine[(2 * q) * CST] = o.re[q / 3][q % 3];
            mine[(2 * q + 1) * CST] = o.im[q / 3][q % 3];
          }
        }
      }
      __syncthreads();
      // 2. the column operations
      sweep_tile<P, LS, DAG ? 1 : 0, NT>(tile_buf, nx, cf);
      __syncthreads();
      // 3. epilogue: out = [x +] a v
      if (act) {
        if constexpr (P == P64) {
          Spinor<double> o;
#pragma unroll
          for (int q = 0; q < 12; q++) {
            const double2 v = mine[q * CST];
            o.c[q / 3][q % 3] = mk(A.a * v.x, A.a * v.y);
          }
          if (XPAY) {
            const Spinor<double> xv = unpack64(load_raw<P64>(A.x, i));
#pragma unroll
            for (int s2 = 0; s2 < 4; s2++)
#pragma unroll
              for (int r = 0; r < 3; r++) o.c[s2][r] = xv.c[s2][r] + o.c[s2][r];
          }
          if (CGR) {
            nrm_sh[rhs * NT + threadIdx.x] += cg_epilogue_64<CGR>(A, i, cg_alpha[rhs], o);
          } else {
            store_spinor<P64>(A.out, i, o);
            if (NORM) nrm_sh[rhs * NT + threadIdx.x] += norm2(o);
          }
        } else {
          const float2 a2 = f2b((float)A.a);
          SpX2 o;
#pragma unroll
          for (int q = 0; q < 6; q++) {
            o.re[q / 3][q % 3] = mul2(a2, mine[(2 * q) * CST]);
            o.im[q / 3][q % 3] = mul2(a2, mine[(2 * q + 1) * CST]);
          }
          if (XPAY) {
            float xn;
            const SpX2 xv = unpack(load_raw<P>(A.x, i), &xn);
            const float2 xs = f2b(xn);
#pragma unroll
            for (int p = 0; p < 2; p++)
#pragma unroll
              for (int cc = 0; cc < 3; cc++) {
                o.re[p][cc] = fma2(xv.re[p][cc], xs, o.re[p][cc]);
                o.im[p][cc] = fma2(xv.im[p][cc], xs, o.im[p][cc]);
              }
          }
          if (CGR) {
            nrm_sh[rhs * NT + threadIdx.x] += cg_epilogue_x2<P, CGR>(A, i, (float)cg_alpha[rhs], o);
          } else {
            const double n2 = store_x2<P>(A.out, i, o);
            if (NORM) nrm_sh[rhs * NT + threadIdx.x] += n2;
          }
        }
      }
      __syncthreads();  // every entry is read back before the next right-hand side's hop
    }
  }
  if (NORM || CGR) hop_reduce<NT, CGR>(A, nrm_sh, red);
}

template <int P, int LS, bool DAG, bool XPAY, bool NORM, int CGR, int MINB>
static cudaError_t hop_m5_launch_v(const DslashArgs &A, const M5Coef &cf, cudaStream_t st) {
  constexpr int NT = 128;
  constexpr int DEPTH = P == P64 ? 1 : 2;
  constexpr int TX = NT / LS;
  const size_t shm = hop_m5_shm<P, LS>(TX, NT, A.g.nrhs, NORM || CGR);
  if (shm > 200 * 1024) return cudaErrorNotSupported;
  const void *fn = (const void *)hop_m5_kernel<P, NT, MINB, DAG, XPAY, NORM, CGR, LS, DEPTH>;
  static bool opted = false;
  if (!opted && shm + 1024 > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e != cudaSuccess) return e;
    opted = true;
  }
  const long ntiles = (A.g.n4cb + TX - 1) / TX;
  const long nb = std::min(ntiles, (long)resident_blocks(fn, NT, shm));
  hop_m5_kernel<P, NT, MINB, DAG, XPAY, NORM, CGR, LS, DEPTH><<<(unsigned)nb, NT, shm, st>>>(A, cf);
  return launched();
}

template <int P, int LS, bool DAG, bool XPAY, bool NORM, int CGR>
static cudaError_t hop_m5_launch_m(const DslashArgs &A, const M5Coef &cf, cudaStream_t st) {
  if constexpr (P != P64) {
    return hop_m5_launch_v<P, LS, DAG, XPAY, NORM, CGR, 4>(A, cf, st);
  } else {
    // FP64: 168 registers for 3 blocks an SM (24^3x64, Ls 16: 1330, 1317 and 1310 us the
    // hops, against 1515, 1375 and 1354 with 255 for 2) where there are tiles for a
    // third block and room beside its tables.  Not at Ls 4, whose 80 KB a block let two
    // run, nor on fields that two blocks an SM cover: registers spent on nothing.
    // CG to 1e-8 with 2 and 3: 16^3x32, Ls 4 23.9 and 27.4 ms; 8^4, Ls 8 (128 tiles)
    // 4.84 and 5.01, 3 sources 9.1 and 9.7; 8^4, Ls 16 (256) 8.13 and 8.26; 12^3x16, Ls 8
    // (864) 15.4 and 14.8.
    if constexpr (LS > 4) {
      const long ntiles = (A.g.n4cb + 128 / LS - 1) / (128 / LS);
      if (ntiles > 2 * 148) return hop_m5_launch_v<P, LS, DAG, XPAY, NORM, CGR, 3>(A, cf, st);
    }
    return hop_m5_launch_v<P, LS, DAG, XPAY, NORM, CGR, 2>(A, cf, st);
  }
}

template <int P, int LS>
static cudaError_t hop_m5_launch_ls(const DslashArgs &A, const M5Coef &cf, int xpay, int norm, cudaStream_t st) {
  if (A.cg) {  // the CG residual update: dag 1, xpay
    if (!A.dag || !xpay || !A.cg_x.data) return cudaErrorInvalidValue;
    if (A.cg_shift) return hop_m5_launch_m<P, LS, true, true, false, 2>(A, cf, st);
    return hop_m5_launch_m<P, LS, true, true, false, 1>(A, cf, st);
  }
  if (!A.dag) {
    if (xpay || norm) return cudaErrorNotSupported;
    return hop_m5_launch_m<P, LS, false, false, false, 0>(A, cf, st);
  }
  if (xpay && norm) return hop_m5_launch_m<P, LS, true, true, true, 0>(A, cf, st);
  if (xpay) return hop_m5_launch_m<P, LS, true, true, false, 0>(A, cf, st);
  if (norm) return cudaErrorNotSupported;
  return hop_m5_launch_m<P, LS, true, false, false, 0>(A, cf, st);
}

// The fused hop + M5 for one storage precision; cudaErrorNotSupported for a
// shape without a fused form (5-D checkerboarding, the 5th-direction hop, an
// Ls not listed), for which the caller runs the hop and the M5 kernel.
template <int P>
static cudaError_t hop_m5_launch_p(const DslashArgs &A, const M5Coef &cf, int xpay, int norm, cudaStream_t st) {
  if (A.five_d || A.hop5 || A.g.ncls != 1 || A.g.cs[0] != A.g.ls) return cudaErrorNotSupported;
  switch (A.g.ls) {
    case 4: return hop_m5_launch_ls<P, 4>(A, cf, xpay, norm, st);
    case 8: return hop_m5_launch_ls<P, 8>(A, cf, xpay, norm, st);
    case 12: return hop_m5_launch_ls<P, 12>(A, cf, xpay, norm, st);
    case 16: return hop_m5_launch_ls<P, 16>(A, cf, xpay, norm, st);
    case 20: return hop_m5_launch_ls<P, 20>(A, cf, xpay, norm, st);
    case 24: return hop_m5_launch_ls<P, 24>(A, cf, xpay, norm, st);
    case 32: return hop_m5_launch_ls<P, 32>(A, cf, xpay, norm, st);
    default: return cudaErrorNotSupported;
  }
}

}  // namespace cpsb
