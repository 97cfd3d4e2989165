// gbf_dslash.cu -- the even-odd Wilson hopping kernel with fused epilogues.
//
// Computes, for every 5D site n of the output parity p (thread per site):
//   hop(x) = -1/2 sum_mu cc_mu [ (1 + s g_mu) U_mu(x) in(x+mu)
//                               + (1 - s g_mu) U_mu(x-mu)^+ in(x-mu) ]
// with s = -1 for Dhop and s = +1 for Dhop^dag (the statement of
// lib/gpt/qcd/fermion/reference/wilson_clover.py:182-200, which Grid's
// WilsonKernels implement for opcodes 3001/3002/4001/4002, and the 4D part of
// Grid's Cayley Meooe for Mobius), followed by the epilogue
//   out = c1 * L1(hop) + c2 * L2(X)       (L1, L2 site-local operators)
// and optionally the deterministic reduction of <Y, out> or |out|^2 with a
// CG finaliser.  The input spinor is projected to two spin components before
// the colour multiply (8 x 2 SU(3) matvecs per site) and the lower two spin
// components of each term are rebuilt from the upper two.
//
// Roofline: HBM-bound in FP32/FP16 (per output site: 8 neighbour spinors that
// the L2 mostly serves once, 8 links, 1 output); FP64 is bound by the FP64
// pipe on GB300 (about 1.2 TFLOP/s measured).
#include <array>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <mutex>
#include <tuple>
#include "gbf_launch.cuh"
#include "gbf_split.cuh"

// resident blocks of 256 threads per SM requested for the FP32/FP16 variants
// (register cap 65536 / (256 * minblocks))
#ifndef GBF_DSLASH_MINB
#define GBF_DSLASH_MINB 2
#endif
// the same for the double-float variant (2: 128 registers, a few spills in
// the clover epilogue, measured faster than 1 block of 255 registers)
#ifndef GBF_DSLASH_MINB_DD
#define GBF_DSLASH_MINB_DD 2
#endif

namespace gbf {

// Offset (in 16-byte units) of the double-float accumulators in dynamic
// shared memory: after the s-matrix tile and the reduction scratch.
__host__ __device__ inline unsigned dd_acc_offset16(int LK, unsigned bd) {
  const size_t s = smat_smem_bytes(LK, (int)bd, 8) + 2 * (size_t)bd * 8;
  return (unsigned)((s + 15) / 16);
}

// Epilogue of the hopping kernels for the 5D site n (4D site cb of the
// output parity): out = c1 L1(hop) + c2 L2(X), store, and the per-thread
// part of the optional reduction.  Every thread of the block calls (the
// s-matrix op synchronises the block).
template <int P, int LK, bool LOOP>
__device__ __forceinline__ void hop_epilogue(const DslashArgs& a, const HopIO& io, bool active, long long n, int cb,
                                             cplx<typename SpinorT<P>::R> (&res)[12], double& red_re,
                                             double* smem_d) {
  using R = typename SpinorT<P>::R;
  using V = cplx<R>;
  if constexpr (LK == LOC_NONE) {  // the pure hop
    if (active) store_spinor<P>(io.out, a.g.N, n, res);
    return;
  }
  const Geo& g = a.g;
  const int p = io.p;
  if (LK == LOC_SMAT) {
    if (a.l1.kind == LOC_SMAT) {
      R* tile = reinterpret_cast<R*>(smem_d);
      R* mat = tile + 24 * blockDim.x;
      if (a.l1.cplx) smat_apply_block_c<R>(reinterpret_cast<const R*>(a.l1.smat), g.Ls, tile, mat, res);
      else smat_apply_block<R>(reinterpret_cast<const R*>(a.l1.smat), g.Ls, tile, mat, res, true);
    }
  } else if (LK == LOC_BAND) {
    if (a.l1.kind == LOC_BAND)
      band_apply_block<R, LOOP>(a.l1, g.Ls, g.fLs, reinterpret_cast<typename SplitWord<R>::T*>(smem_d), res);
  } else if (active && a.l1.kind != LOC_NONE) {
    if constexpr (P == PDD) {
      if (a.l1.kind == LOC_CLOVER) clover_apply_dd_lowreg(a.l1.clov[p], g.Vh, cb, res);
      else local_apply_thread<R>(a.l1, g.Vh, p, cb, res);
    } else {
      local_apply_thread<R>(a.l1, g.Vh, p, cb, res);
    }
  }
  if (active) {
    if (!a.c1.is_one()) {
      const R c1 = coef<R>(a.c1);
#pragma unroll
      for (int k = 0; k < 12; ++k) {
        nrm<R>(res[k]);
        res[k] = scl<R>(c1, res[k]);
      }
    }
    if (io.X) {
      V xv[12];
      if (LK == LOC_BAND && a.l2.kind == LOC_BAND) {
        const unsigned r = (unsigned)n;
        band_load<P>(a.l2, g.Ls, (int)(r - g.fLs.div(r) * (unsigned)g.Ls), io.X, (unsigned)g.N, r, xv);
      } else {
        load_spinor<P>(io.X, g.N, n, xv);
      }
      if (LK == LOC_CLOVER && a.l2.kind != LOC_NONE) {
        if constexpr (P == PDD) {
          if (a.l2.kind == LOC_CLOVER) clover_apply_dd_lowreg(a.l2.clov[p], g.Vh, cb, xv);
          else local_apply_thread<R>(a.l2, g.Vh, p, cb, xv);
        } else {
          local_apply_thread<R>(a.l2, g.Vh, p, cb, xv);
        }
      }
      const R c2 = coef<R>(a.c2);
#pragma unroll
      for (int k = 0; k < 12; ++k) res[k] = mk<R>(fma(c2, xv[k].x, res[k].x), fma(c2, xv[k].y, res[k].y));
    }
  }
  // (the Y term is read before the store: loads are not moved across it.  In
  // double-float the store comes first and frees registers: the normal operator
  // on 32^4 1333 -> 1298 us, zmobius on 16^4 Ls 10 1023 -> 1014)
  if (P == PDD && active) store_spinor<P>(io.out, g.N, n, res);
  if (a.red && active) {
    if (a.red == 1) {
      V yv[12];
      load_spinor<P>(a.Y, g.N, n, yv);
      red_re += site_dot_re<R>(yv, res);
    } else {
      red_re += site_norm2<R>(res);
    }
  }
  if (P != PDD && active) store_spinor<P>(io.out, g.N, n, res);
}

// BOTH: launched for both parities too.  Compiled apart for double-float, which
// is at its 128 registers and spills more with the selection of the parity
// (normal operator, with it / without: 32^4 1290 / 1268 us, Mobius 16^4 Ls 12 870
// / 860), but not with dense s-matrices (zmobius 1014 / 1030)
template <int P, int LS, int LK, bool LOOP, bool BOTH = !LOOP>
__global__ void __launch_bounds__(256, (P == P64 ? 1 : P == PDD ? GBF_DSLASH_MINB_DD : GBF_DSLASH_MINB)) dslash_kernel(const DslashArgs a) {
  pdl_begin();
  using R = typename SpinorT<P>::R;
  using V = cplx<R>;
  extern __shared__ __align__(16) double smem_d[];
  const Geo& g = a.g;
  const HopIO io = hop_io<BOTH>(a);
  if (a.check_done && a.ra.st->all_done) return;
  const int p = io.p, q = 1 - p;
  double red_re = 0;
  // block-uniform loop over tiles of blockDim sites; LOOP = false when the
  // grid covers every tile (one tile per block, no loop is compiled)
  const long long ntiles = (g.N + blockDim.x - 1) / blockDim.x;
  long long tile = blockIdx.x;
  do {
  const long long n = tile * blockDim.x + threadIdx.x;
  const bool active = n < g.N;
  V res[12];
#pragma unroll
  for (int k = 0; k < 12; ++k) res[k] = cz<R>();
  int cb = 0;
  if constexpr (P == PDD) {
    if (active) {
      // double-float, rolled direction loop (one iteration is about 1.5k
      // instructions; unrolled eight times the kernel would not fit the
      // instruction cache).  The 12 accumulators live in shared memory
      // ([component][thread], 16 B each) during the loop, which frees 48
      // registers per thread for more resident warps.
      cb = (int)g.fN5.div((unsigned)n);
      const unsigned i5 = (unsigned)n - (unsigned)cb * (unsigned)g.N5;
      const Coord c = cb_coords(g, cb, p);
      float4* acc = reinterpret_cast<float4*>(smem_d) + dd_acc_offset16(LK, blockDim.x) + threadIdx.x;
      const unsigned bs = blockDim.x;
#pragma unroll
      for (int k = 0; k < 12; ++k) acc[k * bs] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
      for (int d = 0; d < 8; ++d) {
        const int mu = d >> 1;
        const bool fwd = (d & 1) == 0;
        int y[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          const int xm = c.x[m], Lm = g.L[m];
          y[m] = (m != mu) ? xm : fwd ? (xm == Lm - 1 ? 0 : xm + 1) : (xm == 0 ? Lm - 1 : xm - 1);
        }
        const int ycb = cb_index(g, y);
        const unsigned site = (unsigned)ycb * (unsigned)g.N5 + i5;
        const float s = fwd ? a.sgn : -a.sgn;
        // lane-paired form (pdd): u h = Re(u) h + Im(u) (i h), and the
        // backward term's conj(u) negates Im(u)
        {
          const float4* sp = reinterpret_cast<const float4*>(io.in);
          const unsigned N = (unsigned)g.N;
          pdd h[2][3];
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const int pr = gperm(mu, r), cr = gcoef(mu, r);
#pragma unroll
            for (int col = 0; col < 3; ++col) {
              const pdd up = pdd_ld(ldg(sp + (site + (unsigned)(3 * r + col) * N)));
              const pdd lo = pdd_ld(ldg(sp + (site + (unsigned)(3 * pr + col) * N)));
              h[r][col] = pdd_coefmadd_rt(cr, s, lo, up);
            }
          }
          const float4* L = reinterpret_cast<const float4*>(a.links) +
                            (unsigned)(((fwd ? p : q) * 4 + mu) * 9) * (unsigned)g.Vh + (unsigned)(fwd ? cb : ycb);
          const float cs = fwd ? 1.f : -1.f;
          pdd uh[2][3];
#pragma unroll
          for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
              const unsigned k = fwd ? (unsigned)(3 * i + j) : (unsigned)(3 * j + i);
              const float4 qv = ldg(L + k * (unsigned)g.Vh);
              const dd ux(qv.x, qv.z), uy = dd_scale2(cs, dd(qv.y, qv.w));
#pragma unroll
              for (int r = 0; r < 2; ++r) {
                uh[r][i] = j == 0 ? pdd_mul_s(ux, h[r][j]) : pdd_fma_s(ux, h[r][j], uh[r][i]);
                uh[r][i] = pdd_fma_s(uy, pdd_i(h[r][j]), uh[r][i]);
              }
            }
#pragma unroll
          for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int i = 0; i < 3; ++i) {
              float4& m = acc[(3 * r + i) * bs];
              m = pdd_st(pdd_add(pdd_ld(m), uh[r][i]));
            }
#pragma unroll
          for (int r = 2; r < 4; ++r) {
            const bool first = gperm(mu, r) == 0;
            const int cr = gcoef(mu, r);
#pragma unroll
            for (int i = 0; i < 3; ++i) {
              float4& m = acc[(3 * r + i) * bs];
              m = pdd_st(pdd_coefmadd_rt(cr, s, first ? uh[0][i] : uh[1][i], pdd_ld(m)));
            }
          }
        }
      }
#pragma unroll
      for (int k = 0; k < 12; ++k) {
        const float4 m = acc[k * bs];
        res[k] = mk<dd>(dd(m.x, m.z), dd(m.y, m.w));
      }
    }
  } else if (active) {
    cb = (int)g.fN5.div((unsigned)n);
    const unsigned i5 = (unsigned)n - (unsigned)cb * (unsigned)g.N5;
    const Coord c = cb_coords(g, cb, p);
    const R sf = (R)a.sgn;
#pragma unroll
    for (int mu = 0; mu < 4; ++mu) {
#pragma unroll
      for (int dir = 0; dir < 2; ++dir) {
        int y[4] = {c.x[0], c.x[1], c.x[2], c.x[3]};
        const bool fwd = dir == 0;
        bool wrap;
        if (fwd) {
          wrap = (y[mu] == g.L[mu] - 1);
          y[mu] = wrap ? 0 : y[mu] + 1;
        } else {
          wrap = (y[mu] == 0);
          y[mu] = wrap ? g.L[mu] - 1 : y[mu] - 1;
        }
        const int ycb = cb_index(g, y);
        V psi[12];
        load_spinor<P>(io.in, g.N, (unsigned)ycb * (unsigned)g.N5 + i5, psi);
        // project: h_r = psi_r + s * coef_r * psi_perm(r), r = 0, 1
        const R s = fwd ? sf : -sf;
        V h[2][3];
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
          for (int col = 0; col < 3; ++col)
            h[r][col] = coefmadd<R>(gcoef(mu, r), s, psi[3 * gperm(mu, r) + col], psi[3 * r + col]);
        V u[9];
        load_link<LS, R>(a.links, g.Vh, fwd ? p : q, mu, fwd ? cb : ycb, u);
        V uh[2][3];
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            V acc = cz<R>();
#pragma unroll
            for (int j = 0; j < 3; ++j) acc = fwd ? cmadd<R>(acc, u[3 * i + j], h[r][j]) : cmaddc<R>(acc, u[3 * j + i], h[r][j]);
            uh[r][i] = acc;
          }
        if (LS == L32R) {
          // lambda = -cc/2 times the boundary phase (conjugated for the backward link)
          const R lam = (R)g.lam[mu];
          V ph = mk<R>(lam, (R)0);
          if (wrap) ph = mk<R>(lam * (R)g.ph_re[mu], (fwd ? lam : -lam) * (R)g.ph_im[mu]);
#pragma unroll
          for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int i = 0; i < 3; ++i) uh[r][i] = cmul<R>(ph, uh[r][i]);
        }
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
          for (int i = 0; i < 3; ++i) res[3 * r + i] = add<R>(res[3 * r + i], uh[r][i]);
#pragma unroll
        for (int r = 2; r < 4; ++r)
#pragma unroll
          for (int i = 0; i < 3; ++i) res[3 * r + i] = coefmadd<R>(gcoef(mu, r), s, uh[gperm(mu, r)][i], res[3 * r + i]);
      }
    }
  }
  hop_epilogue<P, LK, LOOP>(a, io, active, n, cb, res, red_re, smem_d);
  tile += gridDim.x;
  } while (LOOP && tile < ntiles);
  if (a.red) {
    double* sm = smem_d + smat_smem_bytes(LK, (int)blockDim.x, sizeof(R)) / sizeof(double);
    block_reduce_finalize<false>(a.ra, red_re, 0.0, g.N5, g.Ls, g.nrhs, sm);
  }
}

// ---------------------------------------------------------------------------
// The hop for fields with an inner extent N5 = Ls * n_rhs (Mobius 5D fields,
// packed right-hand sides), FP32 or FP16 spinors, 18-real FP32 links.  A block
// covers S = blockDim / N5 4D sites with all their N5 inner sites (the same
// site -> thread mapping as dslash_kernel).  The N5 threads of a 4D site share
// its 8 neighbour indices and 8 links, which the block copies into shared
// memory as one record per site; each thread then streams its 8 neighbour
// spinors (coalesced 16-byte loads along the inner index) and runs the
// projected matvecs.  No link registers stay live across the loads.
// ---------------------------------------------------------------------------
constexpr int kHop5LinkStride = 41;  // hop5t_kernel: float4 per site (8 links x 5, +1 pad: site rows 4 banks apart)

// hop5t_kernel: links and neighbour indices of the S sites
__host__ __device__ inline size_t hop5_extra_smem(int S) {
  return (size_t)S * kHop5LinkStride * 16 + (size_t)S * 8 * 4;
}

// Resident blocks per SM the hop5 kernels are compiled for: 4 (64 registers)
// for the pure hop, 3 (80) with an epilogue or a looping reduction, the faster
// of each measured on GB300 (16^3x32, Ls 12: pure hop 52.6 us at 64 registers,
// 53.7 at 80; M of 12 packed Wilson-clover sources on 24^4 403 and 353 us)
#ifndef GBF_HOP5_MINB
#define GBF_HOP5_MINB 3
#endif
#ifndef GBF_HOP5_MINB_PURE
#define GBF_HOP5_MINB_PURE 4
#endif

// Order of the hop5 tiles.  lbx < 0: a tile is S consecutive checkerboard
// sites, and with slabT > 0 the (x2, x3) planes are visited slab by slab
// (slabT planes in x2, x3 slowest within a slab), so that a plane's x3
// neighbours are read while they are still in L2.  lbx >= 0: a tile is a
// brick of 2^lbx x 2^lby x 2^lbz x 2^lbt sites (x0/2, x1, x2, x3), whose
// neighbours in all four directions largely coincide (L1 reuse inside the
// block), and the bricks run x0 fastest within slabs of slabT planes in x2.
struct Hop5Order {
  int lbx, lby, lbz, lbt, slabT;
  FastDiv f0, f1, f2;  // by the bricks of a slab in x0, x1, x2
};

// The 4D sites of one tile in that order.
struct TileSites {
  const Geo& g;
  const Hop5Order& ord;
  int cb0;
  unsigned o0 = 0, o1 = 0, o2 = 0, o3 = 0;  // brick origin
  __device__ __forceinline__ TileSites(const Geo& g_, const Hop5Order& o, unsigned tile, int log2S) : g(g_), ord(o) {
    cb0 = (int)(tile << log2S);
    if (ord.lbx >= 0) {
      unsigned r = tile, qq;
      const unsigned n3 = (unsigned)g.L[3] >> ord.lbt;
      qq = ord.f0.div(r); o0 = (r - qq * ord.f0.d) << ord.lbx; r = qq;
      qq = ord.f1.div(r); o1 = (r - qq * ord.f1.d) << ord.lby; r = qq;
      qq = ord.f2.div(r); o2 = (r - qq * ord.f2.d) << ord.lbz; r = qq;
      qq = r / n3; o3 = (r - qq * n3) << ord.lbt;
      o2 += qq * (unsigned)ord.slabT;
    } else if (ord.slabT) {
      const unsigned pt = (unsigned)(g.Lh0 * g.L[1]) >> log2S;  // tiles per (x2, x3) plane
      const unsigned tp = tile / pt, w = tile - tp * pt;
      const unsigned r = tp / (unsigned)ord.slabT, x2 = tp - r * (unsigned)ord.slabT;
      const unsigned b = r / (unsigned)g.L[3], x3 = r - b * (unsigned)g.L[3];
      cb0 = (int)(((b * (unsigned)ord.slabT + x2 + (unsigned)g.L[2] * x3) * pt + w) << log2S);
    }
  }
  __device__ __forceinline__ int site(unsigned jj) const {
    if (ord.lbx < 0) return cb0 + (int)jj;
    const unsigned j0 = jj & ((1u << ord.lbx) - 1u);
    jj >>= ord.lbx;
    const unsigned j1 = jj & ((1u << ord.lby) - 1u);
    jj >>= ord.lby;
    const unsigned j2 = jj & ((1u << ord.lbz) - 1u), j3 = jj >> ord.lbz;
    return (int)((o0 + j0) + (unsigned)g.Lh0 * ((o1 + j1) + (unsigned)g.L[1] * ((o2 + j2) + (unsigned)g.L[2] * (o3 + j3))));
  }
};

// What a 4D site needs besides spinors is one record of 608 bytes: its eight
// links, the backward ones already U^dagger, and its eight neighbour indices
// (make_records_kernel, at gauge import).  Gathering links from their planes
// and computing the indices in every block was a chain of index arithmetic, two
// barriers and 72 scattered loads before the first matvec (without it a hop of
// 32^3x16, Ls 12 ran in 140 instead of 225 us); with records it took 217 ->
// 190 us, the reference's Dhop benchmark 1707 -> 1480 us.
constexpr unsigned kRecordWords = 38;
__device__ __forceinline__ void cp_async16(float4* dst, const float4* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(gaddr(src)) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Records of kRecordSites consecutive sites of parity blockIdx.y from the L32
// links: thread (d, j) gathers direction d of site j, and the block writes the
// records out in order.  It moves 1.2 KB per site and is bound by that; a thread
// that wrote its 72 bytes itself had 64 records in flight per warp and two
// sectors per store (16^3x32: 70 -> 18 us).
constexpr unsigned kRecordSites = 32;
__global__ void __launch_bounds__(8 * kRecordSites) make_records_kernel(Geo g, const float2* links, float2* records) {
  constexpr unsigned kPairs = 2 * kRecordWords, kStride = kPairs + 1;  // float2 per record; odd stride: distinct banks
  __shared__ float2 rec[kRecordSites * kStride];
  const unsigned Vh = (unsigned)g.Vh, p = blockIdx.y, cb0 = blockIdx.x * kRecordSites;
  const unsigned j = threadIdx.x % kRecordSites, d = threadIdx.x / kRecordSites, cb = cb0 + j, mu = d >> 1;
  const bool fwd = (d & 1u) == 0;
  if (cb < Vh) {
    const Coord c = cb_coords(g, (int)cb, (int)p);
    int y[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const int xm = c.x[m], Lm = g.L[m];
      y[m] = m != (int)mu ? xm : fwd ? (xm == Lm - 1 ? 0 : xm + 1) : (xm == 0 ? Lm - 1 : xm - 1);
    }
    const unsigned ycb = (unsigned)cb_index(g, y);
    const float2* L = links + ((size_t)(((fwd ? p : 1u - p) * 4u + mu) * 9u) * Vh + (fwd ? cb : ycb));
    float2* out = rec + j * kStride + 9 * d;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const float2 v = L[(size_t)(fwd ? 3 * i + k : 3 * k + i) * Vh];
        out[3 * i + k] = make_float2(v.x, fwd ? v.y : -v.y);
      }
    reinterpret_cast<int*>(rec + j * kStride + 72)[d] = (int)ycb;
  }
  __syncthreads();
  const unsigned n = (Vh - cb0 < kRecordSites ? Vh - cb0 : kRecordSites) * kPairs;
  float2* dst = records + ((size_t)p * Vh + cb0) * kPairs;
  for (unsigned e = threadIdx.x; e < n; e += blockDim.x) dst[e] = rec[e + e / kPairs];
}

template <int P, int LK, bool LOOP>
__global__ void __launch_bounds__(256, (LK != LOC_NONE || LOOP) ? GBF_HOP5_MINB : GBF_HOP5_MINB_PURE)
    hop5_kernel(const DslashArgs a, unsigned epi_off16, int log2S, const Hop5Order ord) {
  pdl_begin();
  using R = float;
  using V = float2;
  extern __shared__ __align__(16) double smem_d[];
  const Geo& g = a.g;
  const HopIO io = hop_io<!LOOP>(a);
  if (a.check_done && a.ra.st->all_done) return;
  const int p = io.p;
  const unsigned t = threadIdx.x, bd = blockDim.x;
  const unsigned N5 = (unsigned)g.N5;
  float4* recs = reinterpret_cast<float4*>(smem_d) + epi_off16;
  const unsigned j = g.fN5.div(t);
  const unsigned i5 = t - j * N5;
  double red_re = 0;
  const unsigned ntiles = ((unsigned)g.Vh + (1u << log2S) - 1) >> log2S;
  unsigned tile = blockIdx.x;
  do {
    const TileSites ts(g, ord, tile, log2S);
    const int cb = ts.site(j);
    const long long n = (long long)cb * N5 + i5;
    const bool active = cb < g.Vh;
    // the site's record, 38 words copied by the site's threads; the first
    // neighbour is requested meanwhile
    const float4* src = reinterpret_cast<const float4*>(a.records) + (size_t)p * (unsigned)g.Vh * kRecordWords + (size_t)cb * kRecordWords;
    float4* rec = recs + j * kRecordWords;
    V psi[12];
    // (in a loop a variable that only some branch sets carries its value of the
    // pass before: 24 registers through the epilogue, 290 bytes of spills)
    if (LOOP) {
#pragma unroll
      for (int k = 0; k < 12; ++k) psi[k] = cz<R>();
    }
    if (active) {
      for (unsigned c = i5; c < kRecordWords; c += N5) cp_async16(rec + c, src + c);
      load_spinor<P>(io.in, g.N, (unsigned)ldg(reinterpret_cast<const int*>(src + 36)) * N5 + i5, psi);
    }
    cp_async_wait_all();
    __syncthreads();
    V res[12];
#pragma unroll
    for (int k = 0; k < 12; ++k) res[k] = cz<R>();
    if (active) {
      const R sf = (R)a.sgn;
      const int* nbj = reinterpret_cast<const int*>(rec + 36);
#pragma unroll
      for (int mu = 0; mu < 4; ++mu) {
#pragma unroll
        for (int dir = 0; dir < 2; ++dir) {
          const int d = 2 * mu + dir;
          if (d > 0) load_spinor<P>(io.in, g.N, (unsigned)nbj[d] * N5 + i5, psi);
          const R s = dir == 0 ? sf : -sf;
          V h[2][3];
#pragma unroll
          for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int col = 0; col < 3; ++col)
              h[r][col] = coefmadd<R>(gcoef(mu, r), s, psi[3 * gperm(mu, r) + col], psi[3 * r + col]);
          V u[9];  // 72 bytes at 72 d: 16-byte reads from the aligned end
          {
            const char* lb = reinterpret_cast<const char*>(rec) + 72 * d;
            const int odd = dir;  // (72 d is a multiple of 16 for even d)
            if (odd) u[0] = *reinterpret_cast<const float2*>(lb);
            else u[8] = *reinterpret_cast<const float2*>(lb + 64);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const float4 w = *reinterpret_cast<const float4*>(lb + (odd ? 8 : 0) + 16 * c);
              u[2 * c + odd] = make_float2(w.x, w.y);
              u[2 * c + 1 + odd] = make_float2(w.z, w.w);
            }
          }
          V uh[2][3];
#pragma unroll
          for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int i = 0; i < 3; ++i) {
              V acc = cmul<R>(u[3 * i], h[r][0]);
              acc = cmadd<R>(acc, u[3 * i + 1], h[r][1]);
              uh[r][i] = cmadd<R>(acc, u[3 * i + 2], h[r][2]);
            }
#pragma unroll
          for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int i = 0; i < 3; ++i) res[3 * r + i] = add<R>(res[3 * r + i], uh[r][i]);
#pragma unroll
          for (int r = 2; r < 4; ++r)
#pragma unroll
            for (int i = 0; i < 3; ++i) res[3 * r + i] = coefmadd<R>(gcoef(mu, r), s, uh[gperm(mu, r)][i], res[3 * r + i]);
        }
      }
    }
    hop_epilogue<P, LK, LOOP>(a, io, active, n, cb, res, red_re, smem_d);
    tile += gridDim.x;
    if (LOOP) __syncthreads();  // the next tile overwrites the records
  } while (LOOP && tile < ntiles);
  if (a.red) {
    double* sm = smem_d + smat_smem_bytes(LK, (int)blockDim.x, sizeof(R)) / sizeof(double);
    block_reduce_finalize<false>(a.ra, red_re, 0.0, g.N5, g.Ls, g.nrhs, sm);
  }
}

// ---------------------------------------------------------------------------
// The same hop with two inner sites per thread (FP32 or FP16 spinors, 18-real
// FP32 links, per-thread or band epilogue).  Thread (j, h) of a block owns the
// sites i5 = 2h and 2h + 1 of 4D site j: the two share every link, so each link
// word read from shared memory feeds two sites, and the matvecs run in FP32
// pairs (lane x the even, lane y the odd site) at half the instructions.  With
// EVEN (N5 even and 32-byte aligned fields) the two sites' words of a component
// plane are one 256-bit access.
//
// Against hop5_kernel (us, hop alone): FP16 16^3x32 Ls 12 52.5 -> 46.5, 16^4 Ls
// 12 x 12 rhs 304 -> 269; FP32 16^4 Ls 12 x 6 153 -> 133, x 12 274 -> 268; FP32
// below 32 inner sites hop5_kernel's larger number of warps wins (Ls 12: 52.4
// against 54.0, with the band epilogue 281 against 302 for the normal
// operator).  Both are held up by the latency of what they load at 10 to 11
// TB/s from L2; prefetching the next direction into registers (167 of them) or
// into L1 did not help (+-3 %, 8 % slower).
// ---------------------------------------------------------------------------
struct Word8 {
  float4 a, b;  // the even and the odd site's word
};
__device__ __forceinline__ Word8 ldg8(const float4* p) {
  Word8 w;
  asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(w.a.x), "=f"(w.a.y), "=f"(w.a.z), "=f"(w.a.w), "=f"(w.b.x), "=f"(w.b.y), "=f"(w.b.z), "=f"(w.b.w)
               : "l"(gaddr(p)));
  return w;
}
__device__ __forceinline__ void stg8(float4* p, const float4 a, const float4 b) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(gaddr(p)), "f"(a.x), "f"(a.y), "f"(a.z), "f"(a.w),
               "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w)
               : "memory");
}
// plane words of sites n, n + 1 (the second only if two)
template <bool EVEN> __device__ __forceinline__ Word8 load_word8(const float4* p, bool two) {
  if constexpr (EVEN) return ldg8(p);
  Word8 w;
  w.a = ldg(p);
  w.b = two ? ldg(p + 1) : make_float4(0.f, 0.f, 0.f, 0.f);
  return w;
}
// The raw plane words of a pair of spinors: 6 for FP32; 3 and the scales for FP16
template <int P> struct PairRaw {
  Word8 w[P == P32 ? 6 : 3];
  float sa, sb;
};
template <int P, bool EVEN>
__device__ __forceinline__ void load_pair_raw(const void* base, unsigned N, unsigned n, bool two, PairRaw<P>& q) {
  const float4* p = reinterpret_cast<const float4*>(base) + n;
#pragma unroll
  for (unsigned k = 0; k < (P == P32 ? 6u : 3u); ++k) q.w[k] = load_word8<EVEN>(p + k * N, two);
  if constexpr (P == P16) {
    const float* sc = reinterpret_cast<const float*>(reinterpret_cast<const float4*>(base) + 3 * N) + n;
    if (EVEN) {
      const float2 t = ldg(reinterpret_cast<const float2*>(sc));
      q.sa = t.x;
      q.sb = t.y;
    } else {
      q.sa = ldg(sc);
      q.sb = two ? ldg(sc + 1) : 0.f;
    }
  }
}
__device__ __forceinline__ float2 half2_bits(float x) {
  const unsigned u = __float_as_uint(x);
  return __half22float2(*reinterpret_cast<const __half2*>(&u));
}
// component k of the two sites as FP32 numbers (FP16: without the scale)
template <int P> __device__ __forceinline__ void pair_comp(const PairRaw<P>& q, int k, float2& a, float2& b) {
  if constexpr (P == P32) {
    const Word8& w = q.w[k >> 1];
    a = (k & 1) ? make_float2(w.a.z, w.a.w) : make_float2(w.a.x, w.a.y);
    b = (k & 1) ? make_float2(w.b.z, w.b.w) : make_float2(w.b.x, w.b.y);
  } else {
    const Word8& w = q.w[k >> 2];
    const int e = k & 3;
    a = half2_bits(e == 0 ? w.a.x : e == 1 ? w.a.y : e == 2 ? w.a.z : w.a.w);
    b = half2_bits(e == 0 ? w.b.x : e == 1 ? w.b.y : e == 2 ? w.b.z : w.b.w);
  }
}
template <int P, bool EVEN>
__device__ __forceinline__ void load_pair(const void* base, unsigned N, unsigned n, bool two, float2 (&v)[2][12]) {
  PairRaw<P> q;
  load_pair_raw<P, EVEN>(base, N, n, two, q);
#pragma unroll
  for (int k = 0; k < 12; ++k) {
    pair_comp<P>(q, k, v[0][k], v[1][k]);
    if constexpr (P == P16) {
      v[0][k] = make_float2(v[0][k].x * q.sa, v[0][k].y * q.sa);
      v[1][k] = make_float2(v[1][k].x * q.sb, v[1][k].y * q.sb);
    }
  }
}
template <int P, bool EVEN>
__device__ __forceinline__ void store_pair(void* base, unsigned N, unsigned n, bool two, const float2 (&v)[2][12]) {
  if constexpr (P == P32 && EVEN) {
    float4* p = reinterpret_cast<float4*>(base) + n;
#pragma unroll
    for (int k = 0; k < 6; ++k)
      stg8(p + (unsigned)k * N, make_float4(v[0][2 * k].x, v[0][2 * k].y, v[0][2 * k + 1].x, v[0][2 * k + 1].y),
           make_float4(v[1][2 * k].x, v[1][2 * k].y, v[1][2 * k + 1].x, v[1][2 * k + 1].y));
  } else {
    store_spinor<P>(base, N, n, v[0]);
    if (two) store_spinor<P>(base, N, n + 1, v[1]);
  }
}

__device__ __forceinline__ float2 bc2(float x) { return make_float2(x, x); }

// Sum over the block of one double per site, sites in the order j N5 + i5 of
// the tile (2 per thread), per right-hand side, then block_reduce's last-block
// finalisation.  sm: max(bd, S N5) + 64 doubles.
__device__ __forceinline__ void pair_reduce_finalize(const RedArgs& r, double va, double vb, unsigned q, bool two, int SN5, int N5,
                                                     int Ls, int nrhs, double* sm) {
  const int t = threadIdx.x, bd = blockDim.x;
  sm[q] = va;
  if (two) sm[q + 1] = vb;
  __syncthreads();
  for (int k = SN5 >> 1; k >= N5; k >>= 1) {
    for (int e = t; e < k; e += bd) sm[e] += sm[e + k];
    __syncthreads();
  }
  if (nrhs == 1 && (bd & 31) == 0) {
    double v = 0.0;
    for (int e = t; e < N5; e += bd) v += sm[e];
    double* w = sm + (SN5 > bd ? SN5 : bd);
    const double2 s = block_sum_shfl<false>(v, 0.0, w);
    if (t == 0) r.partial[blockIdx.x] = s;
  } else {
    if (t < nrhs) {
      double ar = 0;
      for (int s = 0; s < Ls; ++s) ar += sm[t * Ls + s];
      r.partial[(size_t)blockIdx.x * nrhs + t] = make_double2(ar, 0.0);
      __threadfence();
    }
    __syncthreads();
  }
  // the last block adds the [block][rhs] partials in block order: thread r
  // of the first nrhs groups of `step` threads walks right-hand side r
  if (!last_block(r)) return;
  const FinState f = fin_load(r, t < nrhs ? t : 0);
  const int step = bd / nrhs;  // threads per right-hand side (bd >= nrhs)
  const int rhs = t % nrhs, lane = t / nrhs;
  double v = 0.0;
  if (lane < step)
    for (unsigned b = lane; b < gridDim.x; b += step) v += __ldcg(r.partial + (size_t)b * nrhs + rhs).x;
  __syncthreads();
  sm[t] = v;
  __syncthreads();
  if (t < nrhs) {
    double sum = 0;
    for (int j = 0; j < step; ++j) sum += sm[j * nrhs + t];
    finalize(r, t, sum, 0.0, f);
    __threadfence();
  }
  __syncthreads();
  if (t == 0) {
    int all = 1;
    if (r.fin == FIN_BETA || r.fin == FIN_INIT)
      for (int rhs = 0; rhs < nrhs; ++rhs) all &= __ldcg(&r.st->done[rhs]);
    finalize_all(r, all, f);
  }
}

// MODE 0: one parity, 1: the same with a loop over tiles (reductions), 2: both
// parities (pointers by blockIdx.y, which the other two keep in the argument)
template <int P, int LK, int MODE, bool EVEN>
__global__ void __launch_bounds__(256, 2) hop5p_kernel(const DslashArgs a, unsigned epi_off16, int log2S, FastDiv fH, const Hop5Order ord) {
  pdl_begin();
  constexpr bool LOOP = MODE == 1;
  using V = float2;
  extern __shared__ __align__(16) double smem_d[];
  const Geo& g = a.g;
  const HopIO io = hop_io<MODE == 2>(a);
  if (a.check_done && a.ra.st->all_done) return;
  const int p = io.p, q = 1 - p;
  const unsigned t = threadIdx.x, bd = blockDim.x;
  const unsigned S = 1u << log2S, N = (unsigned)g.N, N5 = (unsigned)g.N5;
  float4* recs = reinterpret_cast<float4*>(smem_d) + epi_off16;
  const unsigned j = fH.div(t);             // 4D site of this thread within the tile
  const unsigned e = t - j * fH.d, i5 = 2u * e;  // its place among the site's threads, its first inner site
  const bool two = EVEN || i5 + 1 < N5;     // whether it has a second one
  const unsigned loc = j * N5 + i5;         // position of the first in the tile
  double ra = 0, rb = 0;
  const unsigned ntiles = ((unsigned)g.Vh + S - 1) >> log2S;
  unsigned tile = blockIdx.x;
  do {
    const TileSites ts(g, ord, tile, log2S);
    const int cb = ts.site(j);
    const unsigned n = (unsigned)cb * N5 + i5;
    const bool active = cb < g.Vh;
    // the site's record, 38 words copied by the site's threads; the first
    // neighbour is requested meanwhile
    const float4* src = reinterpret_cast<const float4*>(a.records) + (size_t)p * (unsigned)g.Vh * kRecordWords + (size_t)cb * kRecordWords;
    float4* rec = recs + j * kRecordWords;
    PairRaw<P> raw;
    if (LOOP) raw = PairRaw<P>{};  // not carried from the pass before (hop5_kernel): 1 KB of spills without
    if (active) {
      for (unsigned c = e; c < kRecordWords; c += fH.d) cp_async16(rec + c, src + c);
      load_pair_raw<P, EVEN>(io.in, N, (unsigned)ldg(reinterpret_cast<const int*>(src + 36)) * N5 + i5, two, raw);
    }
    cp_async_wait_all();
    __syncthreads();
    float2 re[12], im[12];  // lane x: the even site, lane y: the odd one
#pragma unroll
    for (int k = 0; k < 12; ++k) re[k] = im[k] = make_float2(0.f, 0.f);
    if (active) {
      const float sf = a.sgn;
      const int* nbj = reinterpret_cast<const int*>(rec + 36);
#pragma unroll
      for (int mu = 0; mu < 4; ++mu) {
#pragma unroll
        for (int dir = 0; dir < 2; ++dir) {
          const int d = 2 * mu + dir;
          if (d > 0) load_pair_raw<P, EVEN>(io.in, N, (unsigned)nbj[d] * N5 + i5, two, raw);
          const float s = dir == 0 ? sf : -sf;
          float2 hr[2][3], hi[2][3];
#pragma unroll
          for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int col = 0; col < 3; ++col) {
              V ua, ub, la, lb;
              pair_comp<P>(raw, 3 * r + col, ua, ub);
              pair_comp<P>(raw, 3 * gperm(mu, r) + col, la, lb);
              const V ha = coefmadd<float>(gcoef(mu, r), s, la, ua), hb = coefmadd<float>(gcoef(mu, r), s, lb, ub);
              hr[r][col] = make_float2(ha.x, hb.x);
              hi[r][col] = make_float2(ha.y, hb.y);
              if constexpr (P == P16) {  // the scales, on the projected half
                const float2 sc = make_float2(raw.sa, raw.sb);
                hr[r][col] = __fmul2_rn(sc, hr[r][col]);
                hi[r][col] = __fmul2_rn(sc, hi[r][col]);
              }
            }
          V u[9];  // 72 bytes at 72 d: 16-byte reads from the aligned end
          {
            const char* lb = reinterpret_cast<const char*>(rec) + 72 * d;
            const int odd = dir;  // (72 d is a multiple of 16 for even d)
            if (odd) u[0] = *reinterpret_cast<const float2*>(lb);
            else u[8] = *reinterpret_cast<const float2*>(lb + 64);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const float4 w = *reinterpret_cast<const float4*>(lb + (odd ? 8 : 0) + 16 * c);
              u[2 * c + odd] = make_float2(w.x, w.y);
              u[2 * c + 1 + odd] = make_float2(w.z, w.w);
            }
          }
          float2 tr[2][3], ti[2][3];
#pragma unroll
          for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              const float2 ux = bc2(u[3 * i + c].x), uy = bc2(u[3 * i + c].y), ny = bc2(-u[3 * i + c].y);
#pragma unroll
              for (int r = 0; r < 2; ++r) {
                tr[r][i] = c == 0 ? __fmul2_rn(ux, hr[r][c]) : __ffma2_rn(ux, hr[r][c], tr[r][i]);
                tr[r][i] = __ffma2_rn(ny, hi[r][c], tr[r][i]);
                ti[r][i] = c == 0 ? __fmul2_rn(ux, hi[r][c]) : __ffma2_rn(ux, hi[r][c], ti[r][i]);
                ti[r][i] = __ffma2_rn(uy, hr[r][c], ti[r][i]);
              }
            }
#pragma unroll
          for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int i = 0; i < 3; ++i) {
              re[3 * r + i] = __fadd2_rn(re[3 * r + i], tr[r][i]);
              im[3 * r + i] = __fadd2_rn(im[3 * r + i], ti[r][i]);
            }
#pragma unroll
          for (int r = 2; r < 4; ++r) {
            const int code = gcoef(mu, r), f = gperm(mu, r);
            const float2 sp = bc2((code & 1) ? -s : s), sm = bc2((code & 1) ? s : -s);
#pragma unroll
            for (int i = 0; i < 3; ++i) {
              if (code < 2) {
                re[3 * r + i] = __ffma2_rn(sp, tr[f][i], re[3 * r + i]);
                im[3 * r + i] = __ffma2_rn(sp, ti[f][i], im[3 * r + i]);
              } else {
                re[3 * r + i] = __ffma2_rn(sm, ti[f][i], re[3 * r + i]);
                im[3 * r + i] = __ffma2_rn(sp, tr[f][i], im[3 * r + i]);
              }
            }
          }
        }
      }
    }
    V v[2][12];
#pragma unroll
    for (int k = 0; k < 12; ++k) {
      v[0][k] = make_float2(re[k].x, im[k].x);
      v[1][k] = make_float2(re[k].y, im[k].y);
    }
    // ---- epilogue: out = c1 L1(hop) + c2 L2(X), reduction ----
    if (LK == LOC_BAND) {
      if (a.l1.kind == LOC_BAND) band_apply_pair<LOOP>(a.l1, g.Ls, g.fLs, (int)(S * N5), (int)loc, two, reinterpret_cast<float2*>(smem_d), v);
    } else if (active && a.l1.kind != LOC_NONE) {
      local_apply_thread<float>(a.l1, g.Vh, p, cb, v[0]);
      if (two) local_apply_thread<float>(a.l1, g.Vh, p, cb, v[1]);
    }
    if (active) {
      if (!a.c1.is_one()) {
        const float c1 = a.c1.h;
#pragma unroll
        for (int k = 0; k < 12; ++k) {
          v[0][k] = scl<float>(c1, v[0][k]);
          v[1][k] = scl<float>(c1, v[1][k]);
        }
      }
      if (io.X) {
        V x[2][12];
        if (LK == LOC_BAND && a.l2.kind == LOC_BAND) {
          const int s0 = (int)(i5 - g.fLs.div(i5) * (unsigned)g.Ls), s1 = (int)(i5 + 1 - g.fLs.div(i5 + 1) * (unsigned)g.Ls);
          band_load<P>(a.l2, g.Ls, s0, io.X, N, n, x[0]);
          if (two) band_load<P>(a.l2, g.Ls, s1, io.X, N, n + 1, x[1]);
          else {
#pragma unroll
            for (int k = 0; k < 12; ++k) x[1][k] = make_float2(0.f, 0.f);
          }
        } else {
          load_pair<P, EVEN>(io.X, N, n, two, x);
        }
        if (LK == LOC_CLOVER && a.l2.kind != LOC_NONE) {
          local_apply_thread<float>(a.l2, g.Vh, p, cb, x[0]);
          if (two) local_apply_thread<float>(a.l2, g.Vh, p, cb, x[1]);
        }
        const float c2 = a.c2.h;
#pragma unroll
        for (int k = 0; k < 12; ++k) {
          v[0][k] = cfma_s<float>(c2, x[0][k], v[0][k]);
          if (two) v[1][k] = cfma_s<float>(c2, x[1][k], v[1][k]);
        }
      }
      if (a.red) {
        if (a.red == 1) {
          V y[2][12];
          load_pair<P, EVEN>(a.Y, N, n, two, y);
          ra += site_dot_re<float>(y[0], v[0]);
          if (two) rb += site_dot_re<float>(y[1], v[1]);
        } else {
          ra += site_norm2<float>(v[0]);
          if (two) rb += site_norm2<float>(v[1]);
        }
      }
      store_pair<P, EVEN>(io.out, N, n, two, v);
    }
    tile += gridDim.x;
    if (LOOP) __syncthreads();  // the next tile overwrites the records
  } while (LOOP && tile < ntiles);
  if (a.red) {
    double* sm = smem_d + smat_smem_bytes(LK, (int)(S * N5), 4) / sizeof(double);
    pair_reduce_finalize(a.ra, ra, rb, loc, two, (int)(S * N5), g.N5, g.Ls, g.nrhs, sm);
  }
}

// ---------------------------------------------------------------------------
// The hop of hop5_kernel with the neighbour spinors staged in shared memory
// by 1D bulk copies (cp.async.bulk, global -> shared, completion counted in
// bytes on an mbarrier), FP32 spinors.  For a tile of S 4D sites and
// direction d, the N5 inner sites of site j's neighbour are, in each of the
// 6 16-byte component planes of the FP32 layout, one contiguous run of
// N5 * 16 bytes; 6 S copies move them into a ring slot laid out
// [plane][site j][i5], i.e. [plane][thread].  A ring of kRing direction
// slots keeps kRing - 1 directions in flight while one is computed; thread 0
// waits for a slot's barrier (bounded) and a block barrier publishes the data
// and frees the slot used before, which the copy threads then refill.  The
// ring doubles as the epilogue's shared memory once the 8 directions are
// done.  A wait that runs out sets st->kernel_error and the block returns
// (all its threads together, after any copy still in flight has landed).
// ---------------------------------------------------------------------------
constexpr int kRing = 4;

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// bounded wait for the phase of `parity` to complete: about 1 s of SM clocks
__device__ __forceinline__ bool mbar_wait_bounded(unsigned long long* bar, unsigned parity) {
  const unsigned addr = smem_u32(bar);
  const long long t0 = clock64();
  while (true) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(addr), "r"(parity)
        : "memory");
    if (ok) return true;
    if (clock64() - t0 > 2000000000LL) return false;
  }
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, unsigned bytes, unsigned long long* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

__host__ __device__ inline size_t hop5t_ring_bytes(int bd) { return (size_t)kRing * 6 * 16 * bd; }

template <int LK, bool LOOP>
__global__ void __launch_bounds__(256, GBF_HOP5_MINB) hop5t_kernel(const DslashArgs a, int log2S, unsigned links_off16) {
  pdl_begin();
  using R = float;
  using V = float2;
  extern __shared__ __align__(128) double smem_d[];
  const Geo& g = a.g;
  if (a.check_done && a.ra.st->all_done) return;
  const int p = a.out_parity, q = 1 - p;
  const unsigned t = threadIdx.x, bd = blockDim.x;
  const unsigned S = 1u << log2S;
  const unsigned N = (unsigned)g.N, N5 = (unsigned)g.N5;
  float4* ring = reinterpret_cast<float4*>(smem_d);  // [kRing][6][bd], later the epilogue's region
  float4* lsm = reinterpret_cast<float4*>(smem_d) + links_off16;  // after max(ring, epilogue)
  int* nbs = reinterpret_cast<int*>(lsm + S * kHop5LinkStride);
  unsigned long long* full = reinterpret_cast<unsigned long long*>(nbs + 8 * S);
  __shared__ int s_ok;
  if (t == 0) {
    for (int r = 0; r < kRing; ++r) mbar_init(&full[r], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  unsigned par_bits = 0;  // completion parity of each slot, the same in every thread
  const unsigned j = g.fN5.div(t);
  const unsigned i5 = t - j * N5;
  double red_re = 0;
  const long long ntiles = (g.N + bd - 1) / bd;
  long long tile = blockIdx.x;
  do {
    const int cb0 = (int)(tile << log2S);
    const unsigned s_act = (unsigned)min((long long)S, (long long)g.Vh - cb0);  // sites of this tile
    for (unsigned idx = t; idx < 8 * S; idx += bd) {
      const int jj = idx >> 3, d = idx & 7, cbj = cb0 + jj;
      int ycb = 0;
      if (cbj < g.Vh) {
        const Coord c = cb_coords(g, cbj, p);
        const int mu = d >> 1;
        int y[4] = {c.x[0], c.x[1], c.x[2], c.x[3]};
        if ((d & 1) == 0) y[mu] = (y[mu] == g.L[mu] - 1) ? 0 : y[mu] + 1;
        else y[mu] = (y[mu] == 0) ? g.L[mu] - 1 : y[mu] - 1;
        ycb = cb_index(g, y);
      }
      nbs[idx] = ycb;
    }
    __syncthreads();
    // issue direction d into its slot: thread 0 posts the expected bytes,
    // threads 0 .. 6 s_act - 1 each copy one plane run of one site
    auto issue = [&](int d) {
      const int slot = d % kRing;
      if (t < 6 * s_act) {
        if (t == 0) mbar_arrive_expect_tx(&full[slot], 6 * s_act * N5 * 16);
        const unsigned jj = t / 6, k = t - 6 * jj;
        const unsigned ycb = (unsigned)nbs[jj * 8 + d];
        const float4* src = reinterpret_cast<const float4*>(a.in) + (k * N + ycb * N5);
        float4* dst = ring + ((unsigned)slot * 6 + k) * bd + jj * N5;
        bulk_g2s(dst, src, N5 * 16, &full[slot]);
      }
    };
    // the ring was last written by the generic proxy (previous epilogue)
    if (t < 6 * s_act) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
#pragma unroll
    for (int d = 0; d < kRing; ++d) issue(d);
    {
      const float2* L2 = reinterpret_cast<const float2*>(a.links);
      float* lf = reinterpret_cast<float*>(lsm);
      for (unsigned idx = t; idx < 72u * S; idx += bd) {
        const unsigned jj = idx & (S - 1), dk = idx >> log2S;
        const unsigned d = dk / 9u, k = dk - 9u * d;
        const int cbj = cb0 + (int)jj;
        if (cbj >= g.Vh) continue;
        const int mu = d >> 1;
        const bool fwd = (d & 1) == 0;
        const int site = fwd ? cbj : nbs[jj * 8 + d];
        const int par = fwd ? p : q;
        float2 v = ldg(L2 + ((unsigned)((par * 4 + mu) * 9) + k) * (unsigned)g.Vh + (unsigned)site);
        unsigned kk = k;
        if (!fwd) {
          kk = (k % 3u) * 3u + k / 3u;
          v.y = -v.y;
        }
        *reinterpret_cast<float2*>(lf + (jj * kHop5LinkStride + d * 5u) * 4u + 2u * kk) = v;
      }
    }
    const long long n = tile * bd + t;
    const int cb = cb0 + (int)j;
    const bool active = cb < g.Vh;
    V res[12];
#pragma unroll
    for (int k = 0; k < 12; ++k) res[k] = cz<R>();
    const R sf = (R)a.sgn;
    const float4* lj = lsm + j * kHop5LinkStride;
#pragma unroll
    for (int mu = 0; mu < 4; ++mu) {
#pragma unroll
      for (int dir = 0; dir < 2; ++dir) {
        const int d = 2 * mu + dir;
        const int slot = d % kRing;
        if (t == 0) s_ok = mbar_wait_bounded(&full[slot], (par_bits >> slot) & 1u) ? 1 : 0;
        par_bits ^= 1u << slot;
        __syncthreads();  // slot d published (and the links); every thread is done with direction d - 1
        if (!s_ok) {
          if (t == 0) {
            atomicExch(&a.ra.st->kernel_error, 1);
            // let any copy of this block still in flight land before the
            // block's shared memory is released (about 0.1 s)
            for (int w = 0; w < 100000; ++w) __nanosleep(1000);
          }
          __syncthreads();
          return;
        }
        if (d >= 1 && d - 1 + kRing < 8) issue(d - 1 + kRing);
        if (active) {
          const bool fwd = dir == 0;
          V psi[12];
          const float4* src = ring + (unsigned)slot * 6 * bd + t;
#pragma unroll
          for (int k = 0; k < 6; ++k) {
            const float4 w = src[k * bd];
            psi[2 * k] = make_float2(w.x, w.y);
            psi[2 * k + 1] = make_float2(w.z, w.w);
          }
          const R s = fwd ? sf : -sf;
          V h[2][3];
#pragma unroll
          for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int col = 0; col < 3; ++col)
              h[r][col] = coefmadd<R>(gcoef(mu, r), s, psi[3 * gperm(mu, r) + col], psi[3 * r + col]);
          V u[10];
#pragma unroll
          for (int c = 0; c < 5; ++c) {
            const float4 w = lj[d * 5 + c];
            u[2 * c] = make_float2(w.x, w.y);
            u[2 * c + 1] = make_float2(w.z, w.w);
          }
          V uh[2][3];
#pragma unroll
          for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int i = 0; i < 3; ++i) {
              V acc = cmul<R>(u[3 * i], h[r][0]);
              acc = cmadd<R>(acc, u[3 * i + 1], h[r][1]);
              uh[r][i] = cmadd<R>(acc, u[3 * i + 2], h[r][2]);
            }
#pragma unroll
          for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int i = 0; i < 3; ++i) res[3 * r + i] = add<R>(res[3 * r + i], uh[r][i]);
#pragma unroll
          for (int r = 2; r < 4; ++r)
#pragma unroll
            for (int i = 0; i < 3; ++i) res[3 * r + i] = coefmadd<R>(gcoef(mu, r), s, uh[gperm(mu, r)][i], res[3 * r + i]);
        }
      }
    }
    __syncthreads();  // the ring becomes the epilogue's shared memory
    hop_epilogue<P32, LK, LOOP>(a, hop_io(a), active, n, cb, res, red_re, smem_d);
    tile += gridDim.x;
    __syncthreads();  // the next tile refills the ring and the indices
  } while (LOOP && tile < ntiles);
  if (a.red) {
    double* sm = smem_d + smat_smem_bytes(LK, (int)blockDim.x, sizeof(R)) / sizeof(double);
    block_reduce_finalize<false>(a.ra, red_re, 0.0, g.N5, g.Ls, g.nrhs, sm);
  }
}

// ---------------------------------------------------------------------------
// The pure double-float hop (no site-local term, X term or reduction) with two
// threads per 5D site, one right-hand side.  Thread r = 0, 1 of a site projects
// the half spinor h_r = psi_r + s coef psi_perm(r) of every direction, multiplies
// it by the link and accumulates it into upper spin r and into the lower spin
// that takes h_r in that direction; its accumulators (upper spin r, both lower
// spins: 9 double-float complex numbers) live in shared memory.  After the 8
// directions the pair exchanges partial sums through shared memory and thread r
// stores spins 2r and 2r+1.  Against dslash_kernel<PDD> this halves the
// registers a thread needs (same arithmetic per site), so about twice the warps
// are resident to cover the latency of the double-float operation chains.  The
// lower spins are summed as thread 0's directions plus thread 1's (a fixed order).
// ---------------------------------------------------------------------------
#ifndef GBF_DD2_MINB
#define GBF_DD2_MINB 3
#endif
constexpr int kDD2Acc = 9;  // accumulators per thread: upper spin r (3), lower spins 2, 3 (6)

__device__ __forceinline__ cplx<dd> f4dd(const float4 q) { return mk<dd>(dd(q.x, q.z), dd(q.y, q.w)); }
__device__ __forceinline__ float4 ddf4(cplx<dd> v) {
  nrm<dd>(v);
  return make_float4(v.x.h, v.y.h, v.x.l, v.y.l);
}

__global__ void __launch_bounds__(256, GBF_DD2_MINB) dslash_dd2_kernel(const DslashArgs a) {
  pdl_begin();
  extern __shared__ __align__(16) double smem_d[];
  const Geo& g = a.g;
  const HopIO io = hop_io(a);
  if (a.check_done && a.ra.st->all_done) return;
  const int p = io.p, q = 1 - p;
  const unsigned t = threadIdx.x, bs = blockDim.x;
  const unsigned r = t & 1u;
  const unsigned sites = bs >> 1;
  float4* acc = reinterpret_cast<float4*>(smem_d) + t;  // [kDD2Acc][bs]
  const unsigned N = (unsigned)g.N;
  const float4* sp = reinterpret_cast<const float4*>(io.in);
  const float4* lk = reinterpret_cast<const float4*>(a.links);
  const long long n = (long long)blockIdx.x * sites + (t >> 1);
  const bool active = n < g.N;
  int cb = 0;
  if (active) {
    cb = (int)g.fN5.div((unsigned)n);
    const unsigned i5 = (unsigned)n - (unsigned)cb * (unsigned)g.N5;
    const Coord c = cb_coords(g, cb, p);
#pragma unroll
    for (int k = 0; k < kDD2Acc; ++k) acc[k * bs] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
    for (int d = 0; d < 8; ++d) {
      const int mu = d >> 1;
      const bool fwd = (d & 1) == 0;
      int y[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const int xm = c.x[m], Lm = g.L[m];
        y[m] = (m != mu) ? xm : fwd ? (xm == Lm - 1 ? 0 : xm + 1) : (xm == 0 ? Lm - 1 : xm - 1);
      }
      const int ycb = cb_index(g, y);
      const unsigned site = (unsigned)ycb * (unsigned)g.N5 + i5;
      const float s = fwd ? a.sgn : -a.sgn;
      const int pr = gperm(mu, (int)r), cr = gcoef(mu, (int)r);
      {
        // lane-paired form: a complex double-float is one pdd, u h is
        // Re(u) h + Im(u) (i h), two lane-wise fmas per link entry
        pdd h[3], ih[3];
#pragma unroll
        for (int col = 0; col < 3; ++col) {
          const pdd up = pdd_ld(ldg(sp + (site + (3u * r + col) * N)));
          const pdd lo = pdd_ld(ldg(sp + (site + (unsigned)(3 * pr + col) * N)));
          h[col] = pdd_coefmadd_rt(cr, s, lo, up);
          ih[col] = pdd_i(h[col]);
        }
        const int rl = (gperm(mu, 2) == (int)r) ? 2 : 3;
        const int cl = gcoef(mu, rl);
        const float4* L = lk + (unsigned)(((fwd ? p : q) * 4 + mu) * 9) * (unsigned)g.Vh + (unsigned)(fwd ? cb : ycb);
        const float cs = fwd ? 1.f : -1.f;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          pdd uh;
#pragma unroll
          for (int j = 0; j < 3; ++j) {
            const unsigned k = fwd ? (unsigned)(3 * i + j) : (unsigned)(3 * j + i);
            const float4 qv = ldg(L + k * (unsigned)g.Vh);
            const dd ux(qv.x, qv.z), uy = dd_scale2(cs, dd(qv.y, qv.w));  // U or U^dagger entry
            uh = j == 0 ? pdd_mul_s(ux, h[j]) : pdd_fma_s(ux, h[j], uh);
            uh = pdd_fma_s(uy, ih[j], uh);
          }
          // (the sums leave pdd_add normalised)
          float4& m = acc[i * bs];
          m = pdd_st(pdd_add(pdd_ld(m), uh));
          float4& ml = acc[(3 + 3 * (rl - 2) + i) * bs];
          ml = pdd_st(pdd_coefmadd_rt(cl, s, uh, pdd_ld(ml)));
        }
      }
    }
  }
  __syncwarp();  // the partner's accumulators are visible
  ddc w[6];
  if (active) {
    const float4* mine = reinterpret_cast<const float4*>(smem_d) + t;
    const float4* other = reinterpret_cast<const float4*>(smem_d) + (t ^ 1u);
    if (r == 0) {  // spins 0 and 1: own upper sums and the partner's
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        w[i] = f4dd(mine[i * bs]);
        w[3 + i] = f4dd(other[i * bs]);
      }
    } else {  // spins 2 and 3: thread 0's partial plus thread 1's
#pragma unroll
      for (int k = 0; k < 6; ++k) w[k] = add<dd>(f4dd(other[(3 + k) * bs]), f4dd(mine[(3 + k) * bs]));
    }
  }
  if (active) {
    float4* out = reinterpret_cast<float4*>(io.out);
#pragma unroll
    for (int k = 0; k < 6; ++k) out[(unsigned)n + (6u * r + k) * N] = ddf4(w[k]);
  }
}

// ---------------------------------------------------------------------------
// The hop with eight threads per 5D site (per-thread epilogue, one
// right-hand side): thread (d, j) of a block computes the upper half of
// direction d's term for site j (projection and link; d = mu forward, d =
// 4 + mu backward) and leaves its 6 components in shared memory; after a
// barrier thread (q, j), q < 6, sums components 2q and 2q + 1 over the
// directions in dslash_kernel's order, rebuilding the lower spins from the
// upper ones, and applies the epilogue to them, the clover term row by row.  A warp
// holds two directions of the same sense for 16 consecutive sites.
// ---------------------------------------------------------------------------
constexpr int kHop8Block = 8 * kSplitSites;

// a + s coef v with run-time coefficient code and sign s = +-1
template <typename R>
__device__ __forceinline__ cplx<R> coefmadd_rt(int code, float s, cplx<R> v, cplx<R> a) {
  // (the factors are selected, not converted: a float-to-double conversion
  // would cost as much as an FP64 multiply-add)
  const bool im = code >= 2, neg = ((code & 1) != 0) != (s < 0.f);
  const R sy = neg ? R(-1) : R(1), sx = neg != im ? R(-1) : R(1);
  return mk<R>(fma(sx, im ? v.y : v.x, a.x), fma(sy, im ? v.x : v.y, a.y));
}

// The upper two spins of one direction of one site: out[(3 r + i) * stride]
template <int P, int LS, bool FWD>
__device__ __forceinline__ void hop8_term(const DslashArgs& a, const HopIO& io, unsigned cb, unsigned i5, int mu,
                                          typename SplitWord<typename SpinorT<P>::R>::T* out, unsigned stride) {
  using R = typename SpinorT<P>::R;
  using V = cplx<R>;
  const Geo& g = a.g;
  const int p = io.p, q = 1 - p;
  const Coord c = cb_coords(g, (int)cb, p);
  int y[4];
  bool wrap = false;
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const int xm = c.x[m], Lm = g.L[m];
    const bool w = FWD ? xm == Lm - 1 : xm == 0;
    y[m] = (m != mu) ? xm : FWD ? (w ? 0 : xm + 1) : (w ? Lm - 1 : xm - 1);
    wrap = wrap || (m == mu && w);
  }
  const int ycb = cb_index(g, y);
  const unsigned site = (unsigned)ycb * (unsigned)g.N5 + i5;
  const float s = FWD ? a.sgn : -a.sgn;
  const int lp = FWD ? p : q, lcb = FWD ? (int)cb : ycb;
  if constexpr (P == PDD) {
    const float4* sp = reinterpret_cast<const float4*>(io.in);
    const unsigned N = (unsigned)g.N;
    pdd h[2][3], uh[2][3];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int pr = gperm(mu, r), cr = gcoef(mu, r);
#pragma unroll
      for (int col = 0; col < 3; ++col) {
        const pdd up = pdd_ld(ldg(sp + (site + (unsigned)(3 * r + col) * N)));
        const pdd lo = pdd_ld(ldg(sp + (site + (unsigned)(3 * pr + col) * N)));
        h[r][col] = pdd_coefmadd_rt(cr, s, lo, up);
      }
    }
    const float4* L = reinterpret_cast<const float4*>(a.links) + (unsigned)((lp * 4 + mu) * 9) * (unsigned)g.Vh + (unsigned)lcb;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const float4 qv = ldg(L + (unsigned)(FWD ? 3 * i + j : 3 * j + i) * (unsigned)g.Vh);
        const dd ux(qv.x, qv.z), uy = FWD ? dd(qv.y, qv.w) : dd(-qv.y, -qv.w);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          uh[r][i] = j == 0 ? pdd_mul_s(ux, h[r][j]) : pdd_fma_s(ux, h[r][j], uh[r][i]);
          uh[r][i] = pdd_fma_s(uy, pdd_i(h[r][j]), uh[r][i]);
        }
      }
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int i = 0; i < 3; ++i) out[(3 * r + i) * stride] = pdd_st(uh[r][i]);
  } else {
    V psi[12], u[9], h[2][3];
    load_spinor<P>(io.in, g.N, site, psi);
    load_link<LS, R>(a.links, g.Vh, lp, mu, lcb, u);
    const bool sw = mu < 2;  // spin 0 projects with spin 3 (mu < 2) or 2
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int col = 0; col < 3; ++col)
        h[r][col] = coefmadd_rt<R>(gcoef(mu, r), s, (r == 0) == sw ? psi[9 + col] : psi[6 + col], psi[3 * r + col]);
    V ph = cz<R>();
    if constexpr (LS == L32R) {
      const R lam = (R)g.lam[mu];
      ph = mk<R>(lam, (R)0);
      if (wrap) ph = mk<R>(lam * (R)g.ph_re[mu], (FWD ? lam : -lam) * (R)g.ph_im[mu]);
    }
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        V t = cz<R>();
#pragma unroll
        for (int j = 0; j < 3; ++j) t = FWD ? cmadd<R>(t, u[3 * i + j], h[r][j]) : cmaddc<R>(t, u[3 * j + i], h[r][j]);
        out[(3 * r + i) * stride] = LS == L32R ? cmul<R>(ph, t) : t;
      }
  }
}

// Component k of the sum over the directions of the terms con[d][0..5][j]
template <int P, typename W>
__device__ __forceinline__ cplx<typename SpinorT<P>::R> hop8_sum(const W (*con)[6][kSplitSites], unsigned j, unsigned k, float sgn) {
  using R = typename SpinorT<P>::R;
  const bool low = k >= 6;
  const unsigned l = k >= 9 ? 1u : 0u, i = k - (k / 3u) * 3u;  // lower spin 2 + l
  cplx<R> v = cz<R>();
  pdd t{make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
  for (int m = 0; m < 8; ++m) {
    const int mu = m >> 1, d = (m & 1) ? 4 + mu : mu;  // as dslash_kernel: forward, backward of each mu
    // upper component k itself, or the upper spin that feeds lower spin 2 + l
    const unsigned e = low ? 3u * (mu < 2 ? 1u - l : l) + i : k;
    const W w = con[d][e][j];
    const int code = low ? (l ? gcoef(mu, 3) : gcoef(mu, 2)) : 0;
    const float s = low ? (d < 4 ? sgn : -sgn) : 1.f;
    if constexpr (P == PDD) t = pdd_coefmadd_rt(code, s, pdd_ld(w), t);
    else v = coefmadd_rt<R>(code, s, split_unpack(w), v);
  }
  if constexpr (P == PDD) v = split_unpack(pdd_st(t));
  return v;
}

#ifndef GBF_HOP8_MINB_DD
#define GBF_HOP8_MINB_DD 4
#endif
template <int P, int LS, bool LOOP>
__global__ void __launch_bounds__(kHop8Block, P == P64 ? 4 : P == PDD ? GBF_HOP8_MINB_DD : 6) hop8_kernel(const DslashArgs a) {
  pdl_begin();
  using R = typename SpinorT<P>::R;
  using V = cplx<R>;
  using W = typename SplitWord<R>::T;
  __shared__ W con[8][6][kSplitSites];  // the directions' terms
  __shared__ W sum[12][kSplitSites];    // their sum (clover epilogue)
  __shared__ double red_sm[64];
  const Geo& g = a.g;
  const HopIO io = hop_io<!LOOP>(a);
  if (a.check_done && a.ra.st->all_done) return;
  const int p = io.p;
  const unsigned j = threadIdx.x & (kSplitSites - 1), q = threadIdx.x / kSplitSites;
  const unsigned N = (unsigned)g.N, Vh = (unsigned)g.Vh;
  double red_re = 0;
  const unsigned ntiles = (N + kSplitSites - 1) / kSplitSites;
  unsigned tile = blockIdx.x;
  do {
    const unsigned n = tile * kSplitSites + j;
    const bool active = n < N;
    unsigned cb = 0;
    if (active) {
      cb = g.fN5.div(n);
      const unsigned i5 = n - cb * (unsigned)g.N5;
      if (q < 4) hop8_term<P, LS, true>(a, io, cb, i5, (int)q, &con[q][0][j], kSplitSites);
      else hop8_term<P, LS, false>(a, io, cb, i5, (int)q - 4, &con[q][0][j], kSplitSites);
    }
    __syncthreads();
    const bool own = active && q < 6;
    V v[2];
    if (LOOP) v[0] = v[1] = cz<R>();  // not carried from the pass before (hop5_kernel)
    if (own) {
      v[0] = hop8_sum<P>(con, j, 2 * q, a.sgn);
      v[1] = hop8_sum<P>(con, j, 2 * q + 1, a.sgn);
      if (a.l1.kind == LOC_CLOVER) {
        sum[2 * q][j] = split_pack(v[0]);
        sum[2 * q + 1][j] = split_pack(v[1]);
      }
    }
    // publishes `sum`; the next tile's terms overwrite `con` only after it
    if (LOOP || a.l1.kind == LOC_CLOVER) __syncthreads();
    if (own) {
      if (a.l1.kind != LOC_NONE)
        local_comp2<R>(a.l1, Vh, p, cb, q, v, [&](unsigned b, unsigned k) { return split_unpack(sum[6 * b + k][j]); });
      if (!a.c1.is_one()) {
        const R c1 = coef<R>(a.c1);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          nrm<R>(v[e]);
          v[e] = scl<R>(c1, v[e]);
        }
      }
      if (io.X) {
        V x[2] = {load_comp<P>(io.X, N, n, 2 * q), load_comp<P>(io.X, N, n, 2 * q + 1)};
        if (a.l2.kind != LOC_NONE)
          local_comp2<R>(a.l2, Vh, p, cb, q, x, [&](unsigned b, unsigned k) { return load_comp<P>(io.X, N, n, 6 * b + k); });
        const R c2 = coef<R>(a.c2);
#pragma unroll
        for (int e = 0; e < 2; ++e) v[e] = mk<R>(fma(c2, x[e].x, v[e].x), fma(c2, x[e].y, v[e].y));
      }
      store_comp2<P>(io.out, N, n, q, v);
      if (a.red == 1) {
        const V yv[2] = {load_comp<P>(a.Y, N, n, 2 * q), load_comp<P>(a.Y, N, n, 2 * q + 1)};
        red_re += dot_comp2<R>(yv, v);
      } else if (a.red) {
        red_re += norm_comp2<R>(v);
      }
    }
    tile += gridDim.x;
  } while (LOOP && tile < ntiles);
  if (a.red) block_reduce_finalize<false>(a.ra, red_re, 0.0, 1, 1, 1, red_sm);
}

// ---------------------------------------------------------------------------
// host-side launcher
// ---------------------------------------------------------------------------
static int sm_count() {
  static const int sms = [] {
    int d = 0, c = 152;
    if (cudaGetDevice(&d) == cudaSuccess) cudaDeviceGetAttribute(&c, cudaDevAttrMultiProcessorCount, d);
    return c;
  }();
  return sms;
}

// Blocks of `kernel` resident per SM at block size bd and dynamic shared
// memory smem; cached per (kernel, bd, smem).  Also raises the kernel's
// dynamic shared-memory limit to the largest smem requested so far (the limit
// only grows, so every cached configuration stays launchable).
int resident_blocks(const void* kernel, int bd, size_t smem) {
  static std::mutex mu;
  static std::map<std::tuple<const void*, int, size_t>, int> cache;
  static std::map<const void*, size_t> limit;
  const auto key = std::make_tuple(kernel, bd, smem);
  std::lock_guard<std::mutex> lock(mu);
  auto it = cache.find(key);
  if (it != cache.end()) return it->second;
  // (raised for every size above the current limit: a kernel's static shared
  // memory counts against the same 48 KB default as the dynamic request)
  if (smem > limit[kernel]) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    limit[kernel] = smem;
  }
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, bd, smem) != cudaSuccess || nb < 1) {
    cudaGetLastError();
    nb = 1;
  }
  cache[key] = nb;
  return nb;
}

// Grid of a reducing launch: one full wave of resident blocks (every block
// then loops over an equal share of the tiles, with no partial last wave),
// and no more blocks than tiles.  The [block][rhs] partials stay few.
// min_partials > 0 allows more blocks, up to min_partials / nrhs, before the
// grid is capped (for kernels whose looping variant is slower).
long long reduce_grid(long long ntiles, int nrhs, int resident, long long min_partials) {
  long long cap = (long long)sm_count() * (resident > 0 ? resident : 1);
  const long long alt = min_partials / (nrhs > 0 ? nrhs : 1);
  if (alt > cap) cap = alt;
  return ntiles < cap ? ntiles : cap;
}

int block_size_for(int N5, int cap) {
  // blockDim = S * N5 with S a power of two and blockDim <= max(cap, N5)
  int S = 1;
  while (S * 2 * N5 <= cap) S *= 2;
  return N5 > 256 ? -1 : S * N5;
}

// The largest such block size up to `cap` of which every SM gets two blocks,
// but at least one warp: a short field is spread over all SMs (an 8^4 half
// field is 8 blocks of 256 but 64 of 32).
int spread_block(long long N, int N5, int cap) {
  int bd = block_size_for(N5, cap);
  if (bd <= 0) return bd;
  while (bd / 2 >= 32 && bd / 2 % N5 == 0 && N / bd < 2 * sm_count()) bd /= 2;
  return bd;
}

int pick_bd(int requested, int N5, int deflt) {
  if (requested > 0 && requested <= 256 && requested % N5 == 0) {
    const int S = requested / N5;
    if ((S & (S - 1)) == 0) return requested;
  }
  return deflt;
}

// Default block size of dslash_kernel.  Measured on GB300, M of the
// Wilson-clover operator (us at 256 / 64 / 32 threads): FP64 32^4 2156 /
// 2050 / 2049, 24^4 779 / 694 / 693, 16^4 160 / 160 / 144 (one block per SM
// at 254 registers: a smaller block evens out the last wave and reaches the
// FP64 units of all four SM partitions); FP32 32^4 170 / 164 / 164, 24^4
// 70.0 / 65.9 / 65.9.  Double-float keeps 256 (32^4: 749 against 815 at 64),
// and so do packed right-hand sides (their neighbours share links in L1).
static int dslash_default_bd(int P, const Geo& g, int LK) {
  if (LK != LOC_CLOVER) return spread_block(g.N, g.N5, 256);  // the s-matrix tile wants many sites per block
  if (P == PDD || g.N5 > 1) return spread_block(g.N, g.N5, 256);
  return P == P64 ? 32 : 64;
}

size_t dslash_smem_bytes(int P, int LK, int bd) {
  size_t rb = (P == P64 || P == PDD) ? 8 : 4;
  size_t s = smat_smem_bytes(LK, bd, rb) + 2 * (size_t)bd * 8;
  if (P == PDD) s = 16 * (size_t)dd_acc_offset16(LK, bd) + 12 * 16 * (size_t)bd;  // + accumulators
  return s;
}

// The double-float kernel's looping variant needs more registers (spills):
// its reducing launches keep one tile per block up to 4096 blocks.
static long long dslash_min_partials(int P) { return P == PDD ? 4096 : 0; }

template <int P, int LS, int LK, bool LOOP>
static cudaError_t launch_tl(const DslashArgs& a, cudaStream_t st) {
  const int bd = pick_bd(a.bd, a.g.N5, dslash_default_bd(P, a.g, LK));
  if (bd <= 0) return cudaErrorInvalidValue;
  const long long ntiles = (a.g.N + bd - 1) / bd;
  const size_t sm = dslash_smem_bytes(P, LK, bd);
  auto k = dslash_kernel<P, LS, LK, LOOP>;
  if constexpr (P == PDD && LK != LOC_SMAT && !LOOP) {
    if (!a.both) k = dslash_kernel<P, LS, LK, false, false>;
  }
  const int res = resident_blocks((const void*)k, bd, sm);
  const long long nb = a.red ? reduce_grid(ntiles, a.g.nrhs, res, dslash_min_partials(P)) : ntiles;
  launch_pdl(k, dim3((unsigned)nb, a.both ? 2 : 1), bd, sm, st, a);
  return cudaGetLastError();
}

// hop5: the epilogue's shared memory first, then the links and indices
// Order of the hop5 tiles for tiles of S 4D sites.  The brick is
// min(S, 4) sites in x0/2 by the rest in x1 where those divide the lattice,
// else S consecutive sites.  The slab depth T (x2 planes) is the largest
// divisor of L2 below L2 (a multiple of the brick's x2 extent) whose three x3
// steps (T planes each; input, output and X term) stay within 64 MB of L2;
// no slabs when the whole field fits in 64 MB.  GBF_HOP5_SLAB=<T> forces T
// (0: none); GBF_HOP5_BRICK=<b0,b1,b2,b3> forces the brick (0: consecutive
// sites).
static Hop5Order hop5_order(const DslashArgs& a, int S) {
  static const int forced_slab = [] {
    const char* e = std::getenv("GBF_HOP5_SLAB");
    return e ? std::atoi(e) : -1;
  }();
  static const std::array<int, 4> forced_brick = [] {
    std::array<int, 4> b{-1, -1, -1, -1};
    const char* e = std::getenv("GBF_HOP5_BRICK");
    if (e) {
      if (std::sscanf(e, "%d,%d,%d,%d", &b[0], &b[1], &b[2], &b[3]) != 4) b = {0, 0, 0, 0};
    }
    return b;
  }();
  const Geo& g = a.g;
  Hop5Order o{-1, 0, 0, 0, 0, FastDiv(), FastDiv(), FastDiv()};
  int br[4] = {S < 4 ? S : 4, S < 4 ? 1 : S / 4, 1, 1};
  if (forced_brick[0] >= 0) {
    for (int i = 0; i < 4; ++i) br[i] = forced_brick[i];
  }
  const int ext[4] = {g.Lh0, g.L[1], g.L[2], g.L[3]};
  bool brick = br[0] > 0 && (long long)br[0] * br[1] * br[2] * br[3] == S;
  for (int i = 0; i < 4 && brick; ++i) brick = br[i] > 0 && (br[i] & (br[i] - 1)) == 0 && ext[i] % br[i] == 0;
  const long long P = (long long)g.Lh0 * g.L[1];
  if (!brick && P % S) return o;
  const int bz = brick ? br[2] : 1;
  const double step = (double)P * g.N5 * 96.0 * (a.X ? 3 : 2);
  int T = 0;
  if (forced_slab >= 0) {
    T = (forced_slab > 0 && forced_slab < g.L[2] && g.L[2] % forced_slab == 0 && forced_slab % bz == 0) ? forced_slab : 0;
  } else if ((double)g.L[2] * g.L[3] * step > 64e6) {
    for (int t = bz; t < g.L[2]; t += bz)
      if (g.L[2] % t == 0 && 3.0 * t * step <= 64e6) T = t;
  }
  if (brick) {
    int l[4];
    for (int i = 0; i < 4; ++i) {
      l[i] = 0;
      while ((1 << l[i]) < br[i]) ++l[i];
    }
    const int slab = T ? T : g.L[2];
    o = Hop5Order{l[0], l[1], l[2], l[3], slab, FastDiv((unsigned)g.Lh0 >> l[0]), FastDiv((unsigned)g.L[1] >> l[1]), FastDiv((unsigned)slab >> l[2])};
  } else {
    o.slabT = T;
  }
  return o;
}

template <int P, int LK, bool LOOP>
static cudaError_t launch_hop5_tl(const DslashArgs& a, int bd, cudaStream_t st) {
  const int S = bd / a.g.N5;
  int log2S = 0;
  while ((1 << log2S) < S) ++log2S;
  const size_t epi = smat_smem_bytes(LK, bd, 4) + (a.red ? 2 * (size_t)bd * 8 : 0);
  const unsigned off16 = (unsigned)((epi + 15) / 16);
  const size_t sm = 16 * ((size_t)off16 + (size_t)S * kRecordWords);
  const long long ntiles = ((long long)a.g.Vh + S - 1) / S;
  auto k = hop5_kernel<P, LK, LOOP>;
  const int res = resident_blocks((const void*)k, bd, sm);
  const long long nb = a.red ? reduce_grid(ntiles, a.g.nrhs, res) : ntiles;
  if constexpr (!LOOP && LK != LOC_NONE) {
    if (a.red && nb < ntiles) return launch_hop5_tl<P, LK, true>(a, bd, st);
  }
  launch_pdl(k, dim3((unsigned)nb, a.both ? 2 : 1), bd, sm, st, a, off16, log2S, hop5_order(a, S));
  return cudaGetLastError();
}
template <int P, int LK>
static cudaError_t launch_hop5(const DslashArgs& a, cudaStream_t st) {
  // about 96 threads: blocks of 192 or 256 leave more of an SM's threads
  // waiting at the same barrier (Ls 12 normal operator 988 us, 1018 at 192).  A
  // looping block with dense s-matrices loads them for every tile and wants
  // more sites in it (zmobius 16^4 Ls 10 x 4, reducing hop 184 us at 80, 154 at 160)
  const int bd = pick_bd(a.bd, a.g.N5, spread_block(a.g.N, a.g.N5, LK == LOC_SMAT && a.red ? 192 : 96));
  return bd > 0 ? launch_hop5_tl<P, LK, false>(a, bd, st) : cudaErrorInvalidValue;
}

// 4D sites per block of hop5p_kernel: a requested block size (a multiple of
// N5) gives its number of sites; by default the one with the most threads
// resident per SM (16 warps of 128 registers: 36 inner sites run best in
// blocks of 144 threads, 405 us, not in 72, 431 us, which fill 2 1/4 warps)
static int hop5p_sites(const DslashArgs& a) {
  const int N5 = a.g.N5, H = (N5 + 1) / 2;
  int S = 1;
  if (a.bd > 0 && a.bd % N5 == 0 && ((a.bd / N5) & (a.bd / N5 - 1)) == 0) {
    S = a.bd / N5;
  } else {
    int best = 0;
    for (int c = 1; c * H <= 256; c *= 2) {
      const int threads = 16 / ((c * H + 31) / 32) * c * H;
      if (threads > best || (threads == best && c * H <= 64)) {
        best = threads;
        S = c;
      }
    }
  }
  while (S * H < a.g.nrhs) S *= 2;  // the reduction gives every right-hand side a thread
  return S;
}
// hop5p: two inner sites per thread, S 4D sites per block
template <int P, int LK, int MODE, bool EVEN>
static cudaError_t launch_hop5p_tl(const DslashArgs& a, int S, cudaStream_t st) {
  int log2S = 0;
  while ((1 << log2S) < S) ++log2S;
  const int H = (a.g.N5 + 1) / 2, bd = S * H;
  const size_t epi = smat_smem_bytes(LK, S * a.g.N5, 4) + (a.red ? ((size_t)S * a.g.N5 + 64) * 8 : 0);
  const unsigned off16 = (unsigned)((epi + 15) / 16);
  const size_t sm = 16 * ((size_t)off16 + (size_t)S * kRecordWords);
  const long long ntiles = ((long long)a.g.Vh + S - 1) / S;
  auto k = hop5p_kernel<P, LK, MODE, EVEN>;
  const int res = resident_blocks((const void*)k, bd, sm);
  const long long nb = a.red ? reduce_grid(ntiles, a.g.nrhs, res) : ntiles;
  if constexpr (MODE == 0) {
    if (a.red && nb < ntiles) return launch_hop5p_tl<P, LK, 1, EVEN>(a, S, st);
  }
  launch_pdl(k, dim3((unsigned)nb, a.both ? 2 : 1), bd, sm, st, a, off16, log2S, FastDiv((unsigned)H), hop5_order(a, S));
  return cudaGetLastError();
}
template <int P, int LK>
static cudaError_t launch_hop5p(const DslashArgs& a, cudaStream_t st) {
  const int N5 = a.g.N5, S = hop5p_sites(a);
  const size_t al = (size_t)a.in | (size_t)a.out | (size_t)a.X | (a.red == 1 ? (size_t)a.Y : 0) | (a.both ? a.half : 0);
  const bool even = N5 % 2 == 0 && al % 32 == 0;
  if (a.both) return even ? launch_hop5p_tl<P, LK, 2, true>(a, S, st) : launch_hop5p_tl<P, LK, 2, false>(a, S, st);
  return even ? launch_hop5p_tl<P, LK, 0, true>(a, S, st) : launch_hop5p_tl<P, LK, 0, false>(a, S, st);
}

// the bulk-copy hop: ring (also the epilogue's region), links, indices, barriers
static size_t hop5t_links_off(int LK, int bd) {
  const size_t ring = hop5t_ring_bytes(bd), epi = dslash_smem_bytes(P32, LK, bd);
  return ((ring > epi ? ring : epi) + 15) / 16 * 16;
}
static size_t hop5t_smem(int LK, int bd, int S) { return hop5t_links_off(LK, bd) + hop5_extra_smem(S) + kRing * 8; }
template <int LK, bool LOOP>
static cudaError_t launch_hop5t_tl(const DslashArgs& a, int bd, cudaStream_t st) {
  const int S = bd / a.g.N5;
  int log2S = 0;
  while ((1 << log2S) < S) ++log2S;
  const size_t sm = hop5t_smem(LK, bd, S);
  const long long ntiles = (a.g.N + bd - 1) / bd;
  auto k = hop5t_kernel<LK, LOOP>;
  const int res = resident_blocks((const void*)k, bd, sm);
  const long long nb = a.red ? reduce_grid(ntiles, a.g.nrhs, res) : ntiles;
  launch_pdl(k, (unsigned)nb, bd, sm, st, a, log2S, (unsigned)(hop5t_links_off(LK, bd) / 16));
  return cudaGetLastError();
}
template <int LK>
static cudaError_t launch_hop5t(const DslashArgs& a, cudaStream_t st) {
  const int bd = pick_bd(a.bd, a.g.N5, block_size_for(a.g.N5, 256));
  if (bd <= 0) return cudaErrorInvalidValue;
  const int S = bd / a.g.N5;
  const long long ntiles = (a.g.N + bd - 1) / bd;
  const int res = resident_blocks((const void*)hop5t_kernel<LK, true>, bd, hop5t_smem(LK, bd, S));
  const bool loop = a.red && reduce_grid(ntiles, a.g.nrhs, res) < ntiles;
  return loop ? launch_hop5t_tl<LK, true>(a, bd, st) : launch_hop5t_tl<LK, false>(a, bd, st);
}

// the two-threads-per-site double-float hop (one rhs, per-thread epilogue)
static size_t dd2_smem(int bd) { return (size_t)kDD2Acc * 16 * bd; }
static cudaError_t launch_dd2(const DslashArgs& a, cudaStream_t st) {
  const int bd = 128;  // 32^3x16, Ls 12 1328 us, 1376 at 256
  const size_t sm = dd2_smem(bd);
  auto k = dslash_dd2_kernel;
  resident_blocks((const void*)k, bd, sm);  // raises the kernel's shared-memory limit
  const long long nb = (a.g.N + bd / 2 - 1) / (bd / 2);
  launch_pdl(k, dim3((unsigned)nb, a.both ? 2 : 1), bd, sm, st, a);
  return cudaGetLastError();
}
static bool dd2_enabled();

template <int P, int LS, bool LOOP>
static cudaError_t launch_hop8_tl(const DslashArgs& a, cudaStream_t st) {
  const long long ntiles = (a.g.N + kSplitSites - 1) / kSplitSites;
  auto k = hop8_kernel<P, LS, LOOP>;
  const long long nb = a.red ? reduce_grid(ntiles, 1, resident_blocks((const void*)k, kHop8Block, 0)) : ntiles;
  launch_pdl(k, dim3((unsigned)nb, a.both ? 2 : 1), kHop8Block, 0, st, a);
  return cudaGetLastError();
}
template <int P, int LS>
static cudaError_t launch_hop8(const DslashArgs& a, cudaStream_t st) {
  const long long ntiles = (a.g.N + kSplitSites - 1) / kSplitSites;
  const int res = resident_blocks((const void*)hop8_kernel<P, LS, true>, kHop8Block, 0);
  const bool loop = a.red && reduce_grid(ntiles, 1, res) < ntiles;
  return loop ? launch_hop8_tl<P, LS, true>(a, st) : launch_hop8_tl<P, LS, false>(a, st);
}
// out = the hop and nothing else: the kernels compiled for it have no epilogue
static bool pure_hop(const DslashArgs& a) { return a.l1.kind == LOC_NONE && a.c1.is_one() && !a.X && !a.red; }

// Where hop8_kernel takes over: up to this many sites per half field.  GPU
// times of one hop (us, one thread per site / eight): FP64 8^4 30.8 / 7.1,
// 12^4 30 / 22.9, 16^4 55.7 / 59.4 (above, its uneven summation loses on the
// FP64 pipe); FP32 8^4 4.54 / 2.42, 12^4 4.72 / 3.85, 14^4 4.82 / 5.2;
// double-float, the normal operator: 16^4 108 / 98, 24^4 479 / 468, 32^4 1268
// / 1414, its launch with a reduction 20^4 90 / 82, 22^4 109 / 114, 24^4 137 /
// 156 (one wave of looping blocks), and its pure hop 32^4 250 / 245, 16^3x32 Ls
// 12 347 / 341, 32^3x16 Ls 12 1381 / 1422 (against two threads per site).
static bool use_hop8(int P, const DslashArgs& a) {
  const bool pure = pure_hop(a);
  return a.g.nrhs == 1 && (a.g.Ls == 1 || !a.red) && a.g.N <= (P != PDD ? 12288 : pure ? 1000000 : a.red ? 100000 : 170000);
}

// a launch for both parities as one launch per parity
template <typename F>
static cudaError_t each_parity(const DslashArgs& a, F launch) {
  if (!a.both) return launch(a);
  DslashArgs b = a;
  b.both = 0;
  for (int p = 0; p < 2; ++p) {
    b.out_parity = p;
    b.in = (const char*)a.in + (1 - p) * a.half;
    b.out = (char*)a.out + p * a.half;
    if (a.X) b.X = (const char*)a.X + p * a.half;
    const cudaError_t e = launch(b);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

template <int P, int LS, int LK>
static cudaError_t launch_t(const DslashArgs& a, cudaStream_t st) {
  if constexpr (P != P16 && LK == LOC_CLOVER) {
    if (use_hop8(P, a)) return launch_hop8<P, LS>(a, st);
  }
  // the pure hop (no site-local term, no X, no reduction) of one rhs: two
  // threads per site measured faster there (12.34 -> 11.55 ms on the
  // reference's Dhop benchmark); with the clover epilogue it was slower
  // (0.328 -> 0.345 ms per launch at 32^4), so the CG launches keep one thread
  if (P == PDD && LK == LOC_CLOVER && a.g.nrhs == 1 && pure_hop(a) && dd2_enabled())
    return launch_dd2(a, st);
  const int bd = pick_bd(a.bd, a.g.N5, dslash_default_bd(P, a.g, LK));
  if (bd <= 0) return cudaErrorInvalidValue;
  const long long ntiles = (a.g.N + bd - 1) / bd;
  const int res = resident_blocks((const void*)dslash_kernel<P, LS, LK, true>, bd, dslash_smem_bytes(P, LK, bd));
  const bool loop = a.red && reduce_grid(ntiles, a.g.nrhs, res, dslash_min_partials(P)) < ntiles;
  return loop ? launch_tl<P, LS, LK, true>(a, st) : launch_tl<P, LS, LK, false>(a, st);
}

// GBF_HOP5 in the environment selects the hop of FP32/FP16 fields with an
// inner extent: unset or 1 the record hops (hop5_kernel, hop5p_kernel),
// 0 the per-thread hop, 2 the bulk-copy staged hop (hop5t_kernel, FP32, inner
// extent >= 8); the default is the fastest measured.  Without a reduction FP32
// results are bitwise equal; in FP16 hop5p_kernel applies a site's scale after
// the projection and the others before it, a rounding in FP32 apart
static bool hop5_enabled() {
  static const bool on = [] {
    const char* e = std::getenv("GBF_HOP5");
    return !(e && e[0] == '0');
  }();
  return on;
}
// GBF_DD2=0 selects the one-thread-per-site double-float hop where hop8_kernel ends
static bool dd2_enabled() {
  static const bool on = [] {
    const char* e = std::getenv("GBF_DD2");
    return !(e && e[0] == '0');
  }();
  return on;
}
static bool hop5_bulk() {
  static const bool on = [] {
    const char* e = std::getenv("GBF_HOP5");
    return e && e[0] == '2';
  }();
  return on;
}

// Fields for hop5_kernel and hop5p_kernel: 8 inner sites or more, or 4 to 7 on
// fields that fill the chip (four packed Wilson-clover sources, normal
// operator on 24^4 329 -> 294 us against dslash_kernel; seven slices on
// 12x8x10x14, 47040 sites, 29.5 and 30.1 us)
bool hop_reads_records(int P, int LS, const Geo& g) {
  return hop5_enabled() && LS == L32 && (P == P32 || P == P16) && (g.N5 >= 8 || (g.N5 >= 4 && g.N >= 100000));
}

size_t record_bytes(const Geo& g) { return (size_t)2 * g.Vh * kRecordWords * 16; }
cudaError_t launch_make_records(const Geo& g, const void* links, void* records, cudaStream_t st) {
  const dim3 grid((unsigned)((g.Vh + kRecordSites - 1) / kRecordSites), 2);
  make_records_kernel<<<grid, 8 * kRecordSites, 0, st>>>(g, (const float2*)links, (float2*)records);
  return cudaGetLastError();
}

cudaError_t launch_dslash(int P, int LS, const DslashArgs& a, cudaStream_t st) {
  const int LK = a.l1.kind == LOC_SMAT ? LOC_SMAT : (a.l1.kind == LOC_BAND || a.l2.kind == LOC_BAND) ? LOC_BAND : LOC_CLOVER;
  // the bulk-copy hop of FP32 fields when selected (GBF_HOP5=2)
  if (hop5_bulk() && a.g.N5 >= 8 && LS == L32 && P == P32) {
    return each_parity(a, [&](const DslashArgs& b) {
      return LK == LOC_SMAT ? launch_hop5t<LOC_SMAT>(b, st) : LK == LOC_BAND ? launch_hop5t<LOC_BAND>(b, st) : launch_hop5t<LOC_CLOVER>(b, st);
    });
  }
  if (a.records && hop_reads_records(P, LS, a.g)) {
    if (LK == LOC_SMAT) return P == P32 ? launch_hop5<P32, LOC_SMAT>(a, st) : launch_hop5<P16, LOC_SMAT>(a, st);
    // two inner sites per thread: FP16, or FP32 fields of 32 inner sites or more
    if (P == P16) return LK == LOC_BAND ? launch_hop5p<P16, LOC_BAND>(a, st) : launch_hop5p<P16, LOC_CLOVER>(a, st);
    if (a.g.N5 >= 32) return LK == LOC_BAND ? launch_hop5p<P32, LOC_BAND>(a, st) : launch_hop5p<P32, LOC_CLOVER>(a, st);
    if (LK == LOC_BAND) return launch_hop5<P32, LOC_BAND>(a, st);
    return pure_hop(a) ? launch_hop5<P32, LOC_NONE>(a, st) : launch_hop5<P32, LOC_CLOVER>(a, st);
  }
#define GBF_D(PP, LL)                                                     \
  if (P == PP && LS == LL) {                                             \
    if (LK == LOC_SMAT) return launch_t<PP, LL, LOC_SMAT>(a, st);        \
    if (LK == LOC_BAND) return launch_t<PP, LL, LOC_BAND>(a, st);        \
    return launch_t<PP, LL, LOC_CLOVER>(a, st);                          \
  }
  GBF_D(P64, L64)
  GBF_D(P32, L32)
  GBF_D(P32, L32R)
  GBF_D(P16, L32)
  GBF_D(P16, L32R)
  GBF_D(PDD, LDD)
#undef GBF_D
  return cudaErrorInvalidValue;
}

}  // namespace gbf
