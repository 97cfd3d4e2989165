// gbf_kernels.cuh -- device building blocks shared by the kernel files:
// site-local operators (clover, s-matrix), the deterministic block reduction
// and its last-block finalisation, and the CG scalar updates.
#pragma once
#include <type_traits>
#include "gbf_common.cuh"

namespace gbf {

// shared-memory word of one complex number (16-byte access for double and
// double-float)
template <typename R> struct SplitWord;
template <> struct SplitWord<float> { using T = float2; };
template <> struct SplitWord<double> { using T = double2; };
template <> struct SplitWord<dd> { using T = float4; };
__device__ __forceinline__ float2 split_pack(float2 v) { return v; }
__device__ __forceinline__ double2 split_pack(double2 v) { return v; }
__device__ __forceinline__ float4 split_pack(ddc v) { return make_float4(v.x.h, v.y.h, v.x.l, v.y.l); }
__device__ __forceinline__ float2 split_unpack(float2 v) { return v; }
__device__ __forceinline__ double2 split_unpack(double2 v) { return v; }
__device__ __forceinline__ ddc split_unpack(float4 q) { return mk<dd>(dd(q.x, q.z), dd(q.y, q.w)); }

// f x + y and f x for a real f and complex x, y (double-float: lane-paired,
// un-normalised as fma)
template <typename R> __device__ __forceinline__ cplx<R> cfma_s(R f, cplx<R> x, cplx<R> y) { return mk<R>(fma(f, x.x, y.x), fma(f, x.y, y.y)); }
template <> __device__ __forceinline__ ddc cfma_s<dd>(dd f, ddc x, ddc y) {
  return split_unpack(pdd_st(pdd_fma_s(f, pdd_ld(split_pack(x)), pdd_ld(split_pack(y)))));
}
template <typename R> __device__ __forceinline__ cplx<R> cmul_s(R f, cplx<R> x) { return mk<R>(f * x.x, f * x.y); }
template <> __device__ __forceinline__ ddc cmul_s<dd>(dd f, ddc x) { return split_unpack(pdd_st(pdd_mul_s(f, pdd_ld(split_pack(x))))); }

// A real coefficient in every arithmetic type, split on the host: converting
// a double argument in the kernel would use the FP64 pipe in every thread.
struct Coef {
  double d;
  float h, l;
  Coef() = default;
  __host__ __device__ constexpr Coef(double v) : d(v), h((float)v), l((float)(v - (double)(float)v)) {}
  __host__ __device__ bool is_one() const { return h == 1.f && l == 0.f; }
};
template <typename R> __device__ __forceinline__ R coef(const Coef& c);
template <> __device__ __forceinline__ float coef<float>(const Coef& c) { return c.h; }
template <> __device__ __forceinline__ double coef<double>(const Coef& c) { return c.d; }
template <> __device__ __forceinline__ dd coef<dd>(const Coef& c) { return dd(c.h, c.l); }

// A site-local operator applied in a kernel epilogue.
//   LOC_CLOVER: per 4D site two Hermitian 6x6 blocks (spins {0,1}, {2,3});
//               72 reals per site: block b = 6 diagonal reals followed by the
//               15 strictly-lower complex entries (row-major i > j).
//               Storage per parity: FP64 double2 [36][Vh], FP32 float4 [18][Vh].
//   LOC_SMAT:   one real Ls x Ls matrix per chirality acting on the s index,
//               the same at every 4D site; [2][Ls][Ls] in the arithmetic type.
//   LOC_BAND:   an s-matrix that is a polynomial in the fifth-dimension hop K
//               of constant real Cayley coefficients, applied in O(Ls).  With
//               prev(s) = s - dir[chirality] and, where that leaves [0, Ls),
//               the other end times wall (K_{s,prev} = 1 or wall; g2w = g2 wall):
//                 inv = 0:  y_s = g1 x_s + g2 x_prev
//                 inv = 1:  z_s = x_s + rho z_prev,  y_s = g1 x_s + g2 z_prev,
//               z before the first slice being cs[chirality] times
//               sum_j rho^j x_{last - j} (cs = wall / (1 - wall rho^Ls) closes
//               the cycle; terms beyond nsum are below the precision's ulp).
//   LOC_SCALAR: multiplication by a real constant.
//   LOC_TWIST:  multiplication by a complex constant per chirality, z[0] + i z[1]
//               on spins 0, 1 and z[2] + i z[3] on spins 2, 3 (twisted mass
//               a + i mu g5, its inverse and adjoints).
struct LocalOp {
  int kind;
  const void* clov[2];  // per parity
  const void* smat;
  int cplx;             // LOC_SMAT: complex matrices ([2][Ls][Ls] (re, im) pairs; zmobius)
  Coef scalar;
  Coef z[4];
  // LOC_BAND
  int inv, nsum, dir[2];
  Coef g1, g2, rho, g2w[2], cs[2];  // g2w = g2 wall
};

template <typename R> struct CloverLoad;
template <> struct CloverLoad<double> {
  static __device__ __forceinline__ void block(const void* base, int Vh, int cb, int b, double (&c)[36]) {
    const double2* p = reinterpret_cast<const double2*>(base) + ((unsigned)cb + 18u * (unsigned)b * (unsigned)Vh);
#pragma unroll
    for (int k = 0; k < 18; ++k) {
      double2 q = ldg(p + (unsigned)k * (unsigned)Vh);
      c[2 * k] = q.x;
      c[2 * k + 1] = q.y;
    }
  }
};
template <> struct CloverLoad<float> {
  static __device__ __forceinline__ void block(const void* base, int Vh, int cb, int b, float (&c)[36]) {
    const float4* p = reinterpret_cast<const float4*>(base) + ((unsigned)cb + 9u * (unsigned)b * (unsigned)Vh);
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      float4 q = ldg(p + (unsigned)k * (unsigned)Vh);
      c[4 * k] = q.x; c[4 * k + 1] = q.y; c[4 * k + 2] = q.z; c[4 * k + 3] = q.w;
    }
  }
};
// off-diagonal index of (i, j), i > j
__host__ __device__ constexpr int tri(int i, int j) { return i * (i - 1) / 2 + j; }

template <typename R>
__device__ __forceinline__ void clover_apply(const void* base, int Vh, int cb, cplx<R> (&v)[12]) {
#pragma unroll
  for (int b = 0; b < 2; ++b) {
    R c[36];
    CloverLoad<R>::block(base, Vh, cb, b, c);
    cplx<R> o[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      cplx<R> acc = scl<R>(c[i], v[6 * b + i]);
#pragma unroll
      for (int j = 0; j < 6; ++j) {
        if (j < i) {
          const int t = tri(i, j);
          acc = cmadd<R>(acc, mk<R>(c[6 + 2 * t], c[6 + 2 * t + 1]), v[6 * b + j]);
        } else if (j > i) {
          const int t = tri(j, i);
          acc = cmaddc<R>(acc, mk<R>(c[6 + 2 * t], c[6 + 2 * t + 1]), v[6 * b + j]);
        }
      }
      o[i] = acc;
    }
#pragma unroll
    for (int i = 0; i < 6; ++i) v[6 * b + i] = o[i];
  }
}

// Double-float clover for site-local kernels: all loads of a block issued
// together, the two blocks in a rolled loop (the block is selected into w and
// written back by predicated moves) to keep the code in the instruction cache.
template <>
__device__ __forceinline__ void clover_apply<dd>(const void* base, int Vh, int cb, ddc (&v)[12]) {
  const float4* p0 = reinterpret_cast<const float4*>(base) + cb;
#pragma unroll 1
  for (int b = 0; b < 2; ++b) {
    const float4* p = p0 + 18u * (unsigned)b * (unsigned)Vh;
    float4 q[18];
#pragma unroll
    for (int k = 0; k < 18; ++k) q[k] = ldg(p + (unsigned)k * (unsigned)Vh);
    ddc w[6], o[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) w[i] = b ? v[6 + i] : v[i];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      o[2 * k] = scl<dd>(dd(q[k].x, q[k].z), w[2 * k]);
      o[2 * k + 1] = scl<dd>(dd(q[k].y, q[k].w), w[2 * k + 1]);
    }
#pragma unroll
    for (int i = 1; i < 6; ++i)
#pragma unroll
      for (int j = 0; j < i; ++j) {
        const float4 e = q[3 + tri(i, j)];
        const ddc cij = mk<dd>(dd(e.x, e.z), dd(e.y, e.w));
        o[i] = cmadd<dd>(o[i], cij, w[j]);
        o[j] = cmaddc<dd>(o[j], cij, w[i]);
      }
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      if (b) v[6 + i] = o[i];
      else v[i] = o[i];
    }
  }
}

// Double-float clover for the register-capped hopping kernel: entry by entry
// (each off-diagonal entry is loaded right before its two uses, row i and,
// conjugated, row j), so that no more than one entry is live.
__device__ __forceinline__ void clover_apply_dd_lowreg(const void* base, int Vh, int cb, ddc (&v)[12]) {
  const float4* p0 = reinterpret_cast<const float4*>(base) + cb;
#pragma unroll
  for (int b = 0; b < 2; ++b) {
    const float4* p = p0 + 18u * (unsigned)b * (unsigned)Vh;
    ddc* w = v + 6 * b;
    ddc o[6];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float4 q = ldg(p + (unsigned)k * (unsigned)Vh);
      o[2 * k] = scl<dd>(dd(q.x, q.z), w[2 * k]);
      o[2 * k + 1] = scl<dd>(dd(q.y, q.w), w[2 * k + 1]);
    }
#pragma unroll
    for (int i = 1; i < 6; ++i)
#pragma unroll
      for (int j = 0; j < i; ++j) {
        const float4 q = ldg(p + (unsigned)(3 + tri(i, j)) * (unsigned)Vh);
        const ddc cij = mk<dd>(dd(q.x, q.z), dd(q.y, q.w));
        o[i] = cmadd<dd>(o[i], cij, w[j]);
        o[j] = cmaddc<dd>(o[j], cij, w[i]);
      }
#pragma unroll
    for (int i = 0; i < 6; ++i) w[i] = o[i];
  }
}

// Per-thread local op (everything except LOC_SMAT, which needs the block).
template <typename R>
__device__ __forceinline__ void local_apply_thread(const LocalOp& l, int Vh, int parity, int cb, cplx<R> (&v)[12]) {
  if (l.kind == LOC_CLOVER) {
    clover_apply<R>(l.clov[parity], Vh, cb, v);
  } else if (l.kind == LOC_TWIST) {
    const cplx<R> z0 = mk<R>(coef<R>(l.z[0]), coef<R>(l.z[1])), z1 = mk<R>(coef<R>(l.z[2]), coef<R>(l.z[3]));
#pragma unroll
    for (int k = 0; k < 12; ++k) {
      nrm<R>(v[k]);
      v[k] = cmul<R>(k < 6 ? z0 : z1, v[k]);
    }
  } else if (l.kind == LOC_SCALAR) {
    const R s = coef<R>(l.scalar);
#pragma unroll
    for (int k = 0; k < 12; ++k) {
      nrm<R>(v[k]);
      v[k] = scl<R>(s, v[k]);
    }
  }
}

// Shared-memory words reserved for the s-matrices of one block: two
// chiralities of Ls x Ls complex entries at the largest Ls.
constexpr int kSmatWords = 4 * kMaxLs * kMaxLs;

// Bytes of the s-matrix part of a kernel's dynamic shared memory (arithmetic
// type of rb bytes): the tile, and for the dense form the matrices.
__host__ __device__ constexpr size_t smat_smem_bytes(int LK, int bd, size_t rb) {
  return LK == LOC_SMAT ? (24 * (size_t)bd + kSmatWords) * rb + 8
       : LK == LOC_BAND ? ((size_t)(12 * ((bd + 14) / 16 * 16 + 1)) * 2 * rb + 15) / 16 * 16
                        : 0;
}

// s-matrix op through shared memory.  Threads of one block hold complete
// s-columns (blockDim is a multiple of N5, i5 = rhs*Ls + s fastest).
// tile: 24*blockDim reals, one contiguous spinor per thread so the s-column
// is read back with 16-byte loads (the threads of one column read the same
// address: shared-memory broadcast); mat: 2*Ls*Ls reals.  All threads call.
template <typename R> struct Vec4;
template <> struct Vec4<float> { using T = float4; };
template <> struct Vec4<double> { using T = double2; };
template <> struct Vec4<dd> { using T = float4; };

template <typename R>
__device__ __forceinline__ void smat_apply_block(const R* mat_g, int Ls, R* tile, R* mat, cplx<R> (&v)[12], bool load_mat) {
  using W = typename Vec4<R>::T;
  constexpr int per = (int)(sizeof(W) / sizeof(R));  // reals per vector load
  const int t = threadIdx.x, bd = blockDim.x;
  if (load_mat)
    for (int k = t; k < 2 * Ls * Ls; k += bd) mat[k] = mat_g[k];
  R* mine = tile + 24 * t;
#pragma unroll
  for (int k = 0; k < 12; ++k) {
    mine[2 * k] = v[k].x;
    mine[2 * k + 1] = v[k].y;
  }
  __syncthreads();
  const int s = t % Ls;
  const R* col = tile + 24 * (t - s);
  const R* m0 = mat + s * Ls;
  const R* m1 = mat + Ls * Ls + s * Ls;
  R acc[24];
#pragma unroll
  for (int k = 0; k < 24; ++k) acc[k] = rzero<R>();
  for (int sp = 0; sp < Ls; ++sp) {
    const R a0 = m0[sp], a1 = m1[sp];
    const W* src = reinterpret_cast<const W*>(col + 24 * sp);
#pragma unroll
    for (int q = 0; q < 24 / per; ++q) {
      const W w = src[q];
      const R* e = reinterpret_cast<const R*>(&w);
#pragma unroll
      for (int j = 0; j < per; ++j) {
        const int k = q * per + j;
        acc[k] = fma(k < 12 ? a0 : a1, e[j], acc[k]);
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 12; ++k) v[k] = mk<R>(acc[2 * k], acc[2 * k + 1]);
  __syncthreads();
}

// LOC_BAND through shared memory, [12 components][band_stride(bd)] words.
// All threads of the block call; bd is a multiple of Ls and fLs divides by it.
// The stride is 1 mod 16 words: the threads of a scan, one per component of a
// column, then read distinct banks.
//
// inv = 1: one thread per (column, component) walks the slices, so a real
// number is written and read twice and read once more for the sum -- 5 words
// and 3 + multiply-adds per real instead of the Ls reads and Ls multiply-adds
// of the dense matrix (smat_apply_block), which on 16^3x32, Ls 12, 12 rhs kept
// the shared-memory pipe at 94 % in the site-local kernel.
__host__ __device__ constexpr int band_stride(int bd) { return (bd + 14) / 16 * 16 + 1; }

// g1 x + t.  In FP32 the low word of g1 is applied too: its rounding would be
// the same relative error in every slice and every application (G of b 1.5, c
// 0.5: -3.6e-8), which does not average out as the roundings of the sums do.
template <typename R> __device__ __forceinline__ cplx<R> band_diag(const Coef& g1, cplx<R> x, cplx<R> t) {
  if constexpr (std::is_same<R, float>::value) t = cfma_s<R>(g1.l, x, t);
  return cfma_s<R>(coef<R>(g1), x, t);
}
template <typename R>
__device__ __forceinline__ void band_scan(const LocalOp& l, int Ls, const FastDiv& fLs, int sites, int st,
                                          typename SplitWord<R>::T* tile) {
  using V = cplx<R>;
  using W = typename SplitWord<R>::T;
  const R g2 = coef<R>(l.g2), rho = coef<R>(l.rho);
  const int items = (int)fLs.div((unsigned)sites) * 12;
  for (int idx = threadIdx.x; idx < items; idx += blockDim.x) {
    const int col = idx / 12, k = idx - 12 * col;
    const int ch = k >= 6 ? 1 : 0, dir = l.dir[ch];
    W* x = tile + k * st + col * Ls;
    const int first = dir > 0 ? 0 : Ls - 1, last = Ls - 1 - first;
    auto at = [&](int s) -> W& { return x[s]; };
    V z = split_unpack(at(last - (l.nsum - 1) * dir));
    for (int j = l.nsum - 2; j >= 0; --j) {
      z = cfma_s<R>(rho, z, split_unpack(at(last - j * dir)));
      nrm<R>(z);
    }
    z = cmul_s<R>(coef<R>(l.cs[ch]), z);
    nrm<R>(z);
    for (int m = 0; m < Ls; m += 4) {
      V xv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (m + i < Ls) xv[i] = split_unpack(at(first + (m + i) * dir));
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (m + i < Ls) {
          V y = band_diag<R>(l.g1, xv[i], cmul_s<R>(g2, z));  // the smaller product is the one rounded
          z = cfma_s<R>(rho, z, xv[i]);
          nrm<R>(z);
          nrm<R>(y);
          at(first + (m + i) * dir) = split_pack(y);
        }
    }
  }
}
// inv = 0 for slice s of the column at `col`
template <typename R>
__device__ __forceinline__ void band_neighbours(const LocalOp& l, int Ls, int s, int col, int st, const typename SplitWord<R>::T* tile,
                                                cplx<R> (&v)[12]) {
  const R g2 = coef<R>(l.g2);
#pragma unroll
  for (int ch = 0; ch < 2; ++ch) {
    int sp = s - l.dir[ch];
    R f = g2;
    if (sp < 0 || sp >= Ls) {
      sp = sp < 0 ? Ls - 1 : 0;
      f = coef<R>(l.g2w[ch]);
    }
    const typename SplitWord<R>::T* x = tile + col + sp;
#pragma unroll
    for (int k = 6 * ch; k < 6 * ch + 6; ++k) v[k] = band_diag<R>(l.g1, v[k], cmul_s<R>(f, split_unpack(x[k * st])));
  }
}

// one site per thread
template <typename R, bool TAIL_SYNC>
__device__ __forceinline__ void band_apply_block(const LocalOp& l, int Ls, const FastDiv& fLs,
                                                 typename SplitWord<R>::T* tile, cplx<R> (&v)[12]) {
  const int t = threadIdx.x, bd = blockDim.x, st = band_stride(bd);
#pragma unroll
  for (int k = 0; k < 12; ++k) {
    nrm<R>(v[k]);
    tile[k * st + t] = split_pack(v[k]);
  }
  __syncthreads();
  if (l.inv) {
    band_scan<R>(l, Ls, fLs, bd, st, tile);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 12; ++k) v[k] = split_unpack(tile[k * st + t]);
  } else {
    const int col = (int)fLs.div((unsigned)t) * Ls;
    band_neighbours<R>(l, Ls, t - col, col, st, tile, v);
  }
  if (TAIL_SYNC) __syncthreads();
}

// two consecutive sites per thread (FP32), at positions t and, if two, t + 1
// of a tile of `sites`
template <bool TAIL_SYNC>
__device__ __forceinline__ void band_apply_pair(const LocalOp& l, int Ls, const FastDiv& fLs, int sites, int t, bool two, float2* tile,
                                                float2 (&v)[2][12]) {
  const int st = band_stride(sites);
#pragma unroll
  for (int k = 0; k < 12; ++k) {
    tile[k * st + t] = v[0][k];
    if (two) tile[k * st + t + 1] = v[1][k];
  }
  __syncthreads();
  if (l.inv) {
    band_scan<float>(l, Ls, fLs, sites, st, tile);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 12; ++k) {
      v[0][k] = tile[k * st + t];
      if (two) v[1][k] = tile[k * st + t + 1];
    }
  } else {
    const int c0 = (int)fLs.div((unsigned)t) * Ls, c1 = (int)fLs.div((unsigned)(t + 1)) * Ls;
    band_neighbours<float>(l, Ls, t - c0, c0, st, tile, v[0]);
    if (two) band_neighbours<float>(l, Ls, t + 1 - c1, c1, st, tile, v[1]);
  }
  if (TAIL_SYNC) __syncthreads();
}

// the six components of chirality ch at site n
template <int P> __device__ __forceinline__ void load_chiral(const void* base, unsigned N, unsigned n, int ch, cplx<typename SpinorT<P>::R> (&w)[6]) {
  if constexpr (P == P32) {
    const float4* p = reinterpret_cast<const float4*>(base) + (n + 3u * (unsigned)ch * N);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float4 q = ldg(p + (unsigned)k * N);
      w[2 * k] = make_float2(q.x, q.y);
      w[2 * k + 1] = make_float2(q.z, q.w);
    }
  } else if constexpr (P == P16) {
    const uint4* p = reinterpret_cast<const uint4*>(base);
    const float s = ldg(reinterpret_cast<const float*>(p + 3 * N) + n);
    const uint4 a = ldg(p + (n + 2u * (unsigned)ch * N));                                     // four of the six
    const uint2 b = ldg(reinterpret_cast<const uint2*>(p + (n + N)) + ch);  // the two in the middle plane
    const unsigned u[6] = {ch ? b.x : a.x, ch ? b.y : a.y, ch ? a.x : a.z, ch ? a.y : a.w, ch ? a.z : b.x, ch ? a.w : b.y};
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&u[k]));
      w[k] = make_float2(f.x * s, f.y * s);
    }
  } else {
    using W = typename SplitWord<typename SpinorT<P>::R>::T;
    const W* p = reinterpret_cast<const W*>(base) + (n + 6u * (unsigned)ch * N);
#pragma unroll
    for (int k = 0; k < 6; ++k) w[k] = split_unpack(ldg(p + (unsigned)k * N));
  }
}

// LOC_BAND with inv = 0 of a field in memory: the neighbouring slices are the
// neighbouring sites of the same column and come from L1
template <int P>
__device__ __forceinline__ void band_load(const LocalOp& l, int Ls, int s, const void* base, unsigned N, unsigned n,
                                          cplx<typename SpinorT<P>::R> (&v)[12]) {
  using R = typename SpinorT<P>::R;
  const R g2 = coef<R>(l.g2);
#pragma unroll
  for (int ch = 0; ch < 2; ++ch) {
    int d = -l.dir[ch];
    R f = g2;
    if (s + d < 0 || s + d >= Ls) {
      d = d < 0 ? Ls - 1 : 1 - Ls;
      f = coef<R>(l.g2w[ch]);
    }
    cplx<R> x[6], w[6];
    load_chiral<P>(base, N, n, ch, x);
    load_chiral<P>(base, N, (unsigned)((int)n + d), ch, w);
#pragma unroll
    for (int k = 0; k < 6; ++k) v[6 * ch + k] = band_diag<R>(l.g1, x[k], cmul_s<R>(f, w[k]));
  }
}

// The same with complex matrices ([2][Ls][Ls] entries of (re, im)), the
// per-slice complex Cayley coefficients of zmobius.
template <typename R>
__device__ __forceinline__ void smat_apply_block_c(const R* mat_g, int Ls, R* tile, R* mat, cplx<R> (&v)[12]) {
  using W = typename Vec4<R>::T;
  constexpr int per = (int)(sizeof(W) / sizeof(R));  // reals per vector load (even)
  const int t = threadIdx.x, bd = blockDim.x;
  for (int k = t; k < 4 * Ls * Ls; k += bd) mat[k] = mat_g[k];
  R* mine = tile + 24 * t;
#pragma unroll
  for (int k = 0; k < 12; ++k) {
    mine[2 * k] = v[k].x;
    mine[2 * k + 1] = v[k].y;
  }
  __syncthreads();
  const int s = t % Ls;
  const R* col = tile + 24 * (t - s);
  const R* m0 = mat + 2 * (s * Ls);
  const R* m1 = mat + 2 * (Ls * Ls + s * Ls);
  R acc[24];
#pragma unroll
  for (int k = 0; k < 24; ++k) acc[k] = rzero<R>();
  for (int sp = 0; sp < Ls; ++sp) {
    const R a0r = m0[2 * sp], a0i = m0[2 * sp + 1], a1r = m1[2 * sp], a1i = m1[2 * sp + 1];
    const W* src = reinterpret_cast<const W*>(col + 24 * sp);
#pragma unroll
    for (int q = 0; q < 24 / per; ++q) {
      const W w = src[q];
      const R* e = reinterpret_cast<const R*>(&w);
#pragma unroll
      for (int j = 0; j < per; j += 2) {
        const int k = q * per + j;
        const R ar = k < 12 ? a0r : a1r, ai = k < 12 ? a0i : a1i;
        acc[k] = fma(ar, e[j], acc[k]);
        acc[k] = fma(-ai, e[j + 1], acc[k]);
        acc[k + 1] = fma(ar, e[j + 1], acc[k + 1]);
        acc[k + 1] = fma(ai, e[j], acc[k + 1]);
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 12; ++k) v[k] = mk<R>(acc[2 * k], acc[2 * k + 1]);
  __syncthreads();
}

// Per-site Re <a, b> and |a|^2: the 12 products of one site are summed in the
// arithmetic precision R (FP32 kernels stay on the FP32 pipe; FP64 throughput
// is 1/58 of FP32 on GB300), the cross-site sums below are FP64.
template <typename R>
__device__ __forceinline__ double site_dot_re(const cplx<R> (&a_)[12], const cplx<R> (&b_)[12]) {
  R r = rzero<R>();
#pragma unroll
  for (int k = 0; k < 12; ++k) {
    cplx<R> a = a_[k], b = b_[k];
    nrm<R>(a);
    nrm<R>(b);
    r = fma(a.x, b.x, r);
    r = fma(a.y, b.y, r);
  }
  return (double)r;
}
template <typename R>
__device__ __forceinline__ double site_norm2(const cplx<R> (&a)[12]) {
  R r = 0;
#pragma unroll
  for (int k = 0; k < 12; ++k) {
    r = fma(a[k].x, a[k].x, r);
    r = fma(a[k].y, a[k].y, r);
  }
  return (double)r;
}
template <>
__device__ __forceinline__ double site_norm2<dd>(const ddc (&a_)[12]) {
  ddc a[12];
#pragma unroll
  for (int k = 0; k < 12; ++k) {
    a[k] = a_[k];
    nrm<dd>(a[k]);
  }
  dd r = rzero<dd>();
#pragma unroll
  for (int k = 0; k < 12; ++k) {
    r = fma(a[k].x, a[k].x, r);
    r = fma(a[k].y, a[k].y, r);
  }
  return (double)r;
}

// ---------------------------------------------------------------------------
// deterministic reduction: block tree over sites (stride N5), per-rhs sum of
// the s entries, per-block partials, last block sums the partials in block
// order and applies a finaliser to the CG state.
// ---------------------------------------------------------------------------
enum Fin { FIN_STORE = 0, FIN_ALPHA = 1, FIN_BETA = 2, FIN_INIT = 3 };

struct RedArgs {
  int fin;
  double2* partial;   // [gridDim][nrhs]
  unsigned* counter;  // zero on entry, restored to zero by the last block
  CGState* st;
  // pinned host copy of the state: FIN_STORE writes its results there too, and
  // then token to *seq, the launch's last write, on which the host waits (a
  // copy would cost another launch, the end of a stream a tick of 4 us)
  CGState* host;
  unsigned* seq;
  unsigned token;
  // FIN_BETA inside a conditional while graph: the last block sets the loop
  // condition to !all_done (all_done also covers maxiter and breakdown)
  unsigned long long cond;
  int use_cond;
};

// What a finaliser needs of the CG state, requested while the partials are
// being added (read one after the other they cost three L2 latencies).
struct FinState {
  double cp, rsq;
  int done, iter, maxiter;
};
__device__ __forceinline__ FinState fin_load(const RedArgs& r, int rhs) {
  FinState f{0.0, 0.0, 0, 0, 0};
  if (r.fin == FIN_STORE) return f;
  const CGState* st = r.st;
  f.cp = __ldcg(&st->cp[rhs]);
  f.rsq = __ldcg(&st->rsq[rhs]);
  f.done = __ldcg(&st->done[rhs]);
  f.iter = __ldcg(&st->iter);
  f.maxiter = __ldcg(&st->maxiter);
  return f;
}

// Applies one right-hand side's sum to the CG state; returns its done flag.
__device__ __forceinline__ int finalize(const RedArgs& r, int rhs, double re, double im, const FinState& f) {
  CGState* st = r.st;
  int done = f.done;
  switch (r.fin) {
    case FIN_STORE:
      st->last[rhs] = re;
      st->last_im[rhs] = im;
      if (r.host) {
        r.host->last[rhs] = re;
        r.host->last_im[rhs] = im;
      }
      break;
    case FIN_ALPHA: {
      st->d[rhs] = re;
      double a = 0.0;
      if (!done) {
        if (!(re > 0.0) || !isfinite(re)) {
          st->done[rhs] = 1;
          st->breakdown = 1;
        } else {
          a = f.cp / re;
        }
      }
      st->alpha[rhs] = a;
      break;
    }
    case FIN_BETA: {
      if (!done) {
        st->beta[rhs] = re / f.cp;
        st->cp[rhs] = re;
        if (re <= f.rsq) done = 1;
        if (!isfinite(re)) {
          done = 1;
          st->breakdown = 1;
        }
        if (done) st->done[rhs] = 1;
      } else {
        st->beta[rhs] = 0.0;
      }
      break;
    }
    case FIN_INIT:
      st->cp[rhs] = re;
      st->alpha[rhs] = 0.0;
      st->beta[rhs] = 0.0;
      done = (re <= f.rsq) ? 1 : 0;
      st->done[rhs] = done;
      break;
  }
  return done;
}

// After every right-hand side is finalised: the loop's flags and the counter
// for the next launch (thread 0; all: whether every right-hand side is done).
__device__ __forceinline__ void finalize_all(const RedArgs& r, int all, const FinState& f) {
  if (r.fin == FIN_BETA || r.fin == FIN_INIT) {
    if (r.fin == FIN_BETA) {
      r.st->iter = f.iter + 1;
      if (f.iter + 1 >= f.maxiter) all = 1;
    }
    r.st->all_done = all;
    if (r.fin == FIN_BETA && r.use_cond) cudaGraphSetConditional(r.cond, all ? 0u : 1u);
  }
  *r.counter = 0;
  if (r.seq) {
    __threadfence_system();
    *(volatile unsigned*)r.seq = r.token;
  }
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// Sum (a, b) (without IM only a) over the block in a fixed order: shuffle
// within warps, then the warp sums in warp 0 (the tree over 32 lanes without
// the steps that would add zeros).  Needs blockDim % 32 == 0 and at most 8
// warps; result valid in thread 0.
template <bool IM>
__device__ __forceinline__ double2 block_sum_shfl(double a, double b, double* sm) {
  const int t = threadIdx.x, lane = t & 31, w = t >> 5, nw = blockDim.x >> 5;
  a = warp_sum(a);
  if (IM) b = warp_sum(b);
  if (nw == 1) {
    __syncwarp();  // as the barrier below: the lanes' stores come before what thread 0 publishes next
    return make_double2(a, IM ? b : 0.0);
  }
  if (lane == 0) {
    sm[w] = a;
    if (IM) sm[32 + w] = b;
  }
  __syncthreads();
  if (w == 0) {
    a = lane < nw ? sm[lane] : 0.0;
    if (IM) b = lane < nw ? sm[32 + lane] : 0.0;
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      a += __shfl_down_sync(0xffffffffu, a, o);
      if (IM) b += __shfl_down_sync(0xffffffffu, b, o);
    }
  }
  return make_double2(a, IM ? b : 0.0);
}

// Thread 0 counts its block in; true in every thread of the last block, which
// then sees all partials.  Called after a barrier of the block (of the warp, if
// it is the only one): thread 0's fence then also covers what the other threads
// have stored, so that the token of a FIN_STORE launch follows its whole output.
__device__ __forceinline__ bool last_block(const RedArgs& r) {
  __shared__ int s_last;
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(r.counter, 1u) == gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  return s_last != 0;
}

// sm: 2*blockDim doubles of shared memory (at least 64).  Every thread of the
// block calls.  Without IM the imaginary part is neither summed nor stored.
template <bool IM = true>
__device__ __forceinline__ void block_reduce_finalize(const RedArgs& r, double vre, double vim, int N5, int Ls, int nrhs, double* sm) {
  const int t = threadIdx.x, bd = blockDim.x;
  const bool shfl = (bd & 31) == 0;
  if (nrhs == 1 && shfl) {
    // one right-hand side: every thread's value belongs to it
    const double2 s = block_sum_shfl<IM>(vre, vim, sm);
    if (t == 0) r.partial[blockIdx.x] = s;
  } else {
    const int S = bd / N5;  // power of two by construction
    sm[t] = vre;
    if (IM) sm[bd + t] = vim;
    __syncthreads();
    for (int k = S >> 1; k >= 1; k >>= 1) {
      if (t < k * N5) {
        sm[t] += sm[t + k * N5];
        if (IM) sm[bd + t] += sm[bd + t + k * N5];
      }
      __syncthreads();
    }
    if (t < nrhs) {
      double ar = 0, ai = 0;
      for (int s = 0; s < Ls; ++s) {
        ar += sm[t * Ls + s];
        if (IM) ai += sm[bd + t * Ls + s];
      }
      r.partial[(size_t)blockIdx.x * nrhs + t] = make_double2(ar, ai);
      __threadfence();
    }
    __syncthreads();
  }
  if (!last_block(r)) return;
  // The partials form a flat [block][rhs] array.  Thread t sums entries
  // t, t + bd, t + 2bd, ... (coalesced); since bd is a multiple of nrhs all of
  // them belong to rhs t % nrhs.  Then thread r < nrhs adds the bd/nrhs
  // thread sums of its rhs in order.  Fixed order: bitwise reproducible.
  FinState f = fin_load(r, t < nrhs ? t : 0);
  const long long total = (long long)gridDim.x * nrhs;
  double ar = 0, ai = 0;
#pragma unroll 4
  for (long long e = t; e < total; e += bd) {
    const double2 q = __ldcg(r.partial + e);
    ar += q.x;
    if (IM) ai += q.y;
  }
  if (nrhs == 1 && shfl) {
    const double2 s = block_sum_shfl<IM>(ar, ai, sm);
    if (t == 0) finalize_all(r, finalize(r, 0, s.x, s.y, f), f);
  } else {
    sm[t] = ar;
    if (IM) sm[bd + t] = ai;
    __syncthreads();
    if (t < nrhs) {
      double sr = 0, si = 0;
      for (int j = t; j < bd; j += nrhs) {
        sr += sm[j];
        if (IM) si += sm[bd + j];
      }
      finalize(r, t, sr, si, f);
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
}

}  // namespace gbf
