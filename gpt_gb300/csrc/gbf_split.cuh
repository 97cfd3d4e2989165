// gbf_split.cuh -- building blocks of the kernels that spread one 5D site
// over several threads of a block (hop8_kernel in gbf_dslash.cu, local6_kernel
// in gbf_local.cu): single spinor components in memory and in shared memory,
// and single rows of the clover term.
#pragma once
#include <type_traits>
#include "gbf_kernels.cuh"

namespace gbf {

// Sites of one block of the split kernels: 16 consecutive sites, so every
// load of one component is a run of 16 x 16 bytes.
constexpr int kSplitSites = 16;

// x with its sign flipped where mask is 0x80000000 (0: unchanged), on the
// integer pipe: a negation selected at run time would be an FP64 operation
__device__ __forceinline__ float flip_sign(float x, unsigned mask) { return __uint_as_float(__float_as_uint(x) ^ mask); }
__device__ __forceinline__ double flip_sign(double x, unsigned mask) {
  return __hiloint2double((int)((unsigned)__double2hiint(x) ^ mask), __double2loint(x));
}
__device__ __forceinline__ dd flip_sign(dd x, unsigned mask) { return dd(flip_sign(x.h, mask), flip_sign(x.l, mask)); }

// component k = 3 spin + colour of the spinor at site n (layouts: see gbf_common.cuh)
template <int P> __device__ __forceinline__ cplx<typename SpinorT<P>::R> load_comp(const void* base, unsigned N, unsigned n, unsigned k);
template <> __device__ __forceinline__ double2 load_comp<P64>(const void* base, unsigned N, unsigned n, unsigned k) {
  return ldg(reinterpret_cast<const double2*>(base) + (n + k * N));
}
template <> __device__ __forceinline__ float2 load_comp<P32>(const void* base, unsigned N, unsigned n, unsigned k) {
  return ldg(reinterpret_cast<const float2*>(reinterpret_cast<const float4*>(base) + (n + (k >> 1) * N)) + (k & 1u));
}
template <> __device__ __forceinline__ ddc load_comp<PDD>(const void* base, unsigned N, unsigned n, unsigned k) {
  return split_unpack(ldg(reinterpret_cast<const float4*>(base) + (n + k * N)));
}
// components 2q and 2q + 1
template <int P> __device__ __forceinline__ void store_comp2(void* base, unsigned N, unsigned n, unsigned q, const cplx<typename SpinorT<P>::R> (&v)[2]);
template <> __device__ __forceinline__ void store_comp2<P64>(void* base, unsigned N, unsigned n, unsigned q, const double2 (&v)[2]) {
  double2* p = reinterpret_cast<double2*>(base);
  p[n + 2u * q * N] = v[0];
  p[n + (2u * q + 1u) * N] = v[1];
}
template <> __device__ __forceinline__ void store_comp2<P32>(void* base, unsigned N, unsigned n, unsigned q, const float2 (&v)[2]) {
  reinterpret_cast<float4*>(base)[n + q * N] = make_float4(v[0].x, v[0].y, v[1].x, v[1].y);
}
template <> __device__ __forceinline__ void store_comp2<PDD>(void* base, unsigned N, unsigned n, unsigned q, const ddc (&v)[2]) {
  float4* p = reinterpret_cast<float4*>(base);
#pragma unroll
  for (unsigned e = 0; e < 2; ++e) {
    ddc w = v[e];
    nrm<dd>(w);  // memory holds normalised pairs
    p[n + (2u * q + e) * N] = split_pack(w);
  }
}

// entries of the clover storage: diagonal i and lower entry t = tri(i, j) of block b
template <typename R> struct CloverEntry;
template <> struct CloverEntry<double> {
  static __device__ __forceinline__ double diag(const void* base, unsigned Vh, unsigned cb, unsigned b, unsigned i) {
    return ldg(reinterpret_cast<const double*>(reinterpret_cast<const double2*>(base) + ((18u * b + (i >> 1)) * Vh + cb)) + (i & 1u));
  }
  static __device__ __forceinline__ double2 lower(const void* base, unsigned Vh, unsigned cb, unsigned b, unsigned t) {
    return ldg(reinterpret_cast<const double2*>(base) + ((18u * b + 3u + t) * Vh + cb));
  }
};
template <> struct CloverEntry<float> {
  static __device__ __forceinline__ float diag(const void* base, unsigned Vh, unsigned cb, unsigned b, unsigned i) {
    return ldg(reinterpret_cast<const float*>(reinterpret_cast<const float4*>(base) + ((9u * b + (i >> 2)) * Vh + cb)) + (i & 3u));
  }
  static __device__ __forceinline__ float2 lower(const void* base, unsigned Vh, unsigned cb, unsigned b, unsigned t) {
    const unsigned e = 6u + 2u * t;
    return ldg(reinterpret_cast<const float2*>(reinterpret_cast<const float4*>(base) + ((9u * b + (e >> 2)) * Vh + cb)) + ((e >> 1) & 1u));
  }
};
template <> struct CloverEntry<dd> {
  static __device__ __forceinline__ dd diag(const void* base, unsigned Vh, unsigned cb, unsigned b, unsigned i) {
    const float4 q = ldg(reinterpret_cast<const float4*>(base) + ((18u * b + (i >> 1)) * Vh + cb));
    return (i & 1u) ? dd(q.y, q.w) : dd(q.x, q.z);
  }
  static __device__ __forceinline__ ddc lower(const void* base, unsigned Vh, unsigned cb, unsigned b, unsigned t) {
    return split_unpack(ldg(reinterpret_cast<const float4*>(base) + ((18u * b + 3u + t) * Vh + cb)));
  }
};

// row i of chiral block b of the clover term applied to the six components
// get(0..5) of that chirality: the same products in the same order as
// clover_apply
template <typename R, typename Get>
__device__ __forceinline__ cplx<R> clover_row(const void* base, unsigned Vh, unsigned cb, unsigned b, unsigned i, Get get) {
  cplx<R> acc = scl<R>(CloverEntry<R>::diag(base, Vh, cb, b, i), get(i));
#pragma unroll
  for (unsigned m = 0; m < 5; ++m) {
    const bool low = m < i;
    const unsigned j = low ? m : m + 1u;
    const unsigned t = low ? (i * (i - 1u)) / 2u + j : (j * (j - 1u)) / 2u + i;
    cplx<R> c = CloverEntry<R>::lower(base, Vh, cb, b, t);
    c.y = flip_sign(c.y, low ? 0u : 0x80000000u);  // the upper triangle holds the conjugates
    acc = cmadd<R>(acc, c, get(j));
  }
  return acc;
}

// double-float: the same in lane-paired form (struct pdd)
template <typename Get>
__device__ __forceinline__ ddc clover_row_dd(const void* base, unsigned Vh, unsigned cb, unsigned b, unsigned i, Get get) {
  pdd acc = pdd_nrm(pdd_mul_s(CloverEntry<dd>::diag(base, Vh, cb, b, i), pdd_ld(split_pack(get(i)))));
#pragma unroll
  for (unsigned m = 0; m < 5; ++m) {
    const bool low = m < i;
    const unsigned j = low ? m : m + 1u;
    const unsigned t = low ? (i * (i - 1u)) / 2u + j : (j * (j - 1u)) / 2u + i;
    const ddc c = CloverEntry<dd>::lower(base, Vh, cb, b, t);
    const pdd w = pdd_ld(split_pack(get(j)));
    acc = pdd_fma_s(c.x, w, acc);
    acc = pdd_fma_s(flip_sign(c.y, low ? 0u : 0x80000000u), pdd_i(w), acc);
  }
  return split_unpack(pdd_st(acc));
}

// A site-local operator (everything except LOC_SMAT) for the thread that
// owns components 2q, 2q + 1 of one site: v holds them, get(b, j) returns
// component j of chirality b of the whole spinor (used by the clover term).
template <typename R, typename Get>
__device__ __forceinline__ void local_comp2(const LocalOp& l, unsigned Vh, int parity, unsigned cb, unsigned q, cplx<R> (&v)[2], Get get) {
  const unsigned b = q / 3u;
  if (l.kind == LOC_CLOVER) {
    const unsigned i = 2u * (q - 3u * b);
    const void* base = l.clov[parity];
    auto gb = [&](unsigned j) { return get(b, j); };
#pragma unroll
    for (unsigned e = 0; e < 2; ++e) {
      if constexpr (std::is_same<R, dd>::value) v[e] = clover_row_dd(base, Vh, cb, b, i + e, gb);
      else v[e] = clover_row<R>(base, Vh, cb, b, i + e, gb);
    }
  } else if (l.kind == LOC_TWIST) {
    const cplx<R> z = mk<R>(coef<R>(l.z[2 * b]), coef<R>(l.z[2 * b + 1]));
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      nrm<R>(v[e]);
      v[e] = cmul<R>(z, v[e]);
    }
  } else if (l.kind == LOC_SCALAR) {
    const R s = coef<R>(l.scalar);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      nrm<R>(v[e]);
      v[e] = scl<R>(s, v[e]);
    }
  }
}

// Re <a, b> or |b|^2 of the two components of this thread, summed in R as
// site_dot_re and site_norm2 do
template <typename R>
__device__ __forceinline__ double dot_comp2(const cplx<R> (&a_)[2], const cplx<R> (&b_)[2]) {
  R r = rzero<R>();
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    cplx<R> a = a_[e], b = b_[e];
    nrm<R>(a);
    nrm<R>(b);
    r = fma(a.x, b.x, r);
    r = fma(a.y, b.y, r);
  }
  return (double)r;
}
template <typename R>
__device__ __forceinline__ double norm_comp2(const cplx<R> (&a_)[2]) {
  R r = rzero<R>();
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    cplx<R> a = a_[e];
    nrm<R>(a);
    r = fma(a.x, a.x, r);
    r = fma(a.y, a.y, r);
  }
  return (double)r;
}

}  // namespace gbf
