// gbf_launch.cuh -- argument blocks and host launchers of the device kernels.
#pragma once
#include "gbf_kernels.cuh"

namespace gbf {

// Launch with programmatic stream serialisation (see pdl_begin); every kernel
// given to it starts with pdl_begin().  Off for the calling thread while a
// pdl_off object lives (the body of a conditional graph node takes no
// programmatic edges).  It returns nothing: a launcher ends in `return
// cudaGetLastError()`, which reports a refused launch and clears it, so that
// the next launch (and the next user of the runtime) does not meet it again.
inline int& pdl_off_depth() {
  static thread_local int depth = 0;
  return depth;
}
struct pdl_off {
  pdl_off() { ++pdl_off_depth(); }
  ~pdl_off() { --pdl_off_depth(); }
};
template <typename... P, typename... A>
inline void launch_pdl(void (*kernel)(P...), dim3 grid, int block, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = dim3((unsigned)block);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  c.attrs = at;
  c.numAttrs = pdl_off_depth() ? 0 : 1;
  (void)cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}

// Even-odd hopping kernel (gbf_dslash.cu):
//   out = c1 * L1(Dhop_{p <- 1-p}(in)) + c2 * L2(X)  [+ reduction of <Y,out> or |out|^2]
// With both = 1 one launch covers both output parities (grid.y): in, out and X
// point to the even halves of full fields and `half` is the bytes of a half;
// no reduction.
struct DslashArgs {
  Geo g;
  int out_parity;
  float sgn;  // projector sign on the forward term: -1 Dhop, +1 Dhop^dag
  const void* in;
  void* out;
  const void* links;
  const void* records;  // per-site records of hop5_kernel and hop5p_kernel, or null
  LocalOp l1, l2;  // l2 may not be LOC_SMAT
  Coef c1, c2;
  const void* X;
  int red;  // 0 none, 1 <Y,out>, 2 |out|^2
  const void* Y;
  RedArgs ra;
  int check_done;
  int bd;  // block size (0: default); a multiple of N5 with a power-of-two quotient, <= 256
  int both;     // 1: both output parities
  size_t half;  // bytes of a half (both)
};
cudaError_t launch_dslash(int P, int LS, const DslashArgs& a, cudaStream_t st);
// The fields of one launch's parity: the arguments', or with both = 1 those of
// parity blockIdx.y
struct HopIO {
  const void* in;
  void* out;
  const void* X;
  int p;
};
template <bool MAY_BOTH = true> __device__ __forceinline__ HopIO hop_io(const DslashArgs& a) {
  if (!MAY_BOTH || !a.both) return HopIO{a.in, a.out, a.X, a.out_parity};
  const size_t p = blockIdx.y;
  return HopIO{(const char*)a.in + (1 - p) * a.half, (char*)a.out + p * a.half, a.X ? (const char*)a.X + p * a.half : nullptr, (int)p};
}
// block sizes S * N5, S a power of two: the largest up to cap, and the same
// reduced until every SM gets two blocks
int block_size_for(int N5, int cap);
int spread_block(long long N, int N5, int cap);
// requested block size if valid for N5, else deflt
int pick_bd(int requested, int N5, int deflt);
long long reduce_grid(long long ntiles, int nrhs, int resident, long long min_partials = 0);
int resident_blocks(const void* kernel, int bd, size_t smem);
// per-site records (links and neighbours) of both parities, from packed L32
// links, and the fields whose hop reads them
bool hop_reads_records(int P, int LS, const Geo& g);
size_t record_bytes(const Geo& g);
cudaError_t launch_make_records(const Geo& g, const void* links, void* records, cudaStream_t st);

// Site-local kernel on one parity (gbf_local.cu):
//   if (pre):  W = A + beta_rhs * W   (beta from the CG state; written back)
//   out = L(W or A)
// (both, half: as in DslashArgs; A and out move with the parity, no pre-step)
struct LocalArgs {
  Geo g;
  int both;
  size_t half;
  int parity;
  const void* A;
  void* W;       // pre-step target (p in CG), may be null
  int pre;       // 1: W = A + beta*W before the op
  LocalOp l;
  void* out;
  const CGState* st;
  int check_done;
  int bd;
};
struct LocalIO {
  const void* A;
  void* out;
  int p;
};
__device__ __forceinline__ LocalIO local_io(const LocalArgs& a) {
  if (!a.both) return LocalIO{a.A, a.out, a.parity};
  const size_t p = blockIdx.y;
  return LocalIO{(const char*)a.A + p * a.half, (char*)a.out + p * a.half, (int)p};
}
cudaError_t launch_local(int P, const LocalArgs& a, cudaStream_t st);

// CG update (gbf_local.cu): r -= alpha*mmp; x += alpha*p; reduce |r|^2 -> FIN_BETA
struct CGUpdateArgs {
  Geo g;
  void* r;
  const void* mmp;
  void* x;
  const void* p;
  RedArgs ra;
  int bd;
};
cudaError_t launch_cg_update(int P, const CGUpdateArgs& a, cudaStream_t st);

// Generic BLAS over the nhalves (0 counts as 1) halves of a field (gbf_local.cu):
//   out = a_rhs * x + b_rhs * y  (a, b per rhs, from host arrays in the args)
//   then optional reduction: 2 |out|^2, or instead of it 3 <x, y>, 4 |x|^2
struct BlasArgs {
  Geo g;
  void* out;
  const void* x;
  const void* y;
  Coef a_re[kMaxRhs], a_im[kMaxRhs], b_re[kMaxRhs];
  int red;
  int nhalves;
  size_t half;  // bytes of one half (set by the launcher)
  RedArgs ra;
};
cudaError_t launch_blas(int P, const BlasArgs& a, cudaStream_t st);

// precision conversion of the nhalves halves (N sites each) of a field
cudaError_t launch_convert(int Pout, void* out, int Pin, const void* in, long long N, int nhalves, double scale, cudaStream_t st);

// CG state initialisation from the FIN_STORE result: rsq = eps^2 * last, cp = last
cudaError_t launch_cg_init(CGState* st, int nrhs, double eps, int maxiter, cudaStream_t s);

// natural <-> internal field transfer; natural = complex128 [V][Ls][12] of one rhs
cudaError_t launch_import(int P, const Geo& g, const double2* nat, void* full, int rhs, int to_natural, cudaStream_t st);

// gauge packing: natural complex128 [4][V][9] on the device -> internal links
cudaError_t launch_pack_links(int LS, const Geo& g, const double2* U, void* links, const double* lam_mu, const double* ph,
                              unsigned* err_bits, cudaStream_t st);
// clover: natural gauge -> per parity clover and inverse (FP64 double2[36][Vh] and FP32 float4[18][Vh])
cudaError_t launch_clover(const Geo& g, const double2* U, double diag, double csw_r, double csw_t, void* c64, void* ci64,
                          void* c32, void* ci32, unsigned* err_bits, cudaStream_t st);

// set_mass of a clover operator: clover diagonal += shift (both parities and
// blocks, in place, in the operator's storage precision) and the inverse
// blocks rebuilt; err receives a large value for a singular block
cudaError_t launch_clover_shift(int prec, void* clov, void* clov_inv, int Vh, double shift, unsigned* err, cudaStream_t st);

// FP64 clover storage (double2 [2*nrows32][Vh]) -> FP32 (float4 [nrows32][Vh]);
// nrows32 is a row count (18 per parity block), not an element count
cudaError_t launch_clover_narrow(const void* src64, void* dst32, long long nrows32, int Vh, cudaStream_t st);
// the same from double-float storage (float4 (x.h, y.h, x.l, y.l) per double2)
cudaError_t launch_clover_narrow_dd(const void* srcdd, void* dst32, long long nrows32, int Vh, cudaStream_t st);
// FP64 complex array -> double-float (float4 per complex), n_complex elements
cudaError_t launch_split_dd(const void* src64, void* dst, long long n_complex, cudaStream_t st);

// block CG (gbf_block.cu): Gram matrix out[i k + j] = sum conj(A_i) . B_j of the
// k = nrhs packed vectors (partial: max_blocks x k x k entries; counter zero
// on entry, restored), and out_i = beta Y_i + sum_j X_j W[j k + i]
cudaError_t launch_gram(int P, const Geo& g, const void* A, const void* B, double2* partial, long long max_blocks,
                        unsigned* counter, double2* out, cudaStream_t st);
int gram_launches(int P, const Geo& g);
cudaError_t launch_lincomb(int P, const Geo& g, void* out, const void* Y, double beta, const void* X, const double2* W,
                           cudaStream_t st);
// multi-shift CG update over the active shifts: x_j += a_j p_j ; p_j = b_j p_j + g_j r
constexpr int kMaxShifts = 32;
struct MultiShiftArgs {
  const void* r;
  void* x[kMaxShifts];
  void* p[kMaxShifts];
  double a[kMaxShifts], b[kMaxShifts], g[kMaxShifts];
  int n;
};
cudaError_t launch_multishift(int P, const Geo& g, const MultiShiftArgs& a, cudaStream_t st);

// out1 = b1 Y1 + X1 W1 ; out2 = b2 Y2 + c out1 + X2 W2 in one pass
cudaError_t launch_lincomb2(int P, const Geo& g, void* out1, const void* Y1, double b1, const void* X1, const double2* W1,
                            void* out2, const void* Y2, double b2, double c, const void* X2, const double2* W2,
                            cudaStream_t st);

// mode representation (gbf_block.cu): inner products of a block of separate
// fields with one field, and their linear combination
constexpr int kModeBlock = 8;
struct ModeDotArgs {
  const void* v[kModeBlock];
  int n;
  const void* src;
  double2* partial;   // [gridDim][n]
  unsigned* counter;  // zero on entry, restored
  double2* out;       // out[j] = sum conj(v_j) . src
};
struct ModeAxpyArgs {
  const void* v[kModeBlock];
  double2 w[kModeBlock];
  int n;
  void* out;       // out = (accumulate ? out : 0) + sum_j w_j v_j
  int accumulate;
};
cudaError_t launch_mode_dot(int P, const Geo& g, const ModeDotArgs& a, long long max_partials, cudaStream_t st);
cudaError_t launch_mode_axpy(int P, const Geo& g, const ModeAxpyArgs& a, cudaStream_t st);

// fifth-dimension moves of the MADWF preconditioner (gbf_local.cu):
// dst_s = P- src_s + P+ src_{s + offset}, and a slice copy between fields of
// possibly different Ls (same 4D geometry and nrhs, one half)
cudaError_t launch_chiral_shift(int P, const Geo& g, const void* src, void* dst, int offset, cudaStream_t st);
cudaError_t launch_copy_slices(int P, const Geo& gd, void* dst, int d0, const Geo& gs, const void* src, int s0, int count,
                               double scale, cudaStream_t st);

}  // namespace gbf
