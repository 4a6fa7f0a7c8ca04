// Device task formats shared by the host task builders and the kernels.
#pragma once
#include <atomic>
#include <cuda_runtime.h>
#include <cstdint>

namespace tsc {

// Operand pointer = base[id] + off (complex128 elements).  Base 0 is the null
// pointer (off is then an absolute address / 16); bases 1..3 are rebound per
// launch (input vector, output vector, scratch) so one task list serves every
// Lanczos iteration.
enum BaseId : uint8_t { BASE_ABS = 0, BASE_IN = 1, BASE_OUT = 2, BASE_SCR = 3, BASE_PART = 4 };
enum TermKind : uint8_t { TK_GEMM = 0, TK_AXPY = 1, TK_DIAG = 2 };
enum Op : uint8_t { OP_N = 0, OP_C = 1 };

// One contribution to an output group:
//   GEMM:  C += alpha * op(L)[M x K] * op(R)[K x N]          (whole group)
//   AXPY:  C[r0:r0+rm, c0:c0+rn] += alpha * op(R)[rm x rn]
//   DIAG:  C[r0+i, c0+i] += alpha   for i < rm
struct GTerm {
  long long l_off, r_off;
  int l_ld, r_ld;
  int K;
  int r0, c0, rm, rn;
  double ar, ai;
  // rank: FP64 lists sum GEMM terms of a higher rank after those of a lower one
  uint8_t l_base, r_base, l_op, r_op, kind, pad0, rank, pad2;
};

// Output rectangle C (M x N, column-major, leading dimension c_ld).  After the
// launch C = sum(terms) + beta * C_old; every element of C is written.
struct GGroup {
  long long c_off;
  int c_ld, M, N;
  int t0, t1;
  uint8_t c_base, beta, pad0, pad1;
  // split-precision lists only: >= 0 when the next launch reads this group's
  // output as an A operand; the output is then written, sliced, into the A tiles
  // of that view (ARENA_T, first tile at s_off units) and nowhere else
  long long s_off = -1;
};

// One job of the FP64 kernel, a tile of a group over a range of its terms: rows [m0, mend) x
// columns [n0, nend) of the matrix at bases[c_base] + c_off (the partial buffer, ld = group
// M, for a partial sum that launch_reduce_partials adds up), GEMM terms [t0, tg), then
// element terms [tg, t1).
struct ZJob {
  long long c_off;
  int c_ld, m0, mend, n0, nend;
  int t0, tg, t1;
  uint8_t c_base, beta, pad0, pad1;
};

// Partial sums of one split group: C = sum_{p<nparts} P[p] + beta*C_old.
struct GReduce {
  int group, nparts;
  long long part_off;   // first partial; partial p at part_off + p*M*N
};

// The same for the split-precision kernel: tile (tm, tn) of an M x N group, written to the
// matrix at bases[c_base] + c_off or, with s_off >= 0, sliced to that view (GGroup); nseg =
// accumulator segments of the GEMM terms.
struct SJob {
  long long c_off, s_off;
  int c_ld, M, N, tm, tn;
  int t0, tg, t1, nseg;
  uint8_t c_base, beta, pad0, pad1;
};

struct Bases {
  double2* p[5];   // [BASE_PART]: the partial buffer
};

constexpr int GEMM_TK = 16, GEMM_THREADS = 128;

// next_job: the list's job counter in device memory, zero between launches; launches of
// one list follow one another on a stream (they share it).  tile: TILE_32x32 (4 CTAs per
// SM) or TILE_64x48 (2); bulk (large tile): operands staged by bulk copies.  A wait for
// such copies gives up after wait_limit polls, far above any that a copy takes; the kernel
// then sets FAULT_FP64 in *fault (the caller's device status word) and that CTA and the jobs
// not yet taken leave their tiles unwritten.
cudaError_t launch_grouped_zgemm(const ZJob* jobs, int njobs, const GTerm* terms, Bases bases, int* next_job,
                                 int* fault, int wait_limit, cudaStream_t st, int tile, bool bulk);
constexpr int FAULT_SPLIT = 1, FAULT_FP64 = 2;   // bits of the status word: the kernel whose wait ran out
constexpr int FP64_WAIT_LIMIT = 1 << 20;         // default poll limit of the FP64 kernel's waits
// The same for lists without GEMM terms (tiles of 32x32): AXPY and DIAG terms only.
cudaError_t launch_grouped_axpy(const ZJob* jobs, int njobs, const GTerm* terms, Bases bases, cudaStream_t st);
// ---- split-precision form: operands pre-sliced into stage tiles ----------------------
// A tile of an operand view holds the BF16 planes of op(X) in the kernel's shared-memory
// stage layout: A role 128 rows x 16 k, per slice re and im (24 KB); B role 16 k x 64
// columns, per slice -im, re and im (18 KB).  Views of fixed operators carry the term's
// coefficient and are sliced once per superblock; views of the input vector are sliced
// once per call; phase-1 intermediates are written sliced by the launch that computes them.
constexpr int SPLIT_UNIT = 6144, SPLIT_A_UNITS = 4, SPLIT_B_UNITS = 3;   // bytes; units of a tile
enum SplitArena : uint8_t { ARENA_FIXED = 0, ARENA_IN = 1, ARENA_T = 2 };
struct SView {
  long long src;       // operator: absolute address / 16; input vector: element offset
  long long dst;       // first tile, in SPLIT_UNIT from its arena's base
  double ar, ai;       // coefficient folded into the slices
  int ld, rows, cols;  // source leading dimension; op(X) is rows x cols (A: M x K, B: K x N)
  int nks;             // tiles along K
  uint8_t from_in, op, role, pad;   // role 0: A operand, 1: B operand
};
struct STile {
  int view, t, ks, pad;   // tile (t, ks) of a view: t = row tile (A) or column tile (B)
};
struct SplitArenas {
  unsigned char* a[3];
  long long units[3];   // size of each arena in SPLIT_UNIT (tile accesses are checked against it)
};
// Slices the listed tiles (one CTA each) of `views` into `arena`; `in` is the
// input vector for views with from_in set.
cudaError_t launch_slice_tiles(const SView* views, const STile* tiles, int ntiles, const double2* in,
                               unsigned char* arena, long long arena_units, cudaStream_t st);
// Split-precision form of launch_grouped_zgemm (BF16 slices on tcgen05, FP32
// accumulation in tensor memory); jobs are 128 x 64 tiles of the same groups.
// GEMM terms of its lists reference pre-sliced views: l_base / r_base = arena,
// l_off / r_off = the view's first tile (units), l_ld / r_ld = its tiles along K.
// CTA c runs jobs [starts[c], starts[c + 1]).  Every mbarrier wait of the kernel gives up
// after wait_limit polls; it then sets *fault (the caller's device status word) to 1 and
// the CTA returns with its tiles partly written.
// term_alpha = 0: the GEMM terms' coefficients are folded into their operand views (ar = 1,
// ai = 0 in the list) and accumulator segments run across terms; 1: segments break at every
// term and the epilogue multiplies each by its term's coefficient (views shared by all terms
// of an operator).
cudaError_t launch_grouped_zgemm_split(const SJob* jobs, const int* starts, int nctas, const GTerm* terms, Bases bases,
                                       SplitArenas arenas, int* fault, long long wait_limit, int term_alpha,
                                       cudaStream_t st);
// default poll limit of the split kernel's waits (far above any wait of a healthy launch)
constexpr long long SPLIT_WAIT_LIMIT = 1ll << 20;
constexpr int SPLIT_TILE_M = 128, SPLIT_TILE_N = 64;
// most K steps (of 16) of one accumulator segment of the split kernel
constexpr int SPLIT_SEG = 8;
// CTA tile codes of launch_grouped_zgemm (rows x columns of the output tile)
constexpr int TILE_32x32 = 3232, TILE_64x48 = 6448;
__host__ __device__ inline int tile_rows(int t) { return t / 100; }
__host__ __device__ inline int tile_cols(int t) { return t % 100; }
// Rows (columns) per tile of a group of n rows cut into tiles of at most `tile`: its
// 8-wide sub-tiles dealt evenly to the fewest tiles (67 rows: 40 + 27, not 64 + 3).
__host__ __device__ inline int tile_step(int n, int tile) {
  const int subs = (n + 7) / 8, tiles = (n + tile - 1) / tile;
  return tiles > 0 ? (subs + tiles - 1) / tiles * 8 : 8;
}
// How the four warps of a CTA share mtot x ntot sub-tiles, at most mi x ni each
__host__ __device__ inline void warp_grid(int mtot, int ntot, int mi, int ni, int& wm, int& wn) {
  wm = wn = 2;
  int best = ((mtot + 1) / 2) * ((ntot + 1) / 2);
  if (mtot <= mi && mtot * ((ntot + 3) / 4) < best) {
    best = mtot * ((ntot + 3) / 4);
    wm = 1;
    wn = 4;
  }
  if (ntot <= ni && ((mtot + 3) / 4) * ntot < best) {
    wm = 4;
    wn = 1;
  }
}
// Sets a kernel's dynamic shared-memory limit once per device (the attribute
// belongs to the current device's context; concurrent first calls set the same
// value).  `done` is the kernel's own bitmask of devices already set.
template <class K>
cudaError_t ensure_smem_attr(K kernel, int bytes, std::atomic<unsigned long long>& done) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = 1ull << (dev & 63);
  if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_acq_rel);
  return e;
}
// Launches whose start overlaps the end of the kernel before them on the stream: the block
// scheduling of a short kernel no longer waits for the other's last block.  A kernel launched
// so calls chain_kernels() before its first access to global memory; it returns once the
// kernel before has finished and its writes are visible, and lets the kernel after be
// scheduled in turn.  Every thread of it does so, so a kernel that has finished implies that
// all before it have.  After anything but a kernel that calls it, the launch is an ordinary one.
// The FP64 lists and their reductions are launched so: H.psi at m=40 on 12 columns 36.3 ->
// 32.2 us, m=90 41 -> 37, m=300 197 -> 195, m=1000 the same.  The split kernel (m=90 132 -> 124,
// but m=1000 1481 -> 1509 us from a cold L2) and the Lanczos vector kernels (no difference inside their graph) are not.
#ifdef __CUDACC__
__device__ __forceinline__ void chain_kernels() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <class... P, class... A>
cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, int block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
#endif
cudaError_t launch_reduce_partials(const GReduce* reds, int nred, const GGroup* groups, Bases bases,
                                   long long max_elems, cudaStream_t st);

// ---- vector kernels (Lanczos, eigen.f90 / block.f90:1092-1354) -------------------
// partial sums of Re<x_j, y> for j < nvec (x_j = X + j*ld), deterministic two-pass
cudaError_t launch_multi_dot(const double2* X, long long ld, int nvec, const double2* y, long long n,
                             double* partial, double* out, cudaStream_t st);
// <x, y> = sum conj(x) y into out[0] (real), out[1] (imaginary); partial holds
// 2 * ceil(n / 8192) doubles; deterministic two-pass
cudaError_t launch_zdot(const double2* x, const double2* y, long long n, double* partial, double* out,
                        cudaStream_t st);
cudaError_t launch_scale(double2* w, const double* norm2, long long n, int invert_sqrt, cudaStream_t st);
cudaError_t launch_combine(double2* out, const double2* X, long long ld, int nvec, const double* z,
                           long long n, cudaStream_t st);

// Canonical phase of each column of U (rows x cols, column-major): u *= conj(z)/|z|
// with z = sum_r u_r / (1 + r/10).  Eigensolvers return arbitrary phases; fixing
// them makes renormalised operators independent of the eigensolver.
cudaError_t launch_phase_fix(double2* U, int rows, int cols, cudaStream_t st);

// tridiagonal lowest eigenpair (dstev stand-in): d[0..n), e[0..n-1); writes
// res[0]=E0 and, if want_vec, z[0..n) the normalised eigenvector.
cudaError_t launch_tridiag_lowest(const double* d, const double* e, int n, int want_vec, double* res,
                                  double* z, cudaStream_t st);
// ---- one Lanczos iteration's vector work, the index read on the device -------------
// (replayable as one CUDA graph: *it = last, the 1-based Lanczos index of eigen.f90; V =
// v(1), vectors ld apart; counter: a device int, zero between launches; partial: room for
// it_blocks(n) doubles per value reduced, last + 1 of them in it_project; last <= 126)
int it_blocks(long long n);
// w = v(last+1) -= alpha_last v(last) + beta_(last-1) v(last-1); n2 = |w|^2;
// uv[j] = Re<v(j+1), w> / |w| for j < last
cudaError_t launch_it_project(double2* V, long long ld, const double* alpha, const double* beta, long long n,
                              const int* it, double* partial, int* counter, double* n2, double* uv, cudaStream_t st);
// w = w / sqrt(n2) - sum_{j<last} (uv_j / uu_j) v(j+1)  (Gram_Schmidt_process); nw2 = |w|^2
cudaError_t launch_it_orthogonalize(double2* V, long long ld, const double* n2, const double* uv, const double* uu,
                                    long long n, const int* it, double* partial, int* counter, double* nw2,
                                    cudaStream_t st);
// v(last+1) = x = w / sqrt(nw2); uu[last] = its norm squared
cudaError_t launch_it_normalize(double2* V, long long ld, const double* nw2, long long n, const int* it, double2* x,
                                double* partial, int* counter, double* uu, cudaStream_t st);
// v(last+2) = y; alpha[k] = Re<x, y>, k = last + 1; beta[k-1] = sqrt(n2); res[0] = lowest
// eigenvalue of T_k; packet = {res[0], n2, alpha[k], |z[k-1]|} (z in zbuf, if not null)
cudaError_t launch_it_alpha(double2* V, long long ld, const double2* x, const double2* y, long long n, const int* it,
                            double* partial, int* counter, const double* n2, double* alpha, double* beta, double* res,
                            double* packet, double* zbuf, cudaStream_t st);

}  // namespace tsc
