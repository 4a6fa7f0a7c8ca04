// Split-precision grouped complex GEMM on the 5th-generation tensor cores.
//
// Same task lists as grouped_zgemm (groups = output rectangles, terms
// C += alpha * op(L) * op(R), AXPY/DIAG element terms), computed as Ozaki-style
// splits: every FP64 operand element x is written as three BF16 slices
// x ~ s0 + s1 + s2 (s0 = bf16(x), s1 = bf16(x - s0), s2 = bf16(x - s0 - s1)),
// the slice products whose weight is at least 2^-18 of the leading one --
// (0,0) (0,1) (1,0) (1,1) (0,2) (2,0) -- run as tcgen05.mma kind::f16 with FP32
// accumulators in tensor memory, and the complex product is assembled from four
// real accumulations (Cr += Ar Br - Ai Bi, Ci += Ar Bi + Ai Br).  Each slice
// product is exact in FP32, but every MMA that adds into an FP32 accumulator
// loses a biased part of its last place, so one long chain gathers an error that
// grows like K (5.5e-5 at K=4096 in one accumulator).  Hence two accumulators
// per output -- the (0,0) pair alone ("hi") and the five pairs 2^-8 smaller
// ("lo") -- restarted every SP_SEG K steps; the epilogue adds each segment into
// the output in FP64.  Element terms and the write-back (beta, partial tiles)
// are done in FP64.
//
// Operands arrive pre-sliced.  Every GEMM operand is a view -- an operator
// block (with the term's coefficient folded in, sliced once per superblock; or
// shared by all terms of that operator, the epilogue then scaling each term's
// own segments by its coefficient), a rectangle of the input vector (sliced once
// per call by slice_tiles_kernel), or a phase-1 intermediate (sliced by the
// phase-1 launch's own epilogue) --
// stored as stage tiles of BF16 planes in the canonical K-major, no-swizzle UMMA
// layout: A tiles 128 x 16 (per slice re, im: 24 KB), B tiles 16 x 64 (per slice -im, re,
// im: 18 KB, so that the real and imaginary columns of a product are one N = 128 MMA).
//
// Persistent and warp-specialised: one CTA per SM walks its own list of jobs (128 x 64
// output tiles of a group over a term range), which the host deals out longest first,
// each to the CTA with the least work.  The producer warp streams the K steps, each an A
// and a B tile brought into a shared-memory stage by two bulk asynchronous copies that
// complete on the stage's full barrier; the MMA warp issues the step's 12 MMAs into one of
// two TMEM accumulators and commits them to the stage's empty barrier (and, after a
// segment's last step, to the accumulator's full barrier); 8 epilogue warps (two per TMEM
// lane quadrant) add the other accumulator to the job's FP64 sums in registers while the
// next segment runs, and write the tile once.
//
// Bound: large superblocks by the card's power (YC4x24 m=4000 H.psi 62.6 ms in a first
// call, 70-75 ms held: 1.6 GHz at 1000 W), small ones by the epilogue's FP64 work per segment,
// which terms of a few steps have little MMA time to hide.  Measured, before: 24 MMAs of
// N = 64 issued by one lane, epilogue on whole tiles with spilled sums, descriptors read
// term by term, phase-1 results also stored in FP64:
//   m=4000 91 -> 73-75 ms (0.51 of the measured 1614 TFLOP/s bf16), YC4x12 m=1000
//   2.05 -> 1.48 ms, eight block-sparse problems 1.62 -> 1.11 ms, m=90 0.22 -> 0.13 ms
//   (L2 flushed between calls).
// Every mbarrier wait is bounded (wait_limit polls, a launch argument): on
// timeout the kernel raises a CTA abort flag and the caller's fault word, waits
// for its own MMAs (a fixed, longer bound: issued MMAs always complete), frees
// its tensor memory and returns.
#include <cuda_bf16.h>
#include <cstdint>

#include "tsc_kernels.cuh"

namespace tsc {

namespace {

constexpr int SP_TM = 128, SP_TN = 64, SP_TK = 16, SP_STAGES = 5;
constexpr int SP_PRODUCER_WARP = 0, SP_MMA_WARP = 1, SP_EPI_WARP = 4;   // warps 4..11: epilogue
constexpr int SP_EPI_WARPS = 8;   // two per TMEM lane quadrant, each draining 32 of the tile's 64 columns
constexpr int SP_THREADS = (SP_EPI_WARP + SP_EPI_WARPS) * 32;
// registers a thread: 168 at launch; the epilogue's FP64 sums need more, the others little
constexpr int SP_REGS = 80, SP_EPI_REGS = 208;
static_assert(SP_EPI_WARP * SP_REGS + SP_EPI_WARPS * SP_EPI_REGS <= (SP_EPI_WARP + SP_EPI_WARPS) * 168, "register split");
constexpr int A_PLANE = SP_TM * SP_TK * 2;                     // bytes of one BF16 plane of A
constexpr int B_PLANE = SP_TN * SP_TK * 2;                     // ... of B
constexpr int A_TILE = 6 * A_PLANE, B_TILE = 9 * B_PLANE;       // 24,576 and 18,432
constexpr int STAGE_BYTES = A_TILE + B_TILE;                   // 43,008
constexpr int SMEM_BYTES = SP_STAGES * STAGE_BYTES + 256;      // + mbarriers, TMEM slot, abort flag
static_assert(A_TILE == SPLIT_A_UNITS * SPLIT_UNIT && B_TILE == SPLIT_B_UNITS * SPLIT_UNIT,
              "stage tiles are the arena tiles");
// Two accumulators (double buffer), each [Cr hi | Ci hi | Cr lo | Ci lo]: the
// (0,0) slice pair alone in "hi", the five smaller pairs in "lo".  Both restart
// every SP_SEG K steps; the epilogue adds each segment into the output in FP64,
// so no FP32 chain in tensor memory is longer than 2 * SP_SEG MMAs (hi).
constexpr int SP_SEG = SPLIT_SEG;
constexpr uint32_t TMEM_COLS = 8 * SP_TN;                      // 512: the whole of an SM's tensor memory
// polls of the final wait for the CTA's own MMAs before tensor memory is freed
constexpr long long FIN_WAIT_LIMIT = 1ll << 24;

// instruction descriptor, kind::f16: D f32, A/B bf16, both K-major, N>>3, M>>4; N holds
// the real and the imaginary part of the tile's columns side by side
constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(2 * SP_TN >> 3) << 17) |
                           ((uint32_t)(SP_TM >> 4) << 24);

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Shared-memory matrix descriptor, K-major without swizzle: core matrices of
// 8 rows x 16 bytes stored contiguously (128 B); the two core matrices of one
// K=16 step 128 B apart (leading byte offset), 8-row groups 256 B apart
// (stride byte offset); version 1 (bits 46-47) as sm_100 requires.  The high word is
// the same for every operand; the low word is the address / 16 with the leading offset.
constexpr uint32_t DESC_HI = (256u >> 4) | (1u << 14);
__device__ __forceinline__ uint32_t desc_lo(uint32_t saddr) { return ((saddr & 0x3FFFFu) >> 4) | ((128u >> 4) << 16); }

// One lane of a converged warp.  The whole MMA warp runs the issue loop and elects a lane
// per instruction: its descriptors then live in uniform registers, where one lane inside a
// divergent branch had to move every operand of every MMA (24 MMAs took 2,470 cycles a
// step, 770 of them tensor time).
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile(
      "{\n\t"
      ".reg .pred P;\n\t"
      "elect.sync _|P, 0xFFFFFFFF;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t"
      "}\n"
      : "=r"(p));
  return p != 0;
}

__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t accumulate) {
  if (elect_one())
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        ".reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %3};\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, {%6, %6, %6, %6}, p;\n\t"
        "}\n" ::"r"(d_tmem),
        "r"(a_lo), "r"(b_lo), "r"(DESC_HI), "r"(IDESC), "r"(accumulate), "r"(0u));
}

__device__ __forceinline__ void umma_commit(uint32_t bar) {
  if (elect_one())
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}

// Bounded wait on an mbarrier phase (at most `limit` polls); gives up early
// when another role of the CTA has raised the abort flag.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, long long limit) {
  for (long long i = 0; i < limit; ++i) {
    if (abort_flag && (i & 1023) == 1023 && *abort_flag) return false;
    uint32_t done;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

__device__ __forceinline__ void fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Eight columns of this warp's 32 accumulator lanes, without waiting; the values may be
// used after tmem_wait_ld, which takes them as operands so that no use moves ahead of it.
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld(uint32_t* a, uint32_t* b) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]), "+r"(a[7]),
                 "+r"(b[0]), "+r"(b[1]), "+r"(b[2]), "+r"(b[3]), "+r"(b[4]), "+r"(b[5]), "+r"(b[6]), "+r"(b[7])
               :
               : "memory");
}

// three BF16 slices of x (through FP32, whose 24 bits the slices cover)
__device__ __forceinline__ void split3(double x, __nv_bfloat16& a, __nv_bfloat16& b, __nv_bfloat16& c) {
  const float f = (float)x;
  a = __float2bfloat16_rn(f);
  const float r1 = f - __bfloat162float(a);
  b = __float2bfloat16_rn(r1);
  const float r2 = r1 - __bfloat162float(b);
  c = __float2bfloat16_rn(r2);
}

__device__ __forceinline__ uint32_t pack2(__nv_bfloat16 lo, __nv_bfloat16 hi) {
  return (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
}

// Converts 8 consecutive-k complex values of one row (of A) or column (of B) into the
// planes of a tile, slice-major, at byte offset `off` of each: per slice re and im (A), or
// -im, re and im (B: planes 0-1 and 1-2 are then the two N = 128 operands [-Bi | Br] and
// [Br | Bi]).
template <bool B_ROLE>
__device__ __forceinline__ void store_chunk(unsigned char* planes, int off, const double2* v) {
  uint32_t w[6][4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    __nv_bfloat16 a0, b0, c0, a1, b1, c1;
    split3(v[2 * e].x, a0, b0, c0);
    split3(v[2 * e + 1].x, a1, b1, c1);
    w[0][e] = pack2(a0, a1);
    w[2][e] = pack2(b0, b1);
    w[4][e] = pack2(c0, c1);
    split3(v[2 * e].y, a0, b0, c0);
    split3(v[2 * e + 1].y, a1, b1, c1);
    w[1][e] = pack2(a0, a1);
    w[3][e] = pack2(b0, b1);
    w[5][e] = pack2(c0, c1);
  }
  constexpr int PLANE = B_ROLE ? B_PLANE : A_PLANE;
#pragma unroll
  for (int p = 0; p < 6; ++p) {
    unsigned char* d = planes + (B_ROLE ? p / 2 * 3 + 1 + p % 2 : p) * PLANE + off;
    *reinterpret_cast<uint4*>(d) = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
    if (B_ROLE && p % 2 == 1)   // the negated imaginary part (rounding is symmetric: the slices' signs flip)
      *reinterpret_cast<uint4*>(d - 2 * PLANE) = make_uint4(w[p][0] ^ 0x80008000u, w[p][1] ^ 0x80008000u,
                                                            w[p][2] ^ 0x80008000u, w[p][3] ^ 0x80008000u);
  }
}

// byte offset of the chunk (row r, k-chunk kc) inside a plane
__device__ __forceinline__ int chunk_off(int r, int kc) { return (r >> 3) * 256 + kc * 128 + (r & 7) * 16; }

// Pre-slices one stage tile of an operand view (the slice kernel below): the
// tile's chunk `chunk` -- 8 consecutive k of one row of op(X) (A role, chunks
// 0..255 of a 128 x 16 tile) or of one column (B role, chunks 0..127 of a
// 16 x 64 tile) -- times the view's coefficient, into the tile's planes.
__device__ __forceinline__ void slice_chunk(const SView& v, const double2* X, int t, int ks, int chunk,
                                            unsigned char* tile) {
  double2 x[8];
  const bool a_role = v.role == 0;
  const int r = a_role ? (chunk & 127) : (chunk & 63);
  const int kc = a_role ? (chunk >> 7) : (chunk >> 6);
  const int g = t * (a_role ? SP_TM : SP_TN) + r;   // row (A) or column (B) of op(X)
  const int kb = ks * SP_TK + kc * 8;
  const int gmax = a_role ? v.rows : v.cols, kmax = a_role ? v.cols : v.rows;
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const int k = kb + e;
    double2 y = make_double2(0.0, 0.0);
    if (g < gmax && k < kmax) {
      // A: op(X)[g][k];  B: op(X)[k][g];  op N reads X as stored, op C its conjugate transpose
      const long long i = a_role ? (v.op == OP_N ? (long long)g + (long long)k * v.ld : (long long)k + (long long)g * v.ld)
                                 : (v.op == OP_N ? (long long)k + (long long)g * v.ld : (long long)g + (long long)k * v.ld);
      y = X[i];
      if (v.op == OP_C) y.y = -y.y;
    }
    x[e] = make_double2(v.ar * y.x - v.ai * y.y, v.ar * y.y + v.ai * y.x);
  }
  if (a_role)
    store_chunk<false>(tile, chunk_off(r, kc), x);
  else
    store_chunk<true>(tile, chunk_off(r, kc), x);
}

__global__ void __launch_bounds__(256) slice_tiles_kernel(const SView* __restrict__ views,
                                                          const STile* __restrict__ tiles, const double2* in,
                                                          unsigned char* arena, long long arena_units) {
  const STile tl = tiles[blockIdx.x];
  const SView v = views[tl.view];
  const double2* X = v.from_in ? in + v.src : reinterpret_cast<const double2*>((uintptr_t)v.src * sizeof(double2));
  const int nu = v.role == 0 ? SPLIT_A_UNITS : SPLIT_B_UNITS;
  const long long unit = v.dst + (long long)(tl.t * v.nks + tl.ks) * nu;
  if (unit < 0 || unit + nu > arena_units) return;   // never outside the arena
  unsigned char* tile = arena + unit * SPLIT_UNIT;
  const int nchunk = v.role == 0 ? 256 : 128;
  if ((int)threadIdx.x < nchunk) slice_chunk(v, X, tl.t, tl.ks, threadIdx.x, tile);
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// bulk asynchronous copy global -> shared (no tensor map), completing on an mbarrier
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// Persistent, warp-specialised (roles as described at the top of the file):
// warp 0 streams the stages, warp 1 issues the MMAs into one of two TMEM
// accumulators, warps 4..11 drain the other accumulator into the outputs.
__global__ void __launch_bounds__(SP_THREADS, 1)
grouped_zgemm_split_kernel(const SJob* __restrict__ jobs, const int* __restrict__ starts,
                           const GTerm* __restrict__ terms, const __grid_constant__ Bases bases,
                           const __grid_constant__ SplitArenas arenas, int* fault, long long wait_limit,
                           int term_alpha) {
  extern __shared__ __align__(1024) unsigned char smem[];
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + SP_STAGES * STAGE_BYTES);
  uint64_t* empty = full + SP_STAGES;
  uint64_t* accf = empty + SP_STAGES;
  uint64_t* acce = accf + 2;
  uint64_t* fin = acce + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(fin + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int job0 = starts[blockIdx.x], job1 = starts[blockIdx.x + 1];   // this CTA's jobs

  if (tid == 0) {
    for (int s = 0; s < SP_STAGES; ++s) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&full[s])) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&empty[s])) : "memory");
    }
    for (int a = 0; a < 2; ++a) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&accf[a])) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&acce[a])), "r"(SP_EPI_WARPS) : "memory");
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(fin)) : "memory");
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  if (warp == SP_MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = *tmem_slot;

  auto fail = [&]() {
    *abort_flag = 1;
    atomicOr(fault, FAULT_SPLIT);
  };

  // Each role reads the descriptors of 32 terms at once, one a lane, and broadcasts: read
  // one by one, every short term waited for its own.  Warpgroup 0 (producer, MMA warp and
  // two idle warps) gives registers to the epilogue's two.
  if (warp < SP_EPI_WARP) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(SP_REGS));
    if (warp == SP_PRODUCER_WARP) {
      // ---------------------------------------------------------------- producer
      // Streams the CTA's K steps: per step, the A tile and the B tile of the term's
      // pre-sliced operand views, by two bulk copies that complete on the stage's full barrier.
      int q = 0, s = 0;
      uint32_t phase = 1;   // of the stage's empty barrier: the first round finds the stages free
      bool ok = true;
      for (int jb = job0; jb < job1 && ok; ++jb) {
        const int t0 = jobs[jb].t0, tg = jobs[jb].tg, tm = jobs[jb].tm, tn = jobs[jb].tn;
        for (int tb = t0; tb < tg && ok; tb += 32) {
          unsigned long long A = 0, B = 0;
          int nk = 0;
          bool inside = true;
          if (tb + lane < tg) {
            const GTerm& t = terms[tb + lane];
            nk = (t.K + SP_TK - 1) / SP_TK;
            // A tile (tm, kk) of the A view, B tile (tn, kk) of the B view; every tile the term
            // will copy lies inside its arena, or the CTA stops with a fault
            const long long ua = t.l_off + (long long)SPLIT_A_UNITS * tm * t.l_ld,
                            ub = t.r_off + (long long)SPLIT_B_UNITS * tn * t.r_ld;
            inside = t.l_base <= 2 && t.r_base <= 2 && ua >= 0 && ub >= 0;
            inside = inside && ua + (long long)SPLIT_A_UNITS * nk <= arenas.units[t.l_base] &&
                     ub + (long long)SPLIT_B_UNITS * nk <= arenas.units[t.r_base];
            if (inside) {
              A = (unsigned long long)(arenas.a[t.l_base] + ua * SPLIT_UNIT);
              B = (unsigned long long)(arenas.a[t.r_base] + ub * SPLIT_UNIT);
            }
          }
          if (!__all_sync(0xffffffffu, inside)) {
            ok = false;
            break;
          }
          const int cnt = min(32, tg - tb);
          for (int i = 0; i < cnt && ok; ++i) {
            const int n = __shfl_sync(0xffffffffu, nk, i);
            const unsigned char* a = (const unsigned char*)__shfl_sync(0xffffffffu, A, i);
            const unsigned char* b = (const unsigned char*)__shfl_sync(0xffffffffu, B, i);
            for (int kk = 0; kk < n; ++kk, ++q) {
              if (!__all_sync(0xffffffffu, lane != 0 || mbar_wait(smem_u32(&empty[s]), phase, abort_flag, wait_limit))) {
                ok = false;
                break;
              }
              if (elect_one()) {
                const uint32_t st0 = smem_u32(smem + s * STAGE_BYTES), fb = smem_u32(&full[s]);
                mbar_arrive_expect_tx(fb, STAGE_BYTES);
                bulk_g2s(st0, a + (long long)kk * A_TILE, A_TILE, fb);
                bulk_g2s(st0 + A_TILE, b + (long long)kk * B_TILE, B_TILE, fb);
              }
              __syncwarp();
              if (++s == SP_STAGES) {
                s = 0;
                phase ^= 1;
              }
            }
          }
        }
      }
      if (!ok) fail();
      // every copy issued here has landed before the CTA leaves, consumed or not: the last
      // fill of a stage is the largest step below q that falls to it
      for (int k = q > SP_STAGES ? q - SP_STAGES : 0; k < q; ++k)
        if (!mbar_wait(smem_u32(&full[k % SP_STAGES]), (uint32_t)((k / SP_STAGES) & 1), nullptr, FIN_WAIT_LIMIT)) fail();
      __syncwarp();
    } else if (warp == SP_MMA_WARP) {
      // ---------------------------------------------------------------- MMA issuer
      // Per step and slice pair two MMAs of 128 x 128 x 16:
      //   [Cr | Ci] += Ar [Br | Bi],  [Cr | Ci] += Ai [-Bi | Br].
      // Each reads 8 KB of shared memory in its 64 cycles; as four MMAs of N = 64 the same
      // products read 24 KB where 16 can be read (48 cycles for 32 of work each).
      int q = 0, sg = 0, s = 0;   // steps, accumulator segments (over the CTA's jobs), stage
      uint32_t phase = 0;         // of the stage's full barrier
      const uint32_t lo0 = desc_lo(smem_u32(smem));
      bool ok = true;
      for (int jb = job0; jb < job1 && ok; ++jb) {
        const int t0 = jobs[jb].t0, tg = jobs[jb].tg;
        int si = 0, nks = 0;   // step within the current segment; steps of term (ti - t0) % 32 in its lane
        for (int ti = t0; ti < tg && ok; ++ti) {
          if (((ti - t0) & 31) == 0) nks = ti + lane < tg ? (terms[ti + lane].K + SP_TK - 1) / SP_TK : 0;
          const int nk = __shfl_sync(0xffffffffu, nks, (ti - t0) & 31);
          const bool run_end = term_alpha || ti == tg - 1;
          for (int kk = 0; kk < nk; ++kk, ++q) {
            const int a = sg & 1, ua = sg >> 1;
            if (si == 0) {   // a segment starts: wait until the epilogue has drained this accumulator
              if (ua >= 1 &&
                  !__all_sync(0xffffffffu, mbar_wait(smem_u32(&acce[a]), (uint32_t)((ua - 1) & 1), abort_flag, wait_limit))) {
                ok = false;
                break;
              }
              fence_after_sync();
            }
            const uint32_t hi = tmem + a * (4 * SP_TN), lo = hi + 2 * SP_TN;
            if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&full[s]), phase, abort_flag, wait_limit))) {
              ok = false;
              break;
            }
            fence_after_sync();
            const uint32_t la = lo0 + s * (STAGE_BYTES >> 4), lb = la + (A_TILE >> 4);
  #pragma unroll
            for (int pi = 0; pi < 6; ++pi) {
              // (slice of A, slice of B) products kept
              constexpr int SA[6] = {0, 0, 1, 1, 0, 2}, SB[6] = {0, 1, 0, 1, 2, 0};
              const uint32_t ar = la + 2 * SA[pi] * (A_PLANE >> 4), b = lb + 3 * SB[pi] * (B_PLANE >> 4);
              const uint32_t d = pi == 0 ? hi : lo;
              const uint32_t first = (si == 0 && pi <= 1) ? 0u : 1u;   // first write of hi (pi 0) and lo (pi 1)
              umma_bf16(d, ar, b + (B_PLANE >> 4), first);
              umma_bf16(d, ar + (A_PLANE >> 4), b, 1u);
            }
            umma_commit(smem_u32(&empty[s]));
            if (++s == SP_STAGES) {
              s = 0;
              phase ^= 1;
            }
            ++si;
            if (si == SP_SEG || (run_end && kk == nk - 1)) {   // segment complete: to the epilogue
              umma_commit(smem_u32(&accf[a]));
              sg++;
              si = 0;
            }
          }
        }
      }
      if (!ok) fail();
      // every MMA issued here has completed before the accumulators are freed
      umma_commit(smem_u32(fin));
      if (!mbar_wait(smem_u32(fin), 0u, nullptr, FIN_WAIT_LIMIT)) fail();
      __syncwarp();
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(SP_EPI_REGS));
    // ---------------------------------------------------------------- epilogue
    constexpr int NCB = SP_TN / 16;          // 8-column chunks of one epilogue warp
    const int quad = warp & 3;               // TMEM lane quadrant this warp may read
    const int half = (warp - SP_EPI_WARP) >> 2;   // which half of the tile's 8-column chunks it takes
    int sg = 0;
    bool ok = true;
    for (int jb = job0; jb < job1 && ok; ++jb) {
      const SJob job = jobs[jb];
      const int m0 = job.tm * SP_TM, n0 = job.tn * SP_TN;
      const int row = m0 + quad * 32 + lane;
      // the tile's chunks are dealt evenly to the two warps of a quadrant, and chunks without
      // a row or column of the group are left out: a partly filled tile costs what it holds
      const int chunks = min(2 * NCB, (job.N - n0 + 7) / 8);
      const int cb0 = half ? (chunks + 1) / 2 : 0;
      const int live = m0 + quad * 32 >= job.M ? 0 : half ? chunks / 2 : (chunks + 1) / 2;
      double2* C = bases.p[job.c_base] + job.c_off;
      const long long ldc = job.c_ld;
      const bool slice_out = job.s_off >= 0;
      const int s_nks = (job.N + SP_TK - 1) / SP_TK;
      int ecur = job.t0, erem = 0;         // term_alpha: the next term, the current one's steps not yet covered
      int eks = 0;                         // steps and coefficient of term (ecur - t0) % 32, in its lane
      double ear = 1.0, eai = 0.0;
      double alr = 1.0, ali = 0.0;         // the current segment's coefficient
      // the job's segments summed in FP64 registers (this lane's row, the warp's 32 columns);
      // the output tile is then written once
      double accr[NCB][8], acci[NCB][8];
#pragma unroll
      for (int c = 0; c < NCB; ++c)
#pragma unroll
        for (int j = 0; j < 8; ++j) accr[c][j] = acci[c][j] = 0.0;
      for (int sgi = 0; sgi < job.nseg; ++sgi) {
        const int a = sg & 1, ua = sg >> 1;
        if (term_alpha) {
          if (erem == 0) {
            const int k = (ecur - job.t0) & 31;
            if (k == 0 && ecur + lane < job.tg) {
              const GTerm& t = terms[ecur + lane];
              eks = (t.K + SP_TK - 1) / SP_TK;
              ear = t.ar;
              eai = t.ai;
            }
            erem = __shfl_sync(0xffffffffu, eks, k);
            alr = __shfl_sync(0xffffffffu, ear, k);
            ali = __shfl_sync(0xffffffffu, eai, k);
            ++ecur;
          }
          erem -= erem < SP_SEG ? erem : SP_SEG;
        }
        // warp-uniform: the tensor-memory loads below need every lane
        if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&accf[a]), (uint32_t)(ua & 1), abort_flag, wait_limit))) {
          fail();
          ok = false;
          break;
        }
        fence_after_sync();
        const uint32_t lane_base = tmem + a * (4 * SP_TN) + ((uint32_t)(quad * 32) << 16);
#pragma unroll
        for (int c = 0; c < NCB; ++c) {
          if (c >= live) break;
          const uint32_t t0 = lane_base + (cb0 + c) * 8;
          uint32_t hr[8], hi[8], lr[8], li[8];
          tmem_ld8(t0, hr);
          tmem_ld8(t0 + SP_TN, hi);
          tmem_ld8(t0 + 2 * SP_TN, lr);
          tmem_ld8(t0 + 3 * SP_TN, li);
          tmem_wait_ld(hr, hi);
          tmem_wait_ld(lr, li);
          if (ali == 0.0) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              accr[c][j] += alr * ((double)__uint_as_float(hr[j]) + (double)__uint_as_float(lr[j]));
              acci[c][j] += alr * ((double)__uint_as_float(hi[j]) + (double)__uint_as_float(li[j]));
            }
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const double sr = (double)__uint_as_float(hr[j]) + (double)__uint_as_float(lr[j]);
              const double si = (double)__uint_as_float(hi[j]) + (double)__uint_as_float(li[j]);
              accr[c][j] += alr * sr - ali * si;
              acci[c][j] += alr * si + ali * sr;
            }
          }
        }
        // this warp's part of the accumulator is read out: hand it back to the MMA warp
        fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&acce[a]));
        sg++;
      }
      if (!ok) break;
      // element terms (AXPY / DIAG) in FP64, as grouped_zgemm applies them
      for (int ti = job.tg; ti < job.t1; ++ti) {
        const GTerm t = terms[ti];
        if (t.kind == TK_GEMM) continue;   // of zero depth
        const double2* R = bases.p[t.r_base] + t.r_off;
        const int rr = row - t.r0;
        if (row >= job.M || rr < 0 || rr >= t.rm) continue;
#pragma unroll
        for (int c = 0; c < NCB; ++c)
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (c >= live) break;
            const int col = n0 + (cb0 + c) * 8 + j, cc = col - t.c0;
            if (col >= job.N || cc < 0 || cc >= t.rn) continue;
            double xr, xi;
            if (t.kind == TK_AXPY) {
              const double2 x = (t.r_op == OP_N) ? R[(long long)rr + (long long)cc * t.r_ld]
                                                 : R[(long long)cc + (long long)rr * t.r_ld];
              xr = x.x;
              xi = (t.r_op == OP_C) ? -x.y : x.y;
            } else {
              if (rr != cc) continue;
              xr = 1.0;
              xi = 0.0;
            }
            accr[c][j] += t.ar * xr - t.ai * xi;
            acci[c][j] += t.ar * xi + t.ai * xr;
          }
      }
#pragma unroll
      for (int c = 0; c < NCB; ++c) {
        if (c >= live) break;
        const int c0 = (cb0 + c) * 8;
        if (row < job.M) {
          if (job.beta) {
            // all eight old values in flight before any store (the stores could alias them)
            double2 o[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const int col = n0 + c0 + j;
              o[j] = col < job.N ? C[(long long)row + (long long)col * ldc] : make_double2(0.0, 0.0);
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              accr[c][j] += o[j].x;
              acci[c][j] += o[j].y;
            }
          }
          // a phase-1 intermediate read by the next launch as an A operand goes, sliced,
          // into the A tiles of its view alone (rows >= M and columns >= N of those tiles
          // stay zero from the arena's initial clearing).  Column chunks past the view's
          // last k-step belong to no tile of this row: writing them would land in the next
          // row tile's tiles.
          if (!slice_out) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const int col = n0 + c0 + j;
              if (col < job.N) C[(long long)row + (long long)col * ldc] = make_double2(accr[c][j], acci[c][j]);
            }
          } else if ((n0 + c0) / SP_TK < s_nks) {
            double2 v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j)
              v[j] = (n0 + c0 + j) < job.N ? make_double2(accr[c][j], acci[c][j]) : make_double2(0.0, 0.0);
            const int col0 = n0 + c0;
            const long long unit = job.s_off + (long long)SPLIT_A_UNITS * ((long long)job.tm * s_nks + col0 / SP_TK);
            if (unit + SPLIT_A_UNITS <= arenas.units[ARENA_T])
              store_chunk<false>(arenas.a[ARENA_T] + unit * SPLIT_UNIT, chunk_off(row - m0, (col0 / 8) & 1), v);
          }
        }
      }
    }
  }
  fence_before_sync();
  __syncthreads();
  if (warp == SP_MMA_WARP) {
    fence_after_sync();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
}

}  // namespace

cudaError_t launch_grouped_zgemm_split(const SJob* jobs, const int* starts, int nctas, const GTerm* terms, Bases bases,
                                       SplitArenas arenas, int* fault, long long wait_limit, int term_alpha,
                                       cudaStream_t st) {
  if (nctas <= 0) return cudaSuccess;
  if (!fault || wait_limit < 0) return cudaErrorInvalidValue;
  static std::atomic<unsigned long long> attr{0};
  cudaError_t e = ensure_smem_attr(grouped_zgemm_split_kernel, SMEM_BYTES, attr);
  if (e != cudaSuccess) return e;
  grouped_zgemm_split_kernel<<<nctas, SP_THREADS, SMEM_BYTES, st>>>(jobs, starts, terms, bases, arenas, fault, wait_limit,
                                                                     term_alpha ? 1 : 0);
  return cudaGetLastError();
}

cudaError_t launch_slice_tiles(const SView* views, const STile* tiles, int ntiles, const double2* in,
                               unsigned char* arena, long long arena_units, cudaStream_t st) {
  if (ntiles <= 0) return cudaSuccess;
  slice_tiles_kernel<<<ntiles, 256, 0, st>>>(views, tiles, in, arena, arena_units);
  return cudaGetLastError();
}

}  // namespace tsc
