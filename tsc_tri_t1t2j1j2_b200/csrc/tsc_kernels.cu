// B200 (sm_100a) kernels of the superblock engine.
//
// grouped_zgemm: output-stationary grouped complex-FP64 GEMM.  A job is a tile (64x48 or
// 32x32) of one output group over a range of its terms; a CTA sums them in registers
// (DMMA m8n8k4.f64, 3 real MMAs per complex product by the Gauss three-multiplication
// form) and writes the tile once: no atomics on data, the result does not depend on which
// CTA takes a job.
//
// Bound: the FP64 pipe, which DMMA and every other FP64 instruction share.  Hence
// - persistent CTAs (2 per SM with the large tile) taking jobs from a counter, four warps
//   that only load and four that only multiply, so that nothing but shared-memory reads and
//   the fragments' sums stands between the DMMAs, and the chunks of one job follow those of
//   the job before without a gap;
// - a warp tile of 4 x 3 sub-tiles: 13 side instructions per 36 DMMAs (a 2 x 2 tile has 8
//   per 12; 4 x 4 does not fit the registers with the three sums);
// - three chunks of 16 of K in shared memory, by 16-byte cp.async (zero fill at the edges,
//   rows padded by two elements so that fragment reads are conflict-free) or, for large
//   lists, by bulk copies.
// Measured (8 m n k of the products executed; 32x32 tiles, 6 CTAs per SM, every thread
// loading and multiplying in turn before): YC4x24 m=4000 H.psi 339 -> 254 ms (30.0 -> 40.1
// TFLOP/s), YC4x12 m=1000 4.76 -> 3.50 ms (24.5 -> 33.3).  The three-multiplication bound
// of the 37.0 TFLOP/s pipe is 49.3.  With cp.async m=4000 took 276 ms: 22 of them the side
// instructions, 15 the loading instructions and 16 waiting for data (each taken out in turn).
//
// Vector kernels: the Lanczos recurrences of eigen.f90:64-94 and the classical
// Gram-Schmidt of block.f90:1251-1289 (it_*: every reduction ended in a fixed order by the
// last block to arrive) and a tridiagonal lowest-eigenpair solver standing in for LAPACK dstev
// (eigen.f90:99,117,141): Sturm-sequence bisection for the eigenvalue, inverse
// iteration with a pivoted tridiagonal LU for the eigenvector.
#include "tsc_kernels.cuh"

#include <cfloat>
#include <cmath>

namespace tsc {

namespace {

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool pred) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  int sz = pred ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(sz));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}
__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

constexpr int TK = GEMM_TK;
constexpr int ZSTAGES = 3;   // k chunks of 16 in shared memory: one computed, two on their way
constexpr int ZRING = 16;    // term descriptors held in shared memory
constexpr int ZAHEAD = 8;    // ... fetched this many terms ahead of the loads
constexpr int ZSLOTS = 8;    // job records in shared memory (the loaders are at most ZSTAGES jobs ahead)
static_assert(sizeof(GTerm) % 8 == 0 && sizeof(ZJob) % 8 == 0, "records are copied as 8-byte words");
constexpr int TERM_WORDS = (int)(sizeof(GTerm) / 8), JOB_WORDS = (int)(sizeof(ZJob) / 8);

struct ZMeta {   // what the multiplying warps need to know of a chunk
  double ar, ai;
  unsigned lneg;       // 0x80000000: op(L) conjugates
  uint8_t rneg, ksteps, last, slot;   // op(R) conjugates; k steps of 4; the job's last chunk; job record (ZSLOTS: end)
  uint8_t lt, rt, pad0, pad1;         // operand staged strip by strip along k ([m][k] or [n][k])
};

// Shared memory of a CTA.  Staged by cp.async an operand lies row by row of one k (TM or TN
// long, padded by two elements: no bank conflicts).  Staged by bulk copies it lies as in
// global memory: such rows, or the 16 k of one row or column (padded by one: two-way
// conflicts).
template <int TM, int TN, bool BULK>
struct ZTile {
  static constexpr int LDA = TM + 2, LDB = TN + 2, LDK = TK + 1;
  static constexpr int ELA = BULK && TM * LDK > TK * LDA ? TM * LDK : TK * LDA;
  static constexpr int ELB = BULK && TN * LDK > TK * LDB ? TN * LDK : TK * LDB;
  static constexpr int STAGE = ELA + ELB;            // complex per stage
  static constexpr int OFF_RING = ZSTAGES * STAGE * 16, OFF_JOBS = OFF_RING + (BULK ? 0 : ZRING * TERM_WORDS * 8),
                       OFF_META = OFF_JOBS + ZSLOTS * JOB_WORDS * 8, OFF_BAR = OFF_META + ZSTAGES * (int)sizeof(ZMeta),
                       OFF_NEXT = OFF_BAR + ZSTAGES * 8, OFF_GAVE_UP = OFF_NEXT + ZSLOTS * 4, SMEM = OFF_GAVE_UP + 8;
};

// Named barriers (hardware, no polling) between the loading and the multiplying warps
constexpr int BAR_FULL = 1, BAR_EMPTY = BAR_FULL + ZSTAGES, BAR_LOAD = BAR_EMPTY + ZSTAGES;
template <int N>
__device__ __forceinline__ void bar_sync(int id) {
  asm volatile("barrier.cta.sync %0, %1;" ::"r"(id), "n"(N) : "memory");
}
template <int N>
__device__ __forceinline__ void bar_arrive(int id) {
  asm volatile("barrier.cta.arrive %0, %1;" ::"r"(id), "n"(N) : "memory");
}

__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem));
}
// v with its sign flipped when mask is 0x80000000 (integer pipe: the FP64 pipe is the one that is busy)
__device__ __forceinline__ double flip_sign(double v, unsigned mask) {
  return __hiloint2double(__double2hiint(v) ^ (int)mask, __double2loint(v));
}

// One operand's tile, copied by 128 threads as strips contiguous in global memory: FAST
// elements along the operand's contiguous index, SLOW strips `ld` apart.  Element (f, q)
// goes to shared element f * FS + q * QS; every 16-byte copy is one complex element.  A
// thread takes the elements f0 + i FW, q0 + r STEP: its first address is set up once per
// term and stepped from chunk to chunk, so that a copy costs three instructions (index
// arithmetic in every copy made the loading warps issue as many instructions as the
// multiplying ones).
template <int FAST, int SLOW, int FS, int QS>
struct Strip {
  static constexpr int FW = FAST % 64 == 0 ? 64 : FAST % 32 == 0 ? 32 : 16, STEP = GEMM_THREADS / FW;
  static __device__ __forceinline__ int f0() { return (threadIdx.x & (GEMM_THREADS - 1)) % FW; }
  static __device__ __forceinline__ int q0() { return (threadIdx.x & (GEMM_THREADS - 1)) / FW; }
  // nfast, nslow: valid extents; the rest is zero-filled
  static __device__ __forceinline__ void copy(double2* dst, const double2* p, long long ld, int nfast, int nslow) {
    double2* d = dst + f0() * FS + q0() * QS;
    const long long inc = STEP * ld;
    if (nfast >= FAST && nslow >= SLOW) {
#pragma unroll
      for (int r = 0; r < SLOW / STEP; ++r) {
#pragma unroll
        for (int i = 0; i < FAST / FW; ++i) cp_async16(d + r * STEP * QS + i * FW * FS, p + i * FW, true);
        p += inc;
      }
    } else {
      const int nf = nfast - f0(), nq = nslow - q0();
#pragma unroll
      for (int r = 0; r < SLOW / STEP; ++r) {
#pragma unroll
        for (int i = 0; i < FAST / FW; ++i)   // a copy of size zero reads nothing
          cp_async16(d + r * STEP * QS + i * FW * FS, p + i * FW, r * STEP < nq && i * FW < nf);
        p += inc;
      }
    }
  }
};

// One k chunk of one warp's MT x NT sub-tiles.  Complex products by the
// three-multiplication (Gauss) form: with T1 = Ar Br, T2 = Ai Bi,
// T3 = (Ar + Ai)(Br + Bi), the product is (T1 - T2) + i (T3 - T1 - T2): three DMMAs per
// complex multiply-add instead of four.  Every FP64 instruction beside the DMMAs takes
// time from their pipe (about 4.6 cycles against a DMMA's 16), so the term's coefficient
// rides on the B fragments as a real factor when it is real, with op C's conjugation
// folded into its sign.
template <int MT, int NT, int MI, int NI, bool CPLX>
__device__ __forceinline__ void mma_chunk(double (&t1)[MI][NI][2], double (&t2)[MI][NI][2], double (&t3)[MI][NI][2],
                                          const double2* As, const double2* Bs, int sma, int ska, int snb, int skb,
                                          const ZMeta& m) {
  const double ar = m.ar, ai = CPLX ? m.ai : (m.rneg ? -m.ar : m.ar);
  const unsigned lneg = m.lneg;
  const int ksteps = m.ksteps;
  double2 an[MT], bn = Bs[0];   // fragments on their way: A of the next k step, B of the next column
#pragma unroll
  for (int mi = 0; mi < MT; ++mi) an[mi] = As[mi * sma];
#pragma unroll 1
  for (int kb = 0; kb < ksteps; ++kb) {
    double xr[MT], xi[MT], xs[MT];
#pragma unroll
    for (int mi = 0; mi < MT; ++mi) {
      xr[mi] = an[mi].x;
      xi[mi] = flip_sign(an[mi].y, lneg);
      xs[mi] = xr[mi] + xi[mi];
    }
    // in the last step this reads that step again, unused
    const int kn = kb + 1 < ksteps ? kb + 1 : kb;
#pragma unroll
    for (int mi = 0; mi < MT; ++mi) an[mi] = As[kn * ska + mi * sma];
#pragma unroll
    for (int ni = 0; ni < NT; ++ni) {
      const double2 v = bn;
      bn = ni + 1 < NT ? Bs[kb * skb + (ni + 1) * snb] : Bs[kn * skb];
      double yr, yi;
      if (CPLX) {
        const double vi = m.rneg ? -v.y : v.y;
        yr = ar * v.x - ai * vi;
        yi = ar * vi + ai * v.x;
      } else {
        yr = ar * v.x;
        yi = ai * v.y;
      }
      const double ys = yr + yi;
      // three passes: successive updates of an accumulator are far apart
#pragma unroll
      for (int mi = 0; mi < MT; ++mi) dmma(t1[mi][ni][0], t1[mi][ni][1], xr[mi], yr);
#pragma unroll
      for (int mi = 0; mi < MT; ++mi) dmma(t2[mi][ni][0], t2[mi][ni][1], xi[mi], yi);
#pragma unroll
      for (int mi = 0; mi < MT; ++mi) dmma(t3[mi][ni][0], t3[mi][ni][1], xs[mi], ys);
    }
  }
}

// Straight-line code for every count of sub-tiles a warp can hold (branching around each
// DMMA of a partly filled warp cost 10 instructions per DMMA).
template <int MT, int NT, int MI, int NI>
__device__ __forceinline__ void mma_select(double (&t1)[MI][NI][2], double (&t2)[MI][NI][2], double (&t3)[MI][NI][2],
                                           const double2* As, const double2* Bs, int sma, int ska, int snb, int skb,
                                           const ZMeta& m, int mt, int nt) {
  if constexpr (MT > 1) {
    if (mt < MT) return mma_select<MT - 1, NT, MI, NI>(t1, t2, t3, As, Bs, sma, ska, snb, skb, m, mt, nt);
  }
  if constexpr (NT > 1) {
    if (nt < NT) return mma_select<MT, NT - 1, MI, NI>(t1, t2, t3, As, Bs, sma, ska, snb, skb, m, mt, nt);
  }
  if (m.ai == 0.0)
    mma_chunk<MT, NT, MI, NI, false>(t1, t2, t3, As, Bs, sma, ska, snb, skb, m);
  else
    mma_chunk<MT, NT, MI, NI, true>(t1, t2, t3, As, Bs, sma, ska, snb, skb, m);
}

// Loading half of a CTA, by cp.async: streams the chunks of the CTA's jobs, across term and
// job boundaries, into the stages.
template <int TM, int TN>
__device__ __forceinline__ void zgemm_load(unsigned char* smem, const ZJob* jobs, int njobs, const GTerm* terms,
                                           const Bases& bases, int* next_job) {
  using Z = ZTile<TM, TN, false>;
  using AN = Strip<TM, TK, 1, Z::LDA>;
  using AC = Strip<TK, TM, Z::LDA, 1>;
  using BN = Strip<TK, TN, Z::LDB, 1>;
  using BC = Strip<TN, TK, 1, Z::LDB>;
  const int tid = threadIdx.x & (GEMM_THREADS - 1);
  double2* const stages = reinterpret_cast<double2*>(smem);
  long long* const ring = reinterpret_cast<long long*>(smem + Z::OFF_RING);
  ZJob* const slots = reinterpret_cast<ZJob*>(smem + Z::OFF_JOBS);
  ZMeta* const metas = reinterpret_cast<ZMeta*>(smem + Z::OFF_META);
  int* const nexts = reinterpret_cast<int*>(smem + Z::OFF_NEXT);
  int stage = 0, chunks = 0, seq = 0;
  // opens the stage of the next chunk: the multiplying warps are done with what it held
  auto open = [&]() {
    if (chunks >= ZSTAGES) bar_sync<2 * GEMM_THREADS>(BAR_EMPTY + stage);
  };
  // ends the chunk's loads; the chunk before it has then landed and is handed over
  auto close = [&]() {
    cp_async_commit();
    cp_async_wait<1>();
    if (chunks > 0) bar_arrive<2 * GEMM_THREADS>(BAR_FULL + (stage == 0 ? ZSTAGES - 1 : stage - 1));
    ++chunks;
    stage = stage == ZSTAGES - 1 ? 0 : stage + 1;
  };
  for (int jb = blockIdx.x; jb < njobs; ++seq) {
    const int slot = seq % ZSLOTS;
    bar_sync<GEMM_THREADS>(BAR_LOAD);   // the previous job's descriptors are no longer read
    if (tid < JOB_WORDS)
      reinterpret_cast<long long*>(slots + slot)[tid] = reinterpret_cast<const long long*>(jobs + jb)[tid];
    // the job after this one, taken while this one loads; the last taker of a launch
    // resets the counter for the next launch of the list
    if (tid == GEMM_THREADS - 1) {
      const int k = atomicAdd(next_job, 1);
      if (k == njobs - 1) *next_job = 0;
      nexts[slot] = gridDim.x + k;
    }
    bar_sync<GEMM_THREADS>(BAR_LOAD);
    const ZJob& J = slots[slot];
    const int ng = J.tg - J.t0;   // GEMM terms, first in the job's range
    const int m0 = J.m0, mend = J.mend, n0 = J.n0, nend = J.nend;
    const long long* tw = reinterpret_cast<const long long*>(terms + J.t0);
    jb = nexts[slot];
    for (int i = tid; i < min(ng, ZAHEAD) * TERM_WORDS; i += GEMM_THREADS) ring[i] = tw[i];
    bar_sync<GEMM_THREADS>(BAR_LOAD);
    for (int ti = 0; ti < ng; ++ti) {
      const GTerm& t = reinterpret_cast<const GTerm*>(ring)[ti & (ZRING - 1)];
      const int K = t.K;
      const bool an = t.l_op == OP_N, bn = t.r_op == OP_N;
      const long long lld = t.l_ld, rld = t.r_ld;
      // op N of L is L[m + k ld], op C conj(L[k + m ld]); op N of R is R[k + n ld], op C conj(R[n + k ld])
      const double2* pa = bases.p[t.l_base] + t.l_off +
                          (an ? m0 + AN::f0() + AN::q0() * lld : AC::f0() + (m0 + AC::q0()) * lld);
      const double2* pb = bases.p[t.r_base] + t.r_off +
                          (bn ? BN::f0() + (n0 + BN::q0()) * rld : n0 + BC::f0() + BC::q0() * rld);
      for (int k = 0; k < K; k += TK) {
        open();
        if (k == 0 && ti + ZAHEAD < ng && tid < TERM_WORDS)
          cp_async8(ring + ((ti + ZAHEAD) & (ZRING - 1)) * TERM_WORDS + tid, tw + (ti + ZAHEAD) * TERM_WORDS + tid);
        double2* As = stages + stage * Z::STAGE;
        double2* Bs = As + TK * Z::LDA;
        if (an) {
          AN::copy(As, pa, lld, mend - m0, K - k);
          pa += TK * lld;
        } else {
          AC::copy(As, pa, lld, K - k, mend - m0);
          pa += TK;
        }
        if (bn) {
          BN::copy(Bs, pb, rld, K - k, nend - n0);
          pb += TK;
        } else {
          BC::copy(Bs, pb, rld, nend - n0, K - k);
          pb += TK * rld;
        }
        if (tid == 0) {
          ZMeta m;
          m.ar = t.ar;
          m.ai = t.ai;
          m.lneg = t.l_op == OP_C ? 0x80000000u : 0u;
          m.rneg = t.r_op == OP_C;
          m.ksteps = min(TK / 4, (K - k + 3) / 4);   // k steps past K are zero padding
          m.last = ti == ng - 1 && k + TK >= K;
          m.slot = slot;
          m.lt = m.rt = m.pad0 = m.pad1 = 0;
          metas[stage] = m;
        }
        close();
      }
    }
    if (ng == 0) {   // element terms only: one chunk without a product
      open();
      if (tid == 0) metas[stage] = ZMeta{0.0, 0.0, 0u, 0, 0, 1, (uint8_t)slot, 0, 0, 0, 0};
      close();
    }
  }
  open();
  if (tid == 0) metas[stage] = ZMeta{0.0, 0.0, 0u, 0, 0, 1, (uint8_t)ZSLOTS, 0, 0, 0, 0};
  close();
  cp_async_wait<0>();
  bar_arrive<2 * GEMM_THREADS>(BAR_FULL + (stage == 0 ? ZSTAGES - 1 : stage - 1));
  // leave no arrival of the multiplying warps behind
  for (int s = min(chunks, ZSTAGES); s > 0; --s) bar_sync<2 * GEMM_THREADS>(BAR_EMPTY + (chunks - s) % ZSTAGES);
}

constexpr int Z_FIN_LIMIT = 1 << 24;   // polls of the wait for copies in flight once a wait has run out

__device__ __forceinline__ unsigned z_smem(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void z_bulk(unsigned dst, const double2* src, unsigned bytes, unsigned bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ bool z_wait(unsigned bar, unsigned parity, int limit) {
  for (int i = 0; i < limit; ++i) {
    unsigned done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// The same by bulk copies of the operands' contiguous strips, one a lane, two warps an
// operand.  The copies take no issue slots or load-store unit from the fragment reads,
// which cp.async's 56 instructions a chunk do; with short jobs their latency shows.  The
// loading warps wait for the copies to land, so that the multiplying warps meet them at
// hardware barriers and poll nothing.
// Each such wait gives up after wait_limit polls.  The CTA then ends as a whole: the warp
// sets *fault and the CTA's flag, all four loading warps read it at the end of the next
// chunk, turn the chunk not yet handed over into the end record, wait for the copies in
// flight and issue nothing more; the CTA's job is left unwritten, and the rest of the list
// is taken from the counter without running it, so that the counter ends at zero as after
// any launch.
template <int TM, int TN>
__device__ __forceinline__ void zgemm_load_bulk(unsigned char* smem, const ZJob* jobs, int njobs, const GTerm* terms,
                                                const Bases& bases, int* next_job, int* fault, int wait_limit) {
  using Z = ZTile<TM, TN, true>;
  const int lane = threadIdx.x & 31;
  const int lw = (threadIdx.x >> 5) & 3, sub = lw & 1;   // two warps an operand
  const bool left = lw < 2, lead = lw == 0;
  int* const nexts = reinterpret_cast<int*>(smem + Z::OFF_NEXT);
  double2* const stages = reinterpret_cast<double2*>(smem);
  ZJob* const slots = reinterpret_cast<ZJob*>(smem + Z::OFF_JOBS);
  ZMeta* const metas = reinterpret_cast<ZMeta*>(smem + Z::OFF_META);
  const unsigned bars = z_smem(smem + Z::OFF_BAR);
  int stage = 0, chunks = 0, seq = 0;
  unsigned phase = 0;   // of the stage's copies
  // Set by a wait that ran out at the end of chunk c, in entry c & 1: read at the end of
  // chunk c + 1, behind the barrier that opened it and before the one that the next writer
  // of that entry has to pass.
  volatile int* const gave_up = reinterpret_cast<volatile int*>(smem + Z::OFF_GAVE_UP);
  // opens the stage of the next chunk: the multiplying warps are done with what it held
  auto open = [&](unsigned bytes) {
    if (chunks >= ZSTAGES)
      bar_sync<2 * GEMM_THREADS>(BAR_EMPTY + stage);
    else
      bar_sync<GEMM_THREADS>(BAR_LOAD);
    if (lane == 0)
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bars + 8 * stage), "r"(bytes) : "memory");
    __syncwarp();
  };
  // waits for the copies of the stage before this one and hands it over; within the stream
  // (more) a wait that runs out stops the CTA.  The hand-over after the stream's end must not
  // set the flag: a slower warp may yet have to read that entry.
  auto landed = [&](bool more) {
    const int s = stage == 0 ? ZSTAGES - 1 : stage - 1;
    const unsigned ph = stage == 0 ? phase ^ 1 : phase;
    if (!__all_sync(0xffffffffu, z_wait(bars + 8 * s, ph, wait_limit))) {
      if (lane == 0) {
        atomicOr(fault, FAULT_FP64);
        if (more) gave_up[chunks & 1] = 1;
      }
      z_wait(bars + 8 * s, ph, Z_FIN_LIMIT);
    }
    __syncwarp();
    bar_arrive<2 * GEMM_THREADS>(BAR_FULL + s);
  };
  // ends the chunk's loads and hands over the chunk before it; false in all four warps once
  // a wait has run out
  auto close = [&]() -> bool {
    if (chunks > 0) {
      if (gave_up[(chunks - 1) & 1]) return false;
      landed(true);
    }
    ++chunks;
    if (++stage == ZSTAGES) {
      stage = 0;
      phase ^= 1;
    }
    return true;
  };
  const ZMeta end{0.0, 0.0, 0u, 0, 0, 1, (uint8_t)ZSLOTS, 0, 0, 0, 0};
  int slot = 0;
  const bool ok = [&]() -> bool {
    for (int jb = blockIdx.x; jb < njobs; ++seq) {
      slot = seq % ZSLOTS;
      const ZJob& J = jobs[jb];
      const int t0 = J.t0, tg = J.tg, m0 = J.m0, n0 = J.n0, rows = J.mend - m0, cols = J.nend - n0;
      if (lead && lane < JOB_WORDS)
        reinterpret_cast<long long*>(slots + slot)[lane] = reinterpret_cast<const long long*>(jobs + jb)[lane];
      // the job after this one, taken while this one loads; the last taker of a launch
      // resets the counter for the next launch of the list
      if (lead && lane == 0) {
        const int k = atomicAdd(next_job, 1);
        if (k == njobs - 1) *next_job = 0;
        nexts[slot] = gridDim.x + k;
      }
      for (int tb = t0; tb < tg; tb += 32) {
        // the descriptors of 32 terms at once, one a lane
        const double2* p = nullptr;
        int ld = 0, tK = 0;
        unsigned ops = 0;
        if (tb + lane < tg) {
          const GTerm& t = terms[tb + lane];
          ops = (t.l_op == OP_N ? 0u : 1u) | (t.r_op == OP_N ? 0u : 2u);
          tK = t.K;
          // op N of L is L[m + k ld], op C conj(L[k + m ld]); op N of R is R[k + n ld], op C conj(R[n + k ld])
          ld = left ? t.l_ld : t.r_ld;
          p = left ? bases.p[t.l_base] + t.l_off + (ops & 1 ? (long long)m0 * ld : m0)
                   : bases.p[t.r_base] + t.r_off + (ops & 2 ? n0 : (long long)n0 * ld);
        }
        const int cnt = min(32, tg - tb);
        for (int i = 0; i < cnt; ++i) {
          const int K = __shfl_sync(0xffffffffu, tK, i);
          const unsigned op = __shfl_sync(0xffffffffu, ops, i);
          const bool ac = op & 1, bc = op & 2;
          const bool along_k = left ? ac : !bc;   // strips of one row's (column's) k
          const long long inc = __shfl_sync(0xffffffffu, ld, i);
          const double2* x = (const double2*)__shfl_sync(0xffffffffu, (unsigned long long)p, i);
          const int ext = left ? rows : cols, strip = left ? Z::LDA : Z::LDB, full = left ? TM : TN;
          for (int k = 0; k < K; k += TK) {
            const int kc = min(TK, K - k);
            const int mine = along_k ? max(0, min(32, ext - 32 * sub)) * kc : sub ? 0 : kc * ext;
            open((unsigned)mine * 16u);
            double2* S = stages + stage * Z::STAGE + (left ? 0 : Z::ELA);
            const unsigned bar = bars + 8 * stage, sd = z_smem(S);
            if (along_k) {
              const int r = lane + 32 * sub;
              if (r < ext) z_bulk(sd + r * Z::LDK * 16, x + r * inc, kc * 16, bar);
              x += TK;
            } else {
              if (!sub && lane < kc) z_bulk(sd + lane * strip * 16, x + lane * inc, ext * 16, bar);
              x += TK * inc;
            }
            if (kc & 3) {   // the last k step's rows past K must be zero
              const int kz = ((kc + 3) & ~3) - kc;
              for (int e = lane + 32 * sub; e < kz * full; e += 64) {
                const int kk = kc + e / full, r = e % full;
                S[along_k ? r * Z::LDK + kk : kk * strip + r] = make_double2(0.0, 0.0);
              }
              asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // a later copy writes here again
            }
            if (lead && lane == 0) {
              const GTerm& t = terms[tb + i];
              ZMeta m;
              m.ar = t.ar;
              m.ai = t.ai;
              m.lneg = ac ? 0x80000000u : 0u;
              m.rneg = bc;
              m.ksteps = (kc + 3) / 4;
              m.last = tb + i == tg - 1 && k + TK >= K;
              m.slot = slot;
              m.lt = ac;
              m.rt = !bc;
              m.pad0 = m.pad1 = 0;
              metas[stage] = m;
            }
            if (!close()) return false;
          }
        }
      }
      if (tg == t0) {   // element terms only: one chunk without a product
        open(0);
        if (lead && lane == 0) metas[stage] = ZMeta{0.0, 0.0, 0u, 0, 0, 1, (uint8_t)slot, 0, 0, 0, 0};
        if (!close()) return false;
      }
      bar_sync<GEMM_THREADS>(BAR_LOAD);
      jb = nexts[slot];
    }
    open(0);
    if (lead && lane == 0) metas[stage] = end;
    return close();
  }();
  if (!ok && lead && lane == 0) {
    // the chunk before this one is issued and not handed over: it becomes the end
    metas[stage == 0 ? ZSTAGES - 1 : stage - 1] = end;
    for (int jb = nexts[slot]; jb < njobs;) {
      const int k = atomicAdd(next_job, 1);
      if (k == njobs - 1) *next_job = 0;
      jb = gridDim.x + k;
    }
  }
  landed(false);
  if (!ok) z_wait(bars + 8 * stage, phase, Z_FIN_LIMIT);   // this chunk's copies
  // leave no arrival of the multiplying warps behind (of the chunk given up there is none)
  for (int s = min(chunks, ok ? ZSTAGES : ZSTAGES - 1); s > 0; --s)
    bar_sync<2 * GEMM_THREADS>(BAR_EMPTY + (chunks - s) % ZSTAGES);
}

// Multiplying half of a CTA: sums a job's terms in registers and writes its tile once.
template <int TM, int TN, bool BULK>
__device__ __forceinline__ void zgemm_multiply(unsigned char* smem, const GTerm* terms, const Bases& bases) {
  constexpr int MI = TM / 16, NI = TN / 16;   // 8x8 MMA sub-tiles of one warp, at most
  using Z = ZTile<TM, TN, BULK>;
  const double2* const stages = reinterpret_cast<const double2*>(smem);
  const ZJob* const slots = reinterpret_cast<const ZJob*>(smem + Z::OFF_JOBS);
  const ZMeta* const metas = reinterpret_cast<const ZMeta*>(smem + Z::OFF_META);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int lg = lane >> 2, lt = lane & 3;
  int stage = 0;
  while (true) {
    bar_sync<2 * GEMM_THREADS>(BAR_FULL + stage);
    ZMeta m = metas[stage];
    if (m.slot == ZSLOTS) {
      bar_arrive<2 * GEMM_THREADS>(BAR_EMPTY + stage);
      return;
    }
    const ZJob& J = slots[m.slot];
    // the tile's sub-tiles are dealt to the warps, 2 x 2 or, for flat tiles, 1 x 4 or
    // 4 x 1, whichever leaves the busiest warp the least
    const int mtot = (J.mend - J.m0 + 7) / 8, ntot = (J.nend - J.n0 + 7) / 8;
    int wms, wns;
    warp_grid(mtot, ntot, MI, NI, wms, wns);
    const int mh = (mtot + wms - 1) / wms, nh = (ntot + wns - 1) / wns;
    const int wm = warp % wms, wn = warp / wms;
    const int wrow = wm * mh * 8 + lg, wcol = wn * nh * 8;
    const int mt = max(0, min(mh, mtot - wm * mh)), nt = max(0, min(nh, ntot - wn * nh));
    double t1[MI][NI][2], t2[MI][NI][2], t3[MI][NI][2];
#pragma unroll
    for (int a = 0; a < MI; ++a)
#pragma unroll
      for (int b = 0; b < NI; ++b)
#pragma unroll
        for (int e = 0; e < 2; ++e) t1[a][b][e] = t2[a][b][e] = t3[a][b][e] = 0.0;
    while (true) {
      // strides of a sub-tile and of a k step, in the order the operand was staged
      const bool ak = BULK && m.lt, bk = BULK && m.rt;
      const int sma = ak ? 8 * Z::LDK : 8, ska = ak ? 4 : 4 * Z::LDA;
      const int snb = bk ? 8 * Z::LDK : 8, skb = bk ? 4 : 4 * Z::LDB;
      const double2* As = stages + stage * Z::STAGE + (ak ? wrow * Z::LDK + lt : lt * Z::LDA + wrow);
      const double2* Bs = stages + stage * Z::STAGE + Z::ELA +
                          (bk ? (wcol + lg) * Z::LDK + lt : lt * Z::LDB + wcol + lg);
      if (mt > 0 && nt > 0) mma_select<MI, NI, MI, NI>(t1, t2, t3, As, Bs, sma, ska, snb, skb, m, mt, nt);
      bar_arrive<2 * GEMM_THREADS>(BAR_EMPTY + stage);
      stage = stage == ZSTAGES - 1 ? 0 : stage + 1;
      if (m.last) break;
      bar_sync<2 * GEMM_THREADS>(BAR_FULL + stage);
      m = metas[stage];
      if constexpr (BULK) {   // the loading warps gave up within a job: its tile is not written
        if (m.slot == ZSLOTS) {
          bar_arrive<2 * GEMM_THREADS>(BAR_EMPTY + stage);
          return;
        }
      }
    }
    // the products: real part into t1, imaginary part into t3
#pragma unroll
    for (int mi = 0; mi < MI; ++mi)
#pragma unroll
      for (int ni = 0; ni < NI; ++ni)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const double x1 = t1[mi][ni][e], x2 = t2[mi][ni][e];
          t1[mi][ni][e] = x1 - x2;
          t3[mi][ni][e] = t3[mi][ni][e] - x1 - x2;
        }
    const int row0 = J.m0 + wrow, col0 = J.n0 + wcol + 2 * lt, mend = J.mend, nend = J.nend;
    // element-wise terms on the accumulator layout
    for (int ti = J.tg; ti < J.t1; ++ti) {
      const GTerm t = terms[ti];
      if (t.kind == TK_GEMM) continue;   // of zero depth
      const double2* R = bases.p[t.r_base] + t.r_off;
#pragma unroll
      for (int mi = 0; mi < MI; ++mi)
#pragma unroll
        for (int ni = 0; ni < NI; ++ni)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int row = row0 + mi * 8, col = col0 + ni * 8 + e;
            const int rr = row - t.r0, cc = col - t.c0;
            if (mi >= mt || ni >= nt) continue;
            if (row >= mend || col >= nend || rr < 0 || cc < 0 || rr >= t.rm || cc >= t.rn) continue;
            double vr, vi;
            if (t.kind == TK_AXPY) {
              double2 v = (t.r_op == OP_N) ? R[(long long)rr + (long long)cc * t.r_ld]
                                           : R[(long long)cc + (long long)rr * t.r_ld];
              vr = v.x;
              vi = (t.r_op == OP_C) ? -v.y : v.y;
            } else {
              if (rr != cc) continue;
              vr = 1.0;
              vi = 0.0;
            }
            t1[mi][ni][e] += t.ar * vr - t.ai * vi;
            t3[mi][ni][e] += t.ar * vi + t.ai * vr;
          }
    }
    double2* C = bases.p[J.c_base] + J.c_off;
    const long long ldc = J.c_ld;
    const bool acc_old = J.beta;
#pragma unroll
    for (int mi = 0; mi < MI; ++mi)
#pragma unroll
      for (int ni = 0; ni < NI; ++ni)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int row = row0 + mi * 8, col = col0 + ni * 8 + e;
          if (mi < mt && ni < nt && row < mend && col < nend) {
            double2* p = C + (long long)row + (long long)col * ldc;
            double2 v = make_double2(t1[mi][ni][e], t3[mi][ni][e]);
            if (acc_old) {
              double2 o = *p;
              v.x += o.x;
              v.y += o.y;
            }
            *p = v;
          }
        }
  }
}

// Persistent, warp-specialised: warps 0-3 multiply, warps 4-7 load.  The registers the
// block was launched with are split LREGS : CREGS between the two halves.
template <int TM, int TN, int MINB, int LREGS, int CREGS, bool BULK>
__global__ void __launch_bounds__(2 * GEMM_THREADS, MINB)
grouped_zgemm_kernel(const ZJob* __restrict__ jobs, int njobs, const GTerm* __restrict__ terms,
                     const __grid_constant__ Bases bases, int* next_job, int* fault, int wait_limit) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  chain_kernels();
  if constexpr (BULK) {
    if (threadIdx.x < ZSTAGES)   // one arrival of each loading warp
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;" ::"r"(z_smem(smem_raw + ZTile<TM, TN, BULK>::OFF_BAR) +
                                                                  8 * threadIdx.x)
                   : "memory");
    if (threadIdx.x < 2) reinterpret_cast<int*>(smem_raw + ZTile<TM, TN, BULK>::OFF_GAVE_UP)[threadIdx.x] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncthreads();
  }
  if (threadIdx.x >= GEMM_THREADS) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(LREGS));
    if constexpr (BULK)
      zgemm_load_bulk<TM, TN>(smem_raw, jobs, njobs, terms, bases, next_job, fault, wait_limit);
    else
      zgemm_load<TM, TN>(smem_raw, jobs, njobs, terms, bases, next_job);
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(CREGS));
    zgemm_multiply<TM, TN, BULK>(smem_raw, terms, bases);
  }
}

// Lists without GEMM terms (operator merges, block enlargement): one 32x32 tile per CTA,
// four elements of a column strip per thread, each summed over the job's terms in order
// and written once.  Bound by the operands' bytes.
__global__ void __launch_bounds__(256) grouped_axpy_kernel(const ZJob* __restrict__ jobs, const GTerm* __restrict__ terms,
                                                           const __grid_constant__ Bases bases) {
  const ZJob J = jobs[blockIdx.x];
  const int row = J.m0 + (threadIdx.x & 31), col0 = J.n0 + (threadIdx.x >> 5);
  double2 acc[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) acc[i] = make_double2(0.0, 0.0);
  if (row >= J.mend) return;
  for (int ti = J.t0; ti < J.t1; ++ti) {
    const GTerm t = terms[ti];
    const int rr = row - t.r0;
    if (t.kind == TK_GEMM || rr < 0 || rr >= t.rm) continue;
    const double2* R = bases.p[t.r_base] + t.r_off;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int col = col0 + 8 * i, cc = col - t.c0;
      if (col >= J.nend || cc < 0 || cc >= t.rn) continue;
      double2 v = make_double2(1.0, 0.0);
      if (t.kind == TK_AXPY) {
        v = t.r_op == OP_N ? R[(long long)rr + (long long)cc * t.r_ld] : R[(long long)cc + (long long)rr * t.r_ld];
        if (t.r_op == OP_C) v.y = -v.y;
      } else if (rr != cc) {
        continue;
      }
      acc[i].x += t.ar * v.x - t.ai * v.y;
      acc[i].y += t.ar * v.y + t.ai * v.x;
    }
  }
  double2* C = bases.p[J.c_base] + J.c_off;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int col = col0 + 8 * i;
    if (col >= J.nend) continue;
    double2* p = C + (long long)row + (long long)col * J.c_ld;
    if (J.beta) {
      const double2 o = *p;
      acc[i].x += o.x;
      acc[i].y += o.y;
    }
    *p = acc[i];
  }
}

// C = sum of the partial tiles of a split group in fixed order (+ beta*C_old)
__global__ void reduce_partials_kernel(const GReduce* __restrict__ reds, const GGroup* __restrict__ groups,
                                       Bases bases) {
  chain_kernels();
  const GReduce r = reds[blockIdx.y];
  const GGroup g = groups[r.group];
  const long long mn = (long long)g.M * g.N;
  double2* C = bases.p[g.c_base] + g.c_off;
  const double2* P = bases.p[BASE_PART] + r.part_off;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < mn; e += (long long)gridDim.x * blockDim.x) {
    double sr = 0.0, si = 0.0;
    for (int p = 0; p < r.nparts; ++p) {
      double2 v = P[(long long)p * mn + e];
      sr += v.x;
      si += v.y;
    }
    const long long row = e % g.M, col = e / g.M;
    double2* c = C + row + col * g.c_ld;
    if (g.beta) {
      double2 o = *c;
      sr += o.x;
      si += o.y;
    }
    *c = make_double2(sr, si);
  }
}

// ---------------------------------------------------------------- vector kernels
constexpr int VB = 256;          // threads per block
constexpr int VCHUNK = 8192;     // elements per block in reductions

__global__ void multi_dot_partial(const double2* __restrict__ X, long long ld, int nvec,
                                  const double2* __restrict__ y, long long n, double* __restrict__ partial,
                                  int nblk) {
  __shared__ double red[VB / 32];
  long long beg = (long long)blockIdx.x * VCHUNK;
  long long end = beg + VCHUNK < n ? beg + VCHUNK : n;
  for (int j = 0; j < nvec; ++j) {
    const double2* x = X + (long long)j * ld;
    double acc = 0.0;
    for (long long e = beg + threadIdx.x; e < end; e += VB) {
      double2 a = x[e], b = y[e];
      acc = fma(a.x, b.x, acc);
      acc = fma(a.y, b.y, acc);
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
      double s = 0.0;
      for (int w = 0; w < VB / 32; ++w) s += red[w];
      partial[(long long)j * nblk + blockIdx.x] = s;
    }
    __syncthreads();
  }
}

// partial sums of <x, y> = sum conj(x) y: real parts at partial[b], imaginary at partial[nblk + b]
__global__ void zdot_partial(const double2* __restrict__ x, const double2* __restrict__ y, long long n,
                             double* __restrict__ partial, int nblk) {
  __shared__ double red[2][VB / 32];
  const long long beg = (long long)blockIdx.x * VCHUNK;
  const long long end = beg + VCHUNK < n ? beg + VCHUNK : n;
  double ar = 0.0, ai = 0.0;
  for (long long e = beg + threadIdx.x; e < end; e += VB) {
    const double2 a = x[e], b = y[e];
    ar = fma(a.x, b.x, ar);
    ar = fma(a.y, b.y, ar);
    ai = fma(a.x, b.y, ai);
    ai = fma(-a.y, b.x, ai);
  }
  for (int o = 16; o > 0; o >>= 1) {
    ar += __shfl_xor_sync(0xffffffffu, ar, o);
    ai += __shfl_xor_sync(0xffffffffu, ai, o);
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = ar;
    red[1][threadIdx.x >> 5] = ai;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double sr = 0.0, si = 0.0;
    for (int w = 0; w < VB / 32; ++w) {
      sr += red[0][w];
      si += red[1][w];
    }
    partial[blockIdx.x] = sr;
    partial[nblk + blockIdx.x] = si;
  }
}

__global__ void multi_dot_final(const double* __restrict__ partial, int nblk, int nvec, double* __restrict__ out) {
  int j = blockIdx.x;
  if (j >= nvec) return;
  __shared__ double red[32];
  double acc = 0.0;
  for (int b = threadIdx.x; b < nblk; b += blockDim.x) acc += partial[(long long)j * nblk + b];
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w];
    out[j] = s;
  }
}

// w = w / sqrt(norm2)   (wave_normalize, block.f90:1135-1150)
__global__ void scale_kernel(double2* __restrict__ w, const double* __restrict__ norm2, long long n, int invert_sqrt) {
  const double s = invert_sqrt ? sqrt(*norm2) : *norm2;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
    double2 x = w[e];
    x.x = x.x / s;
    x.y = x.y / s;
    w[e] = x;
  }
}

// out = sum_i z_i x_i   (eigen.f90:146-153)
__global__ void combine_kernel(double2* __restrict__ out, const double2* __restrict__ X, long long ld, int nvec,
                               const double* __restrict__ z, long long n) {
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
    double r = 0.0, im = 0.0;
    for (int j = 0; j < nvec; ++j) {
      double2 x = X[(long long)j * ld + e];
      r = r + z[j] * x.x;
      im = im + z[j] * x.y;
    }
    out[e] = make_double2(r, im);
  }
}

// number of eigenvalues of T below x (Sturm sequence)
__device__ int sturm_count(const double* d, const double* e, int n, double x, double pivmin) {
  int c = 0;
  double q = d[0] - x;
  if (fabs(q) < pivmin) q = -pivmin;
  if (q < 0) c++;
  for (int i = 1; i < n; ++i) {
    q = d[i] - x - e[i - 1] * e[i - 1] / q;
    if (fabs(q) < pivmin) q = -pivmin;
    if (q < 0) c++;
  }
  return c;
}

// Lowest eigenpair of the symmetric tridiagonal T (diag d[0..n), off-diagonal
// e[0..n-1)), the part of dstev the Lanczos loop uses (eigen.f90:99-141).  One
// warp: the eigenvalue by Sturm-count multisection (32 interior points per
// round, each lane counting at one point, so a round shrinks the bracket 33x),
// the eigenvector by inverse iteration in lane 0.  n <= 127.
__device__ void tridiag_lowest_warp(const double* __restrict__ d, const double* __restrict__ e, int n,
                                    int want_vec, double* __restrict__ res, double* __restrict__ z) {
  const int lane = threadIdx.x & 31;
  if (n == 1) {
    if (lane == 0) {
      res[0] = d[0];
      if (want_vec) z[0] = 1.0;
    }
    return;
  }
  double lo = d[0], hi = d[0], emax = 0.0;
  for (int i = 0; i < n; ++i) {
    double r = (i > 0 ? fabs(e[i - 1]) : 0.0) + (i < n - 1 ? fabs(e[i]) : 0.0);
    lo = fmin(lo, d[i] - r);
    hi = fmax(hi, d[i] + r);
    if (i < n - 1) emax = fmax(emax, e[i] * e[i]);
  }
  const double tnorm = fmax(fabs(lo), fabs(hi));
  const double pivmin = DBL_MIN * fmax(1.0, emax);
  lo -= 2.0 * DBL_EPSILON * tnorm + pivmin;
  hi += 2.0 * DBL_EPSILON * tnorm + pivmin;
  // invariant: count(lo) == 0, count(hi) >= 1 (Gershgorin bounds)
  for (int round = 0; round < 64; ++round) {
    if (hi - lo <= 2.0 * DBL_EPSILON * fmax(fabs(lo), fabs(hi)) + pivmin) break;
    const double x = lo + (hi - lo) * (double)(lane + 1) * (1.0 / 33.0);
    const bool above = (x < hi) && (x > lo) && sturm_count(d, e, n, x, pivmin) >= 1;
    const unsigned ball = __ballot_sync(0xffffffffu, above);
    const unsigned below = __ballot_sync(0xffffffffu, (x > lo) && (x < hi) && !above);
    // new bracket: the lowest point with count >= 1, and the highest point
    // under it with count 0 (points outside (lo, hi) by rounding are skipped)
    const int j = ball ? __ffs(ball) - 1 : 32;
    const unsigned under = below & (j >= 32 ? 0xffffffffu : ((1u << j) - 1u));
    const int i = under ? 31 - __clz(under) : -1;
    const double xj = __shfl_sync(0xffffffffu, x, j & 31);
    const double xi = __shfl_sync(0xffffffffu, x, i < 0 ? 0 : i);
    const double nhi = (j < 32) ? xj : hi;
    const double nlo = (i >= 0) ? xi : lo;
    if (nhi >= hi && nlo <= lo) break;   // no representable progress
    lo = nlo;
    hi = nhi;
  }
  const double lam = 0.5 * (lo + hi);
  if (lane != 0) return;
  res[0] = lam;
  if (!want_vec) return;
  // inverse iteration on (T - lam I) with a partially pivoted tridiagonal LU
  // (rows kept as diag/super1/super2 of U plus multipliers); n <= 127.
  double u0[128], u1[128], u2[128], lm[128], y[128];
  int piv[128];
  const double shift = lam;
  const double tiny = DBL_EPSILON * tnorm + pivmin;
  {
    double a = d[0] - shift, b = (n > 1) ? e[0] : 0.0, c = 0.0;
    for (int i = 0; i < n - 1; ++i) {
      double sub = e[i], na = d[i + 1] - shift, nb = (i + 1 < n - 1) ? e[i + 1] : 0.0;
      if (fabs(a) >= fabs(sub)) {
        piv[i] = 0;
        if (fabs(a) < tiny) a = (a < 0 ? -tiny : tiny);
        double l = sub / a;
        lm[i] = l;
        u0[i] = a; u1[i] = b; u2[i] = c;
        a = na - l * b;
        b = nb - l * c;
        c = 0.0;
      } else {
        piv[i] = 1;
        double l = a / sub;
        lm[i] = l;
        u0[i] = sub; u1[i] = na; u2[i] = nb;
        double a2 = b - l * na, b2 = c - l * nb;
        a = a2;
        b = b2;
        c = 0.0;
      }
    }
    if (fabs(a) < tiny) a = (a < 0 ? -tiny : tiny);
    u0[n - 1] = a; u1[n - 1] = 0.0; u2[n - 1] = 0.0;
  }
  for (int i = 0; i < n; ++i) y[i] = 1.0;
  for (int pass = 0; pass < 3; ++pass) {
    // forward: apply row swaps and multipliers to y
    for (int i = 0; i < n - 1; ++i) {
      if (piv[i]) {
        double t = y[i];
        y[i] = y[i + 1];
        y[i + 1] = t;
      }
      y[i + 1] -= lm[i] * y[i];
    }
    // back substitution with U (diag u0, super u1, u2)
    for (int i = n - 1; i >= 0; --i) {
      double s = y[i];
      if (i + 1 < n) s -= u1[i] * y[i + 1];
      if (i + 2 < n) s -= u2[i] * y[i + 2];
      y[i] = s / u0[i];
    }
    double nrm = 0.0;
    for (int i = 0; i < n; ++i) nrm += y[i] * y[i];
    nrm = sqrt(nrm);
    for (int i = 0; i < n; ++i) y[i] /= nrm;
  }
  int imax = 0;
  for (int i = 1; i < n; ++i)
    if (fabs(y[i]) > fabs(y[imax])) imax = i;
  const double sg = y[imax] < 0 ? -1.0 : 1.0;
  for (int i = 0; i < n; ++i) z[i] = sg * y[i];
}


__global__ void tridiag_lowest_kernel(const double* __restrict__ d, const double* __restrict__ e, int n,
                                      int want_vec, double* __restrict__ res, double* __restrict__ z) {
  tridiag_lowest_warp(d, e, n, want_vec, res, z);
}

__global__ void phase_fix_kernel(double2* __restrict__ U, int rows) {
  double2* u = U + (long long)blockIdx.x * rows;
  __shared__ double sr[32], si[32];
  double zr = 0.0, zi = 0.0;
  for (int r = threadIdx.x; r < rows; r += blockDim.x) {
    double w = 1.0 / (1.0 + 0.1 * r);
    zr += u[r].x * w;
    zi += u[r].y * w;
  }
  for (int o = 16; o > 0; o >>= 1) {
    zr += __shfl_xor_sync(0xffffffffu, zr, o);
    zi += __shfl_xor_sync(0xffffffffu, zi, o);
  }
  if ((threadIdx.x & 31) == 0) {
    sr[threadIdx.x >> 5] = zr;
    si[threadIdx.x >> 5] = zi;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0, b = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
      a += sr[w];
      b += si[w];
    }
    sr[0] = a;
    si[0] = b;
  }
  __syncthreads();
  const double a = hypot(sr[0], si[0]);
  if (a < 1e-10) return;
  const double fr = sr[0] / a, fi = -si[0] / a;
  for (int r = threadIdx.x; r < rows; r += blockDim.x) {
    double2 x = u[r];
    u[r] = make_double2(x.x * fr - x.y * fi, x.x * fi + x.y * fr);
  }
}

// ---- one Lanczos iteration's vector work --------------------------------------------
// Four kernels around the H.psi, the iteration's index read on the device (*it is `last`,
// 1-based, as eigen.f90), so that one captured CUDA graph serves every iteration.  Each
// ends its own reductions: every block leaves partial sums, and the last block to finish
// adds them in a fixed order, so results do not depend on the schedule.
//
// Small solves are bound by the number of dependent launches and by the little work each
// has: as update, norm, scale, dots, Gram-Schmidt, norm, scale, norm, copies, dot and the
// eigenvalue (18 kernels, reductions in blocks of 8,192 elements) the vector work of one
// iteration at 6,800 amplitudes and 20 Krylov vectors took 130 us beside 35 us of H.psi.
// Large ones are bound by reading the Krylov basis twice.
constexpr int IT_THREADS = 256, IT_WARPS = IT_THREADS / 32, IT_SUB = 1024, IT_MAXVEC = 128;

__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sum over the block, in every thread (one use of `red` per call site and barrier phase)
__device__ __forceinline__ double block_sum(double v, double* red) {
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
  for (int w = 0; w < IT_WARPS; ++w) s += red[w];
  return s;
}

// True in every thread of the last block to arrive; the counter is then zero again.
__device__ __forceinline__ bool last_block(int* counter) {
  __shared__ int last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last = atomicAdd(counter, 1) == (int)gridDim.x - 1;
    if (last) *counter = 0;
  }
  __syncthreads();
  if (last) __threadfence();
  return last != 0;
}

// Sum of the blocks' partials p[0 .. gridDim.x), by one warp, in every lane
__device__ __forceinline__ double partial_sum(const double* p) {
  double v = 0.0;
  for (int b = threadIdx.x & 31; b < (int)gridDim.x; b += 32) v += __ldcg(p + b);
  return warp_sum(v);
}

// w = v(last+1) -= alpha_last v(last) + beta_(last-1) v(last-1); n2 = |w|^2 and, of the
// normalised w, uv_j = Re<v(j), w> for j <= last, in the same pass (eigen.f90:65-75,
// block.f90:1265-1275).  A warp takes whole vectors: its lanes' sums meet once per vector.
__global__ void __launch_bounds__(IT_THREADS) it_project_kernel(double2* __restrict__ V, long long ld,
                                                                const double* __restrict__ alpha,
                                                                const double* __restrict__ beta, long long n, int sub,
                                                                const int* __restrict__ it, double* __restrict__ partial,
                                                                int* counter, double* __restrict__ n2,
                                                                double* __restrict__ uv) {
  __shared__ double2 sw[IT_SUB];
  __shared__ double sacc[IT_MAXVEC], red[IT_WARPS];
  const int last = *it, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double2* w = V + (long long)last * ld;
  const double2* v = V + (long long)(last - 1) * ld;
  const double2* vprev = last >= 2 ? V + (long long)(last - 2) * ld : nullptr;
  const double a = alpha[last], b = last >= 2 ? beta[last - 1] : 0.0;
  for (int j = tid; j < last; j += IT_THREADS) sacc[j] = 0.0;
  double nrm = 0.0;
  for (long long base = (long long)blockIdx.x * sub; base < n; base += (long long)gridDim.x * sub) {
    const int m = (int)(n - base < sub ? n - base : sub);
    __syncthreads();   // sw is free again
    for (int e = tid; e < m; e += IT_THREADS) {
      double2 x = w[base + e];
      const double2 p = v[base + e];
      x.x = x.x - a * p.x;
      x.y = x.y - a * p.y;
      if (vprev) {
        const double2 q = vprev[base + e];
        x.x = x.x - b * q.x;
        x.y = x.y - b * q.y;
      }
      w[base + e] = x;
      sw[e] = x;
      nrm = fma(x.x, x.x, nrm);
      nrm = fma(x.y, x.y, nrm);
    }
    __syncthreads();
    for (int j = warp; j < last; j += IT_WARPS) {
      const double2* x = V + (long long)j * ld + base;
      double acc0 = 0.0, acc1 = 0.0;
#pragma unroll 8
      for (int e = lane; e < m; e += 32) {
        const double2 p = x[e], y = sw[e];
        acc0 = fma(p.x, y.x, acc0);
        acc1 = fma(p.y, y.y, acc1);
      }
      const double t = warp_sum(acc0 + acc1);
      if (lane == 0) sacc[j] += t;
    }
  }
  nrm = block_sum(nrm, red);
  if (tid == 0) partial[blockIdx.x] = nrm;
  for (int j = tid; j < last; j += IT_THREADS) partial[(long long)(j + 1) * gridDim.x + blockIdx.x] = sacc[j];
  if (!last_block(counter)) return;
  const double total = partial_sum(partial);
  if (tid == 0) *n2 = total;
  const double s = sqrt(total);
  for (int j = warp; j < last; j += IT_WARPS) {
    const double t = partial_sum(partial + (long long)(j + 1) * gridDim.x);
    if (lane == 0) uv[j] = t / s;
  }
}

// w = w / |w| - sum_j (uv_j / uu_j) v(j), the Gram_Schmidt_process of block.f90:1265-1285
// on the normalised vector; nw2 = |w|^2 of the result
__global__ void __launch_bounds__(IT_THREADS) it_orthogonalize_kernel(double2* __restrict__ V, long long ld,
                                                                      const double* __restrict__ n2,
                                                                      const double* __restrict__ uv,
                                                                      const double* __restrict__ uu, long long n,
                                                                      const int* __restrict__ it,
                                                                      double* __restrict__ partial, int* counter,
                                                                      double* __restrict__ nw2) {
  __shared__ double sc[IT_MAXVEC], red[IT_WARPS];
  const int last = *it;
  double2* w = V + (long long)last * ld;
  const double s = sqrt(*n2);
  for (int j = threadIdx.x; j < last; j += IT_THREADS) sc[j] = uv[j] / uu[j];
  __syncthreads();
  double nrm = 0.0;
  for (long long e = (long long)blockIdx.x * IT_THREADS + threadIdx.x; e < n; e += (long long)gridDim.x * IT_THREADS) {
    double2 x = w[e];
    x.x = x.x / s;
    x.y = x.y / s;
    double tr = 0.0, tim = 0.0;
#pragma unroll 8
    for (int j = 0; j < last; ++j) {
      const double2 p = V[(long long)j * ld + e];
      tr = tr + sc[j] * p.x;
      tim = tim + sc[j] * p.y;
    }
    x.x = x.x - tr;
    x.y = x.y - tim;
    w[e] = x;
    nrm = fma(x.x, x.x, nrm);
    nrm = fma(x.y, x.y, nrm);
  }
  nrm = block_sum(nrm, red);
  if (threadIdx.x == 0) partial[blockIdx.x] = nrm;
  if (!last_block(counter)) return;
  const double total = partial_sum(partial);
  if (threadIdx.x == 0) *nw2 = total;
}

// v(last+1) = x = w / |w| (wave_normalize), uu_(last+1) = <w, w> after it
__global__ void __launch_bounds__(IT_THREADS) it_normalize_kernel(double2* __restrict__ V, long long ld,
                                                                  const double* __restrict__ nw2, long long n,
                                                                  const int* __restrict__ it, double2* __restrict__ x,
                                                                  double* __restrict__ partial, int* counter,
                                                                  double* __restrict__ uu) {
  __shared__ double red[IT_WARPS];
  const int last = *it;
  double2* w = V + (long long)last * ld;
  const double s = sqrt(*nw2);
  double nrm = 0.0;
  for (long long e = (long long)blockIdx.x * IT_THREADS + threadIdx.x; e < n; e += (long long)gridDim.x * IT_THREADS) {
    double2 y = w[e];
    y.x = y.x / s;
    y.y = y.y / s;
    w[e] = y;
    x[e] = y;
    nrm = fma(y.x, y.x, nrm);
    nrm = fma(y.y, y.y, nrm);
  }
  nrm = block_sum(nrm, red);
  if (threadIdx.x == 0) partial[blockIdx.x] = nrm;
  if (!last_block(counter)) return;
  const double total = partial_sum(partial);
  if (threadIdx.x == 0) uu[last] = total;
}

// Lowest eigenvalue of the symmetric tridiagonal (d, e) in shared memory, by the block's
// Sturm counts at IT_THREADS points a round (the bracket shrinks 257-fold: 7 rounds, where
// a warp's 33-fold takes 11; the serial chain of divisions in one count is the cost).  The
// same invariant and end as tridiag_lowest_warp.
__device__ double tridiag_lowest_block(const double* d, const double* e, int n) {
  __shared__ double slo, shi;
  __shared__ int first[IT_WARPS], under[IT_WARPS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (n == 1) return d[0];
  double lo = d[0], hi = d[0], emax = 0.0;
  for (int i = 0; i < n; ++i) {
    const double r = (i > 0 ? fabs(e[i - 1]) : 0.0) + (i < n - 1 ? fabs(e[i]) : 0.0);
    lo = fmin(lo, d[i] - r);
    hi = fmax(hi, d[i] + r);
    if (i < n - 1) emax = fmax(emax, e[i] * e[i]);
  }
  const double tnorm = fmax(fabs(lo), fabs(hi));
  const double pivmin = DBL_MIN * fmax(1.0, emax);
  lo -= 2.0 * DBL_EPSILON * tnorm + pivmin;
  hi += 2.0 * DBL_EPSILON * tnorm + pivmin;
  for (int round = 0; round < 64; ++round) {
    if (hi - lo <= 2.0 * DBL_EPSILON * fmax(fabs(lo), fabs(hi)) + pivmin) break;
    const double x = lo + (hi - lo) * (double)(tid + 1) * (1.0 / (IT_THREADS + 1));
    const bool in = (x > lo) && (x < hi), above = in && sturm_count(d, e, n, x, pivmin) >= 1;
    const unsigned ball = __ballot_sync(0xffffffffu, above);
    if (lane == 0) first[warp] = ball ? warp * 32 + __ffs(ball) - 1 : IT_THREADS;
    __syncthreads();
    int j = IT_THREADS;   // the lowest point with count >= 1
    for (int w = 0; w < IT_WARPS; ++w) j = min(j, first[w]);
    // the highest point under it with count 0 (points outside (lo, hi) by rounding are skipped)
    const unsigned below = __ballot_sync(0xffffffffu, in && !above && tid < j);
    if (lane == 0) under[warp] = below ? warp * 32 + 31 - __clz(below) : -1;
    __syncthreads();
    int i = -1;
    for (int w = 0; w < IT_WARPS; ++w) i = max(i, under[w]);
    if (tid == j) shi = x;
    if (tid == i) slo = x;
    __syncthreads();
    const double nhi = j < IT_THREADS ? shi : hi, nlo = i >= 0 ? slo : lo;
    __syncthreads();
    if (nhi >= hi && nlo <= lo) break;   // no representable progress
    lo = nlo;
    hi = nhi;
  }
  return 0.5 * (lo + hi);
}

// v(last+2) = y = H x, alpha_k = Re<x, y> with k = last + 1; then, in the last block,
// beta_(k-1) = sqrt(n2), res[0] = the lowest Ritz value of T_k (alpha_1..k, beta_1..k-1)
// and the packet {res[0], n2, alpha_k, |z_k|} (z, written when zbuf is not null, is that
// eigenvalue's unit eigenvector).
__global__ void __launch_bounds__(IT_THREADS) it_alpha_kernel(double2* __restrict__ V, long long ld,
                                                              const double2* __restrict__ x,
                                                              const double2* __restrict__ y, long long n,
                                                              const int* __restrict__ it, double* __restrict__ partial,
                                                              int* counter, const double* __restrict__ n2,
                                                              double* __restrict__ alpha, double* __restrict__ beta,
                                                              double* __restrict__ res, double* __restrict__ packet,
                                                              double* __restrict__ zbuf) {
  __shared__ double sd[IT_MAXVEC], se[IT_MAXVEC], red[IT_WARPS];
  const int k = *it + 1, tid = threadIdx.x;
  double2* next = V + (long long)k * ld;
  double acc = 0.0;
  for (long long e = (long long)blockIdx.x * IT_THREADS + tid; e < n; e += (long long)gridDim.x * IT_THREADS) {
    const double2 p = x[e], q = y[e];
    next[e] = q;
    acc = fma(p.x, q.x, acc);
    acc = fma(p.y, q.y, acc);
  }
  acc = block_sum(acc, red);
  if (tid == 0) partial[blockIdx.x] = acc;
  if (!last_block(counter) || k < 1 || k >= IT_MAXVEC) return;
  const double ak = partial_sum(partial), b = sqrt(*n2);
  for (int i = tid; i < k; i += IT_THREADS) {
    sd[i] = i + 1 == k ? ak : alpha[i + 1];
    se[i] = (i + 1 < k - 1) ? beta[i + 1] : (i + 1 == k - 1 ? b : 0.0);
  }
  __syncthreads();
  // with the vector its solver's own eigenvalue is taken, one search for both
  const double lam = zbuf ? 0.0 : tridiag_lowest_block(sd, se, k);
  if (tid >= 32) return;
  if (zbuf) tridiag_lowest_warp(sd, se, k, 1, res, zbuf);
  __syncwarp();
  if (tid == 0) {
    alpha[k] = ak;
    beta[k - 1] = b;
    if (!zbuf) res[0] = lam;
    packet[0] = res[0];
    packet[1] = *n2;
    packet[2] = ak;
    packet[3] = zbuf ? fabs(zbuf[k - 1]) : 0.0;
  }
}

inline int grid_for(long long n) {
  long long b = (n + VB - 1) / VB;
  if (b > 148 * 16) b = 148 * 16;
  if (b < 1) b = 1;
  return (int)b;
}

}  // namespace

template <int TM, int TN, int MINB, int LREGS, int CREGS, bool BULK>
cudaError_t launch_tile(const ZJob* jobs, int njobs, const GTerm* terms, Bases bases, int* next_job, int* fault,
                        int wait_limit, cudaStream_t st) {
  // what the halves hold is what the block was launched with: 65536 / (MINB * 256) a thread
  static_assert(LREGS + CREGS == 2 * (65536 / (MINB * 2 * GEMM_THREADS)), "register split");
  auto kernel = grouped_zgemm_kernel<TM, TN, MINB, LREGS, CREGS, BULK>;
  const int smem = ZTile<TM, TN, BULK>::SMEM;
  static std::atomic<unsigned long long> attr{0};
  cudaError_t e = ensure_smem_attr(kernel, smem, attr);
  if (e != cudaSuccess) return e;
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (nsm <= 0) nsm = 148;
  const int grid = njobs < nsm * MINB ? njobs : nsm * MINB;
  return launch_chained(kernel, grid, 2 * GEMM_THREADS, smem, st, jobs, njobs, terms, bases, next_job, fault,
                        wait_limit);
}

cudaError_t launch_grouped_zgemm(const ZJob* jobs, int njobs, const GTerm* terms, Bases bases, int* next_job,
                                 int* fault, int wait_limit, cudaStream_t st, int tile, bool bulk) {
  if (njobs <= 0) return cudaSuccess;
  if (tile == TILE_32x32)
    return launch_tile<32, 32, 4, 40, 88, false>(jobs, njobs, terms, bases, next_job, fault, wait_limit, st);
  if (!bulk) return launch_tile<64, 48, 2, 40, 216, false>(jobs, njobs, terms, bases, next_job, fault, wait_limit, st);
  if (!fault || wait_limit < 0) return cudaErrorInvalidValue;
  return launch_tile<64, 48, 2, 48, 208, true>(jobs, njobs, terms, bases, next_job, fault, wait_limit, st);
}

cudaError_t launch_grouped_axpy(const ZJob* jobs, int njobs, const GTerm* terms, Bases bases, cudaStream_t st) {
  if (njobs <= 0) return cudaSuccess;
  grouped_axpy_kernel<<<njobs, 256, 0, st>>>(jobs, terms, bases);
  return cudaGetLastError();
}

cudaError_t launch_reduce_partials(const GReduce* reds, int nred, const GGroup* groups, Bases bases,
                                   long long max_elems, cudaStream_t st) {
  if (nred <= 0) return cudaSuccess;
  long long bx = (max_elems + 255) / 256;
  if (bx > 64) bx = 64;
  if (bx < 1) bx = 1;
  dim3 grid((unsigned)bx, (unsigned)nred);
  return launch_chained(reduce_partials_kernel, grid, 256, 0, st, reds, groups, bases);
}

cudaError_t launch_multi_dot(const double2* X, long long ld, int nvec, const double2* y, long long n,
                             double* partial, double* out, cudaStream_t st) {
  if (nvec <= 0) return cudaSuccess;
  int nblk = (int)((n + VCHUNK - 1) / VCHUNK);
  if (nblk < 1) nblk = 1;
  multi_dot_partial<<<nblk, VB, 0, st>>>(X, ld, nvec, y, n, partial, nblk);
  multi_dot_final<<<nvec, 256, 0, st>>>(partial, nblk, nvec, out);
  return cudaGetLastError();
}

cudaError_t launch_zdot(const double2* x, const double2* y, long long n, double* partial, double* out,
                        cudaStream_t st) {
  int nblk = (int)((n + VCHUNK - 1) / VCHUNK);
  if (nblk < 1) nblk = 1;
  zdot_partial<<<nblk, VB, 0, st>>>(x, y, n, partial, nblk);
  multi_dot_final<<<2, 256, 0, st>>>(partial, nblk, 2, out);
  return cudaGetLastError();
}

cudaError_t launch_scale(double2* w, const double* norm2, long long n, int invert_sqrt, cudaStream_t st) {
  scale_kernel<<<grid_for(n), VB, 0, st>>>(w, norm2, n, invert_sqrt);
  return cudaGetLastError();
}

cudaError_t launch_combine(double2* out, const double2* X, long long ld, int nvec, const double* z, long long n,
                           cudaStream_t st) {
  combine_kernel<<<grid_for(n), VB, 0, st>>>(out, X, ld, nvec, z, n);
  return cudaGetLastError();
}

cudaError_t launch_phase_fix(double2* U, int rows, int cols, cudaStream_t st) {
  if (rows <= 0 || cols <= 0) return cudaSuccess;
  phase_fix_kernel<<<cols, 128, 0, st>>>(U, rows);
  return cudaGetLastError();
}

cudaError_t launch_tridiag_lowest(const double* d, const double* e, int n, int want_vec, double* res, double* z,
                                  cudaStream_t st) {
  if (n < 1 || n > 127) return cudaErrorInvalidValue;
  tridiag_lowest_kernel<<<1, 32, 0, st>>>(d, e, n, want_vec, res, z);
  return cudaGetLastError();
}

int it_blocks(long long n) {
  const long long b = (n + IT_THREADS - 1) / IT_THREADS;
  return (int)(b < 1 ? 1 : b > 148 * 4 ? 148 * 4 : b);
}

cudaError_t launch_it_project(double2* V, long long ld, const double* alpha, const double* beta, long long n,
                              const int* it, double* partial, int* counter, double* n2, double* uv, cudaStream_t st) {
  // a block's share in pieces of at most IT_SUB, in multiples of the block
  const int nb = it_blocks(n);
  long long sub = ((n + nb - 1) / nb + IT_THREADS - 1) / IT_THREADS * IT_THREADS;
  if (sub > IT_SUB) sub = IT_SUB;
  if (sub < IT_THREADS) sub = IT_THREADS;
  it_project_kernel<<<nb, IT_THREADS, 0, st>>>(V, ld, alpha, beta, n, (int)sub, it, partial, counter, n2, uv);
  return cudaGetLastError();
}

cudaError_t launch_it_orthogonalize(double2* V, long long ld, const double* n2, const double* uv, const double* uu,
                                    long long n, const int* it, double* partial, int* counter, double* nw2,
                                    cudaStream_t st) {
  it_orthogonalize_kernel<<<it_blocks(n), IT_THREADS, 0, st>>>(V, ld, n2, uv, uu, n, it, partial, counter, nw2);
  return cudaGetLastError();
}

cudaError_t launch_it_normalize(double2* V, long long ld, const double* nw2, long long n, const int* it, double2* x,
                                double* partial, int* counter, double* uu, cudaStream_t st) {
  it_normalize_kernel<<<it_blocks(n), IT_THREADS, 0, st>>>(V, ld, nw2, n, it, x, partial, counter, uu);
  return cudaGetLastError();
}

cudaError_t launch_it_alpha(double2* V, long long ld, const double2* x, const double2* y, long long n, const int* it,
                            double* partial, int* counter, const double* n2, double* alpha, double* beta, double* res,
                            double* packet, double* zbuf, cudaStream_t st) {
  it_alpha_kernel<<<it_blocks(n), IT_THREADS, 0, st>>>(V, ld, x, y, n, it, partial, counter, n2, alpha, beta, res,
                                                       packet, zbuf);
  return cudaGetLastError();
}

}  // namespace tsc
