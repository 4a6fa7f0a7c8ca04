// Host set-up of the engine: device memory, lattice tables, SU(2) 6j symbols,
// site operators, bases and task-list packing.
#include <algorithm>
#include <array>
#include <chrono>
#include <climits>
#include <cmath>
#include <cstdlib>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <queue>
#include <set>
#include <tuple>
#include <unordered_map>
#include <vector>

#include "../../include/tsc_gpu.h"
#include "tsc_engine.hpp"

namespace tsc {

std::shared_mutex& capture_mutex() {
  static std::shared_mutex m;
  return m;
}

void cuda_check(cudaError_t e, const char* what) {
  if (e != cudaSuccess) throw Error(e == cudaErrorMemoryAllocation ? -5 : -3,
                                    std::string(what) + ": " + cudaGetErrorString(e));
}

// One stream-ordered pool per device that keeps freed memory for reuse (the
// default pool hands it back to the driver at every synchronisation, so each
// DMRG step would map its Krylov space and task buffers afresh).  Engines trim
// it when they are destroyed.
static std::mutex g_pool_mu;
static cudaMemPool_t g_pools[256] = {};

cudaMemPool_t device_pool() {
  int dev = 0;
  cuda_check(cudaGetDevice(&dev), "cudaGetDevice");
  if (dev < 0 || dev >= 256) throw Error(-1, "device ordinal out of range");
  std::lock_guard<std::mutex> lock(g_pool_mu);
  if (!g_pools[dev]) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    cuda_check(cudaMemPoolCreate(&pool, &props), "cudaMemPoolCreate");
    uint64_t keep = UINT64_MAX;
    cuda_check(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep), "cudaMemPoolSetAttribute");
    g_pools[dev] = pool;
  }
  return g_pools[dev];
}

namespace {
// Per-stream arena: chunks from the device pool, carved best fit, freed blocks
// coalesced with their neighbours inside a chunk.  All blocks of one arena are
// used in the order of its stream, so a block freed by the host can be handed
// out again at once.
struct Arena {
  struct Chunk {
    char* base;
    size_t bytes;
  };
  std::vector<Chunk> chunks;
  std::map<char*, size_t> free_at;             // block start -> bytes
  std::multimap<size_t, char*> free_size;      // bytes -> block start
  std::map<char*, char*> chunk_end;            // chunk base -> one past its end
  size_t reserved = 0;

  void insert_free(char* p, size_t n) {
    free_at[p] = n;
    free_size.emplace(n, p);
  }
  void erase_free(std::map<char*, size_t>::iterator it) {
    auto r = free_size.equal_range(it->second);
    for (auto q = r.first; q != r.second; ++q)
      if (q->second == it->first) {
        free_size.erase(q);
        break;
      }
    free_at.erase(it);
  }
  char* chunk_limit(char* p) const {   // end of the chunk holding p
    auto it = chunk_end.upper_bound(p);
    --it;
    return it->second;
  }
  char* take(size_t n) {
    auto it = free_size.lower_bound(n);
    if (it == free_size.end()) return nullptr;
    char* p = it->second;
    size_t have = it->first;
    free_size.erase(it);
    free_at.erase(p);
    if (have > n) insert_free(p + n, have - n);
    return p;
  }
  void give(char* p, size_t n) {
    char* lim = chunk_limit(p);
    auto nx = free_at.find(p + n);   // merge with the following free block
    if (nx != free_at.end() && p + n < lim) {
      n += nx->second;
      erase_free(nx);
    }
    auto pv = free_at.lower_bound(p);   // and with the preceding one
    if (pv != free_at.begin()) {
      --pv;
      if (pv->first + pv->second == p && chunk_limit(pv->first) == lim) {
        p = pv->first;
        n += pv->second;
        erase_free(pv);
      }
    }
    insert_free(p, n);
  }
};
std::mutex g_arena_mu;
std::unordered_map<cudaStream_t, Arena> g_arena;

constexpr size_t kAlign = 256;
constexpr size_t kMinChunk = 64ull << 20;
constexpr size_t kMaxChunk = 4ull << 30;
constexpr size_t kDirect = 4ull << 30;   // blocks at least this large bypass the arenas
}  // namespace

void release_stream_cache(cudaStream_t s) {
  std::lock_guard<std::mutex> lock(g_arena_mu);
  auto it = g_arena.find(s);
  if (it == g_arena.end()) return;
  for (auto& c : it->second.chunks) cudaFreeAsync(c.base, s);
  g_arena.erase(it);
}

DevBuf::DevBuf(size_t count, cudaStream_t s, bool zero) : n(count), st(s) {
  if (count == 0) return;
  cls = (count * sizeof(double2) + kAlign - 1) / kAlign * kAlign;
  if (cls >= kDirect) {   // large blocks come straight from the pool, which reuses them across sizes
    cuda_check(cudaMallocFromPoolAsync((void**)&p, cls, device_pool(), s), "cudaMallocFromPoolAsync");
    direct = true;
  } else {
    std::lock_guard<std::mutex> lock(g_arena_mu);
    Arena& A = g_arena[s];
    char* q = A.take(cls);
    if (!q) {   // new chunk: geometric growth between 64 MiB and 4 GiB, at least the request
      size_t want = std::max(cls, std::min(kMaxChunk, std::max(kMinChunk, A.reserved / 2)));
      void* base = nullptr;
      cudaError_t e = cudaMallocFromPoolAsync(&base, want, device_pool(), s);
      if (e == cudaErrorMemoryAllocation && want > cls) {   // fall back to the exact request
        cudaGetLastError();
        want = cls;
        e = cudaMallocFromPoolAsync(&base, want, device_pool(), s);
      }
      cuda_check(e, "cudaMallocFromPoolAsync");
      A.chunks.push_back({static_cast<char*>(base), want});
      A.chunk_end[static_cast<char*>(base)] = static_cast<char*>(base) + want;
      A.reserved += want;
      A.insert_free(static_cast<char*>(base), want);
      q = A.take(cls);
    }
    p = reinterpret_cast<double2*>(q);
  }
  if (zero) cuda_check(cudaMemsetAsync(p, 0, count * sizeof(double2), s), "cudaMemsetAsync");
}
DevBuf::~DevBuf() {
  if (!p) return;
  if (direct) {
    cudaFreeAsync(p, st);
    return;
  }
  std::lock_guard<std::mutex> lock(g_arena_mu);
  auto it = g_arena.find(st);
  if (it != g_arena.end()) it->second.give(reinterpret_cast<char*>(p), cls);
}

// ---- SU(2) coefficients --------------------------------------------------------
// Racah's closed form for the 6j symbol with doubled arguments (the reference's
// W6JS, block.f90:3744-3795, evaluates the same sum with a table of factorials).
// factorials as FACTRL builds them (block.f90:3688-3696); initialised once,
// thread-safely, by the first caller of any engine
static const double* factorials() {
  static const std::array<double, 171> f = [] {
    std::array<double, 171> a{};
    a[0] = 1.0;
    for (int i = 1; i <= 170; ++i) a[i] = a[i - 1] * (double)(float)i;
    return a;
  }();
  return f.data();
}

double w6j(int j1, int j2, int j3, int l1, int l2, int l3) {
  const double* g_fact = factorials();
  // triangle (j1 j2 j3), (j1 l2 l3), (l1 j2 l3), (l1 l2 j3) with integer sums
  auto tri = [](int a, int b, int c) { return c <= a + b && c >= std::abs(a - b) && ((a + b + c) & 1) == 0; };
  if (!tri(j1, j2, j3) || !tri(j1, l2, l3) || !tri(l1, j2, l3) || !tri(l1, l2, j3)) return 0.0;
  const int s1 = j1 + j2 + j3, s2 = j1 + l2 + l3, s3 = l1 + j2 + l3, s4 = l1 + l2 + j3;
  const int p1 = j1 + j2 + l1 + l2, p2 = j2 + j3 + l2 + l3, p3 = j3 + j1 + l3 + l1;
  const int wlo = std::max(std::max(s1, s2), std::max(s3, s4));
  const int whi = std::min(p1, std::min(p2, p3));
  double omega = 0.0;
  for (int w = wlo; w <= whi; w += 2) {
    double den = g_fact[(w - s1) / 2] * g_fact[(w - s2) / 2] * g_fact[(w - s3) / 2] * g_fact[(w - s4) / 2] *
                 g_fact[(p1 - w) / 2] * g_fact[(p2 - w) / 2] * g_fact[(p3 - w) / 2];
    if (w % 4 != 0) den = -den;
    omega = omega + g_fact[w / 2 + 1] / den;
  }
  auto delta = [g_fact](int a, int b, int c) {
    return g_fact[(a + b - c) / 2] * g_fact[(a - b + c) / 2] * g_fact[(-a + b + c) / 2] / g_fact[(a + b + c) / 2 + 1];
  };
  double th = delta(j1, j2, j3) * delta(j1, l2, l3) * delta(l1, j2, l3) * delta(l1, l2, j3);
  return omega * std::sqrt(th);
}

// Wigner 3j symbol with doubled arguments by Racah's single-sum formula
// (the reference's W3JS, block.f90:3702-3741, evaluates the same sum):
// (-1)^(j1-j2-m3) sqrt(D(j1 j2 j3) prod (j+-m)!) sum_k (-1)^k / [k! (j3-j2+m1+k)!
// (j3-j1-m2+k)! (j1+j2-j3-k)! (j1-m1-k)! (j2+m2-k)!]
double w3j(int j1, int j2, int j3, int m1, int m2, int m3) {
  const double* f = factorials();
  if (m1 + m2 + m3 != 0) return 0.0;
  if (j3 > j1 + j2 || j3 < std::abs(j1 - j2)) return 0.0;
  if (((j1 + j2 + j3) & 1) || ((j1 - m1) & 1) || ((j2 - m2) & 1)) return 0.0;
  if (std::abs(m1) > j1 || std::abs(m2) > j2 || std::abs(m3) > j3) return 0.0;
  // k in doubled units
  const int klo = std::max(0, std::max(j2 - j3 - m1, j1 - j3 + m2));
  const int khi = std::min(j1 + j2 - j3, std::min(j1 - m1, j2 + m2));
  double sum = 0.0;
  for (int k = klo; k <= khi; k += 2) {
    double den = f[k / 2] * f[(j3 - j2 + m1 + k) / 2] * f[(j3 - j1 - m2 + k) / 2] * f[(j1 + j2 - j3 - k) / 2] *
                 f[(j1 - m1 - k) / 2] * f[(j2 + m2 - k) / 2];
    sum += (k % 4 == 0) ? 1.0 / den : -1.0 / den;
  }
  const double tri = f[(j1 + j2 - j3) / 2] * f[(j1 - j2 + j3) / 2] * f[(-j1 + j2 + j3) / 2] / f[(j1 + j2 + j3) / 2 + 1];
  const double mf = f[(j1 + m1) / 2] * f[(j1 - m1) / 2] * f[(j2 + m2) / 2] * f[(j2 - m2) / 2] * f[(j3 + m3) / 2] *
                    f[(j3 - m3) / 2];
  const double v = sum * std::sqrt(tri * mf);
  return (((j1 - j2 - m3) / 2) % 2 != 0) ? -v : v;
}

// ---- lattice (dmrg_sub.f90:304-644) -------------------------------------------------
void Lattice::init(int nx, int ny, double t1, double t2, double J1, double J2, int oy) {
  Nx = nx;
  Ny = ny;
  nleg = ny;
  num_site = nx * ny;
  openy = oy;
  int N = num_site;
  neib.assign((size_t)(N + 1) * (neibt + 1), 0);
  neiba.assign((size_t)(N + 1) * (N + 1), 0);
  nposi.assign(N + 8, 0);
  nposi_dm.assign(N + 8, 0);
  nposi_lat.assign(N + 8, 0);
  inb1.assign((size_t)(N + 1) * (N + 1), 0);
  nleg11.assign(N + 1, 0);
  inb.assign(N + 8, 0);
  size_t nc = (size_t)(N + 1) * (neibt + 1);
  jt.assign(nc, 0.0);
  jz.assign(nc, 0.0);
  jd.assign(nc, 0.0);
  jn.assign(nc, 0.0);
  for (int s = 1; s <= N; ++s) {
    for (int k = 1; k <= 12; ++k) {
      size_t e = (size_t)s * (neibt + 1) + k;
      jz[e] = k <= 6 ? J1 : J2;
      jt[e] = -(k <= 6 ? t1 : t2) * std::sqrt(2.0);
      jn[e] = -0.25 * jz[e];
    }
    for (int k = 1; k <= 18; ++k) {
      size_t e = (size_t)s * (neibt + 1) + k;
      jd[e] = jz[e] * (-std::sqrt(3.0));
    }
  }
}

void Lattice::setup(int ns, int ns21) {
  int nn = ns + ns21 + 2;
  nxc = (nn - 1) / nleg + 1;
  if (nxc == 1) nxc = 2;
  std::fill(nposi.begin(), nposi.end(), 0);
  std::fill(nposi_dm.begin(), nposi_dm.end(), 0);
  std::fill(nposi_lat.begin(), nposi_lat.end(), 0);
  std::fill(neib.begin(), neib.end(), 0);
  std::fill(neiba.begin(), neiba.end(), 0);
  int totsite = nleg * nxc;
  for (int i = 1; i <= ns + 1; ++i) {
    nposi[i] = 1;
    nposi_lat[i] = i;
    nposi_dm[i] = i;
  }
  nposi[ns + 1] = 2;
  for (int i = 1; i <= ns21 + 1; ++i) {
    nposi[ns + 1 + i] = 3;
    nposi_dm[totsite + 1 - i] = i + ns + 1;
    nposi_lat[i + ns + 1] = totsite + 1 - i;
  }
  nposi[ns + ns21 + 2] = 4;
  auto link = [&](int a, int ka, int b, int kb) {
    NEIB(a, ka) = b;
    NEIB(b, kb) = a;
    NEIBA(a, b) = ka;
    NEIBA(b, a) = kb;
  };
  for (int ix = 1; ix <= nxc; ++ix)
    for (int iy = 1; iy <= nleg; ++iy) {
      int ii = iy + (ix - 1) * nleg;
      int jy = ii - iy + (iy % nleg) + 1;
      if (openy != 0 && iy == nleg) jy = 0;
      if (jy != 0 && (iy != nleg || nleg != 2)) link(ii, 1, jy, 2);
      int jx = ii + nleg;
      if (jx > nleg * nxc) jx = 0;   // open in x
      if (jx != 0) {
        link(ii, 3, jx, 4);
        jy = jx - 1;
        if (iy == 1) jy = openy == 0 ? jy + nleg : 0;
        if (jy != 0) link(ii, 5, jy, 6);
      }
    }
  for (int ix = 1; ix <= nxc; ++ix)
    for (int iy = 1; iy <= nleg; ++iy) {
      int ii = iy + (ix - 1) * nleg;
      int a = NEIB(ii, 1), b = NEIB(a, 3);
      if (a * b != 0) link(ii, 7, b, 8);
      if (nleg != 3) {
        a = NEIB(ii, 3);
        b = NEIB(a, 5);
        if (a * b != 0) link(ii, 9, b, 10);
      }
      a = NEIB(ii, 2);
      b = NEIB(a, 5);
      if (a * b != 0) link(ii, 11, b, 12);
      if (nleg != 3) {
        a = NEIB(ii, 1);
        b = NEIB(a, 1);
        if (a * b != 0 && NEIBA(ii, b) == 0) link(ii, 13, b, 14);
      }
      a = NEIB(ii, 3);
      b = NEIB(a, 3);
      if (a * b != 0 && NEIBA(ii, b) == 0) link(ii, 15, b, 16);
      a = NEIB(ii, 5);
      b = NEIB(a, 5);
      if (a * b != 0 && NEIBA(ii, b) == 0) link(ii, 17, b, 18);
    }
  for (int i = 1; i <= num_site; ++i)
    for (int j = 7; j <= neibt; ++j)
      if (std::fabs(JZ(j, 1)) + std::fabs(JD(j, 1)) + std::fabs(JT(j, 1)) + std::fabs(JN(j, 1)) == 0.0) {
        int nb = NEIB(i, j);
        NEIBA(i, nb) = 0;
        NEIBA(nb, i) = 0;
        NEIB(i, j) = 0;
      }
}

void Lattice::setup0() {
  std::fill(nleg11.begin(), nleg11.end(), 0);
  for (int ns = 1; ns <= num_site - 2; ++ns) {
    int k0 = 0;
    for (int i1 = 1; i1 <= ns; ++i1) {
      int cnt = 0;
      for (int j = 1; j <= neibt; ++j)
        if (NEIB(i1, j) >= ns) cnt++;
      INB1(i1, ns) = cnt ? ++k0 : 10000;
    }
    nleg11[ns] = k0;
  }
}

// ---- engine -------------------------------------------------------------------------
Engine::Engine(int Nx, int Ny, double t1, double t2, double J1, double J2, int delta, int device) {
  std::unique_lock<std::shared_mutex> no_capture(capture_mutex());
  if (Nx < 2 || Ny < 2 || Nx * Ny > 1024) throw Error(-1, "lattice size out of range");
  if (delta < 1) throw Error(-1, "delta must be >= 1");
  int ndev = 0;
  cuda_check(cudaGetDeviceCount(&ndev), "cudaGetDeviceCount");
  if (device < 0 || device >= ndev) throw Error(-1, "no such CUDA device");
  cuda_check(cudaSetDevice(device), "cudaSetDevice");
  device_ = device;
  cuda_check(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking), "cudaStreamCreate");
  cuda_check(cudaEventCreate(&ev0), "cudaEventCreate");
  cuda_check(cudaEventCreate(&ev1), "cudaEventCreate");
  models_.bind(st);
  L.init(Nx, Ny, t1, t2, J1, J2, 0);
  // site operators (dmrg_sub.f90:743-906)
  st_elec_up.up_dif = 1;
  st_elec_up.down_dif = 1;
  st_elec_up.sub = {{0, 0, 1, -std::sqrt(2.0)}};
  st_elec_down.up_dif = -1;
  st_elec_down.down_dif = 1;
  st_elec_down.sub = {{1, 1, -1, -std::sqrt(2.0)}};
  num_elec.sub = {{1, 1, 0, std::sqrt(2.0)}, {0, 0, 0, 0.0}};
  st_sd.down_dif = 2;
  st_sd.sub = {{1, 1, 0, std::sqrt(1.5)}};
  st_sz.sub = {{1, 1, 0, 1.0}, {0, 0, 0, 0.0}};
  int N = L.num_site;
  tot_num_up = 2 * (N / 2 - (N + 2 * delta - 1) / (2 * delta));
  tot_num_down = 0;
  L.setup(N / 2 - 1, N / 2 - 1);
  L.setup0();
  red_buf = std::make_shared<DevBuf>((size_t)(1 << 16) + 1024, st, true);
  d_red = reinterpret_cast<double*>(red_buf->p);
  d_scal = d_red + (1 << 16);
  d_fault = reinterpret_cast<int*>(d_scal + S_FAULT);   // zero: red_buf is zero-filled
  cuda_check(cudaMallocHost((void**)&h_scal, 2048 * sizeof(double)), "cudaMallocHost");
}

void Engine::check_waits(bool earlier) {
  if (!waits_unread_) return;
  cuda_check(cudaMemcpyAsync(h_scal + S_FAULT, d_fault, sizeof(int), cudaMemcpyDeviceToHost, st), "d2h");
  cuda_check(cudaStreamSynchronize(st), "sync");
  waits_unread_ = false;
  int f = 0;
  std::memcpy(&f, h_scal + S_FAULT, sizeof(int));
  if (!f) return;
  cuda_check(cudaMemsetAsync(d_fault, 0, sizeof(int), st), "memset");
  cuda_check(cudaStreamSynchronize(st), "sync");
  throw Error(-3, std::string(earlier ? "an earlier call that does not wait for its launches: " : "") +
                      (f & FAULT_SPLIT ? "split-precision" : "FP64") +
                      " kernel: a bounded wait ran out (output incomplete)");
}

Engine::~Engine() {
  std::unique_lock<std::shared_mutex> no_capture(capture_mutex());
  sb = Superblock();
  bs = BlockSparse();
  models_.clear();
  sys_truns.clear();
  env_truns.clear();
  disk_wave.reset();
  red_buf.reset();
  eig.reset();
  release_stream_cache(st);
  if (st) cudaStreamSynchronize(st);
  try {
    cudaMemPoolTrimTo(device_pool(), 0);
  } catch (...) {
  }
  if (h_scal) cudaFreeHost(h_scal);
  if (graph_exec_) cudaGraphExecDestroy(graph_exec_);
  for (cudaEvent_t e : graph_ev_)
    if (e) cudaEventDestroy(e);
  if (ev0) cudaEventDestroy(ev0);
  if (ev1) cudaEventDestroy(ev1);
  for (cudaEvent_t e : hpsi_events) cudaEventDestroy(e);
  for (cudaEvent_t e : tune_ev_)
    if (e) cudaEventDestroy(e);
  if (st) cudaStreamDestroy(st);
}

DModel Engine::site_model() const {   // Get_hamiltonian_site, dmrg_sub.f90:912-938
  DModel m;
  m.len = 1;
  auto mk = [&](const SiteOp& so, int nsub_override_zero) {
    DBlock b;
    b.len = 1;
    b.num = (int)so.sub.size();
    b.dim = b.num;
    b.up_dif = so.up_dif;
    b.down_dif = so.down_dif;
    b.buf = std::make_shared<DevBuf>((size_t)b.num, st, false);
    std::vector<double2> h(b.num);
    for (int i = 0; i < b.num; ++i) {
      SubDesc s;
      s.num_up = so.sub[i].num_up;
      s.num_down = so.sub[i].num_down;
      s.down_dif = so.sub[i].down_dif;
      s.row_dim = s.sdim = 1;
      s.off = i;
      b.sub.push_back(s);
      h[i] = make_double2(nsub_override_zero ? 0.0 : so.sub[i].val, 0.0);
    }
    cuda_check(cudaMemcpyAsync(b.buf->p, h.data(), b.num * sizeof(double2), cudaMemcpyHostToDevice, st), "upload");
    cuda_check(cudaStreamSynchronize(st), "sync");
    return b;
  };
  m.ham = mk(st_sz, 1);
  m.sub.resize(L.num_site + 1);
  m.sub[1].op[OP_UP] = mk(st_elec_up, 0);
  m.sub[1].op[OP_DOWN] = mk(st_elec_down, 0);
  m.sub[1].op[OP_SD] = mk(st_sd, 0);
  m.sub[1].op[OP_SN] = mk(num_elec, 0);
  return m;
}

// Get_basis, block.f90:2087-2188 (site = st_sz: (1,1) then (0,0), sdim 1)
Basis Engine::get_basis(const DBlock& block) const {
  Basis b;
  b.len = block.len + 1;
  std::vector<std::pair<int, int>> q;   // (N, 2S)
  for (const auto& s : block.sub)
    for (const auto& t : st_sz.sub)
      for (int ss = std::abs(s.num_down - t.num_down); ss <= s.num_down + t.num_down; ss += 2)
        q.push_back({s.num_up + t.num_up, ss});
  // descending 2S, then descending N (QuickSort_Integer, block.f90:2316-2349), unique
  std::sort(q.begin(), q.end(), [](const std::pair<int, int>& a, const std::pair<int, int>& c) {
    if (a.second != c.second) return a.second > c.second;
    return a.first > c.first;
  });
  q.erase(std::unique(q.begin(), q.end()), q.end());
  b.num = (int)q.size();
  b.sec.resize(b.num);
  for (int i = 0; i < b.num; ++i) {
    Sector& S = b.sec[i];
    S.num_up = q[i].first;
    S.num_down = q[i].second;
    for (const auto& s : block.sub)
      for (const auto& t : st_sz.sub) {
        if (s.num_up + t.num_up != S.num_up) continue;
        if (S.num_down < std::abs(s.num_down - t.num_down) || S.num_down > s.num_down + t.num_down) continue;
        Piece p;
        p.bl_num_up = s.num_up;
        p.bl_num_down = s.num_down;
        p.st_num_up = t.num_up;
        p.st_num_down = t.num_down;
        p.sdim = s.sdim;
        p.spos = S.dim;
        S.dim += p.sdim;
        S.pcs.push_back(p);
      }
    b.dim += S.dim;
  }
  return b;
}

// Get_super_basis, block.f90:2194-2247
WLayout Engine::get_super(const Basis& sys_bs, const Basis& env_bs, int tot_up, int tot_down) const {
  WLayout w;
  w.sys_len = sys_bs.len;
  w.env_len = env_bs.len;
  for (const auto& s : sys_bs.sec)
    for (const auto& e : env_bs.sec) {
      if (e.num_up != tot_up - s.num_up) continue;
      if (tot_down < std::abs(e.num_down - s.num_down) || tot_down > e.num_down + s.num_down) continue;
      WSec x;
      x.sys_num_up = s.num_up;
      x.sys_num_down = s.num_down;
      x.env_num_up = e.num_up;
      x.env_num_down = e.num_down;
      x.sys_dim = s.dim;
      x.env_dim = e.dim;
      x.off = w.dim;
      w.dim += (long long)s.dim * e.dim;
      w.sec.push_back(x);
    }
  w.num = (int)w.sec.size();
  return w;
}

// ---- task lists ------------------------------------------------------------------------
int TaskList::add_group(double2* abs_c, uint8_t base, long long c_off, int ld, int M, int N, int beta) {
  GGroup g{};
  g.c_base = base;
  g.c_off = base == BASE_ABS ? (long long)((uintptr_t)abs_c / sizeof(double2)) + c_off : c_off;
  g.c_ld = ld;
  g.M = M;
  g.N = N;
  g.beta = (uint8_t)beta;
  groups.push_back(g);
  gterms.emplace_back();
  return (int)groups.size() - 1;
}

// ---- split-precision form: pre-sliced operand views ----------------------------------
namespace {
struct ViewKey {
  uint8_t base, op, role;
  long long off;
  int ld, rows, cols;
  double ar, ai;
  bool operator<(const ViewKey& o) const {
    return std::tie(base, op, role, off, ld, rows, cols, ar, ai) <
           std::tie(o.base, o.op, o.role, o.off, o.ld, o.rows, o.cols, o.ar, o.ai);
  }
};
int view_tiles_along(const SView& v) {   // row tiles (A) or column tiles (B)
  return v.role == 0 ? (v.rows + SPLIT_TILE_M - 1) / SPLIT_TILE_M : (v.cols + SPLIT_TILE_N - 1) / SPLIT_TILE_N;
}
long long view_units(const SView& v) { return (long long)view_tiles_along(v) * v.nks * (v.role == 0 ? SPLIT_A_UNITS : SPLIT_B_UNITS); }
int view_steps(const ViewKey& k) { return ((k.role == 0 ? k.cols : k.rows) + GEMM_TK - 1) / GEMM_TK; }
// The views of a GEMM term's left and right operand.  The term's coefficient rides on the
// operator operand (on the left one when both are operators), or stays with the term (term_alpha).
std::pair<ViewKey, ViewKey> term_views(const GGroup& g, const GTerm& t, bool term_alpha) {
  const bool fold_a = t.l_base == BASE_ABS;
  const double cr = term_alpha ? 1.0 : t.ar, ci = term_alpha ? 0.0 : t.ai;
  return {ViewKey{t.l_base, t.l_op, 0, t.l_off, t.l_ld, g.M, t.K, fold_a ? cr : 1.0, fold_a ? ci : 0.0},
          ViewKey{t.r_base, t.r_op, 1, t.r_off, t.r_ld, t.K, g.N, fold_a ? 1.0 : cr, fold_a ? 0.0 : ci}};
}
}  // namespace

long long operator_view_bytes(const TaskList& p1, const TaskList& p2, bool term_alpha) {
  std::set<ViewKey> seen;
  long long units = 0;
  for (const TaskList* tl : {&p1, &p2})
    for (size_t gi = 0; gi < tl->groups.size(); ++gi)
      for (const GTerm& t : tl->gterms[gi]) {
        if (t.kind != TK_GEMM || t.K <= 0) continue;
        const auto [a, b] = term_views(tl->groups[gi], t, term_alpha);
        for (const ViewKey& k : {a, b}) {
          if (k.base != BASE_ABS || !seen.insert(k).second) continue;
          SView v{};
          v.rows = k.rows;
          v.cols = k.cols;
          v.role = k.role;
          v.nks = view_steps(k);
          units += view_units(v);
        }
      }
  return units * (long long)SPLIT_UNIT;
}

void build_split_views(TaskList& p1, TaskList& p2, SplitData& sd, cudaStream_t st, bool term_alpha) {
  sd = SplitData();
  std::vector<SView> views[3];
  std::map<ViewKey, int> index[3];
  // phase-1 groups by their scratch offset: the intermediates phase 2 reads
  std::map<long long, int> scr_group;
  for (size_t g = 0; g < p1.groups.size(); ++g)
    if (p1.groups[g].c_base == BASE_SCR) scr_group[p1.groups[g].c_off] = (int)g;
  std::map<int, int> tview_of_group;
  auto add_view = [&](int arena, const ViewKey& k) -> int {
    auto it = index[arena].find(k);
    if (it != index[arena].end()) return it->second;
    SView v{};
    v.src = k.off;
    v.ar = k.ar;
    v.ai = k.ai;
    v.ld = k.ld;
    v.rows = k.rows;
    v.cols = k.cols;
    v.role = k.role;
    v.op = k.op;
    v.from_in = arena == ARENA_IN;
    v.nks = view_steps(k);
    v.dst = sd.units[arena];
    sd.units[arena] += view_units(v);
    views[arena].push_back(v);
    return index[arena][k] = (int)views[arena].size() - 1;
  };
  // the view of one operand of a term; returns (arena, view)
  auto operand = [&](const ViewKey& k) -> std::pair<int, int> {
    if (k.base == BASE_ABS) return {ARENA_FIXED, add_view(ARENA_FIXED, k)};
    if (k.ar != 1.0 || k.ai != 0.0) throw Error(-1, "split views: coefficient on a live operand");
    if (k.base == BASE_IN) return {ARENA_IN, add_view(ARENA_IN, k)};
    if (k.base == BASE_SCR) {
      auto it = scr_group.find(k.off);
      if (it == scr_group.end() || k.role != 0 || k.op != OP_N) throw Error(-1, "split views: unexpected scratch operand");
      GGroup& g = p1.groups[it->second];
      if (g.M != k.rows || g.c_ld != k.ld || g.N != k.cols || p1.gterms[it->second].size() != 1)
        throw Error(-1, "split views: scratch operand is not a whole phase-1 output");
      auto tv = tview_of_group.find(it->second);
      if (tv != tview_of_group.end()) return {ARENA_T, tv->second};
      const int v = add_view(ARENA_T, k);
      g.s_off = views[ARENA_T][v].dst;
      tview_of_group[it->second] = v;
      return {ARENA_T, v};
    }
    throw Error(-1, "split views: operand base");
  };
  for (TaskList* tl : {&p1, &p2})
    for (size_t gi = 0; gi < tl->groups.size(); ++gi) {
      const GGroup& g = tl->groups[gi];
      for (GTerm& t : tl->gterms[gi]) {
        if (t.kind != TK_GEMM || t.K <= 0) continue;
        const auto [ka, kb] = term_views(g, t, term_alpha);
        const auto A = operand(ka), B = operand(kb);
        const SView& va = views[A.first][A.second];
        const SView& vb = views[B.first][B.second];
        t.l_base = (uint8_t)A.first;
        t.l_off = va.dst;
        t.l_ld = va.nks;
        t.r_base = (uint8_t)B.first;
        t.r_off = vb.dst;
        t.r_ld = vb.nks;
        t.l_op = t.r_op = OP_N;
        if (!term_alpha) {
          t.ar = 1.0;
          t.ai = 0.0;
        }
        t.pad0 = 1;   // references pre-sliced views
      }
    }
  // arenas; intermediates' tiles start zeroed (their padding is never written)
  DevBufP* arena[3] = {&sd.fixed, &sd.in, &sd.t};
  for (int a = 0; a < 3; ++a) {
    const long long bytes = std::max<long long>(sd.units[a], 1) * SPLIT_UNIT;
    *arena[a] = std::make_shared<DevBuf>((size_t)(bytes / sizeof(double2)), st, a == ARENA_T);
    sd.arenas.a[a] = reinterpret_cast<unsigned char*>((*arena[a])->p);
    sd.arenas.units[a] = std::max<long long>(sd.units[a], 1);
    sd.nviews[a] = (int)views[a].size();
  }
  auto tiles_of = [&](const std::vector<SView>& vs) {
    std::vector<STile> tl;
    for (size_t v = 0; v < vs.size(); ++v)
      for (int t = 0; t < view_tiles_along(vs[v]); ++t)
        for (int ks = 0; ks < vs[v].nks; ++ks) tl.push_back(STile{(int)v, t, ks, 0});
    return tl;
  };
  auto pack = [&](const std::vector<SView>& vs, const std::vector<STile>& tl, DevBufP& buf, const SView*& dv,
                  const STile*& dt) {
    const size_t bv = (vs.size() * sizeof(SView) + 255) / 256 * 256, bt = tl.size() * sizeof(STile);
    buf = std::make_shared<DevBuf>((bv + bt + 15) / 16 + 1, st, false);
    std::vector<char> host(bv + bt, 0);
    if (!vs.empty()) std::memcpy(host.data(), vs.data(), vs.size() * sizeof(SView));
    if (bt) std::memcpy(host.data() + bv, tl.data(), bt);
    cuda_check(cudaMemcpyAsync(buf->p, host.data(), host.size(), cudaMemcpyHostToDevice, st), "split views upload");
    dv = reinterpret_cast<const SView*>(buf->p);
    dt = reinterpret_cast<const STile*>(reinterpret_cast<char*>(buf->p) + bv);
    cuda_check(cudaStreamSynchronize(st), "split views sync");   // the host staging buffer goes out of scope
  };
  {  // operator views: sliced once, here
    std::vector<STile> tl = tiles_of(views[ARENA_FIXED]);
    DevBufP tmp;
    const SView* dv = nullptr;
    const STile* dt = nullptr;
    pack(views[ARENA_FIXED], tl, tmp, dv, dt);
    cuda_check(launch_slice_tiles(dv, dt, (int)tl.size(), nullptr, sd.arenas.a[ARENA_FIXED],
                                  sd.arenas.units[ARENA_FIXED], st),
               "slice operators");
    cuda_check(cudaStreamSynchronize(st), "slice operators sync");
  }
  std::vector<STile> tin = tiles_of(views[ARENA_IN]);
  pack(views[ARENA_IN], tin, sd.in_lists, sd.d_in_views, sd.d_in_tiles);
  sd.n_in_tiles = (int)tin.size();
  p1.arenas = p2.arenas = sd.arenas;
  p1.term_alpha = p2.term_alpha = term_alpha;
}

void slice_input(const SplitData& sd, const double2* d_in, cudaStream_t st) {
  cuda_check(launch_slice_tiles(sd.d_in_views, sd.d_in_tiles, sd.n_in_tiles, d_in, sd.arenas.a[ARENA_IN],
                                sd.arenas.units[ARENA_IN], st),
             "slice input");
}

void TaskList::upload_split(cudaStream_t st) {
  split = true;
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  upload(st, (nsm > 0 ? nsm : 148) * 2, 4);   // one CTA per SM
}

// Elements of the partial tiles when the terms, in the order built, are cut into chunks of
// K steps for 4 waves of 888 CTAs with 32x32 tiles (split form: 296 with 128x64).  The
// schedule that the no-allocation entry's limit is stated for: what fits with it is taken,
// whatever schedule a list is run with.
long long TaskList::basic_part_elems() const {
  const int TMt = split ? SPLIT_TILE_M : 32, TNt = split ? SPLIT_TILE_N : 32;
  auto cost = [](const GTerm& t) -> long long { return t.kind == TK_GEMM ? (t.K + GEMM_TK - 1) / GEMM_TK + 1 : 1; };
  std::vector<long long> gcost(groups.size(), 1);
  long long total = 0, elems = 0;
  for (size_t gi = 0; gi < groups.size(); ++gi) {
    const GGroup& g = groups[gi];
    for (const GTerm& t : gterms[gi]) gcost[gi] += cost(t);
    if (g.M > 0 && g.N > 0) total += gcost[gi] * ((g.M + TMt - 1) / TMt) * ((g.N + TNt - 1) / TNt);
  }
  const long long target = std::max<long long>(8, total / (4 * (split ? 296 : 888)));
  for (size_t gi = 0; gi < groups.size(); ++gi) {
    const GGroup& g = groups[gi];
    const int nt = (int)gterms[gi].size();
    const int nchunk = (int)std::min<long long>((gcost[gi] + target - 1) / target, std::max(1, nt));
    if (g.M <= 0 || g.N <= 0 || gcost[gi] <= target + target / 2 || nchunk <= 1) continue;
    long long acc = 0, per = (gcost[gi] + nchunk - 1) / nchunk;
    int parts = 1;
    for (int t = 0; t < nt; ++t) {
      acc += cost(gterms[gi][t]);
      if (acc >= per && t + 1 < nt && parts < nchunk) {
        ++parts;
        acc = 0;
      }
    }
    elems += (long long)parts * g.M * g.N;
  }
  return elems;
}

void TaskList::upload(cudaStream_t st, int slots, int waves, int tile_override) {
  std::vector<GTerm> terms;
  // a range of a group's terms, run by one job per tile of the group
  struct Chunk {
    int group, t0, tg, t1;   // GEMM terms [t0, tg), then element terms [tg, t1)
    long long part_off;      // its partial tiles; -1: written to the group
    long long cost;          // of one of its jobs
    int nseg;                // split form: accumulator segments
  };
  std::vector<Chunk> chunks;
  std::vector<GReduce> reds;
  std::vector<int> gemm_end(groups.size());   // end of each group's GEMM terms
  exec_flops = 0;
  auto is_gemm = [](const GTerm& t) { return t.kind == TK_GEMM && t.K > 0; };
  // pass 1: flatten the terms
  size_t nall = 0;
  for (const auto& built : gterms) nall += built.size();
  terms.reserve(nall);
  bool any_gemm = false;
  for (size_t gi = 0; gi < groups.size(); ++gi) {
    GGroup& g = groups[gi];
    g.t0 = (int)terms.size();
    // the kernels run a job's GEMM terms as one pipeline, then its element terms
    const std::vector<GTerm>& built = gterms[gi];
    bool ranked = false;
    for (const GTerm& t : built) {
      if (!is_gemm(t)) continue;
      terms.push_back(t);
      ranked = ranked || t.rank;
      exec_flops += 8.0 * g.M * g.N * t.K;
    }
    if (ranked && !split)
      std::stable_sort(terms.begin() + g.t0, terms.end(), [](const GTerm& a, const GTerm& b) { return a.rank < b.rank; });
    gemm_end[gi] = (int)terms.size();
    any_gemm = any_gemm || gemm_end[gi] > g.t0;
    if (terms.size() - g.t0 < built.size())
      for (const GTerm& t : built)
        if (!is_gemm(t)) terms.push_back(t);
    g.t1 = (int)terms.size();
  }
  // The large tile from 8 GFLOP a list on, the small one below (it keeps more CTAs busy).  Time
  // of an H.psi with the small tile over that with the large one, by the GFLOP of both its
  // lists: 12 columns 0.98 at 3, 0.99 at 10, 1.02 at 14, 1.07 at 25, 1.16 at 114; 24 columns, with
  // more and smaller sectors, 0.90 at 4, 0.97 at 19, 0.99 at 33, 1.08 at 78, 1.13 at 152.  They
  // meet between 14 and 50; from 8 GFLOP an H.psi on the autotuner times both.
  const bool large = exec_flops >= 8e9;
  tile = tile_override ? tile_override : large ? TILE_64x48 : TILE_32x32;
  // Bulk copies from 32 GFLOP a list on (H.psi of two lists, cp.async / bulk: 1.30 / 1.31 ms at
  // 10 + 23 GFLOP, 3.69 / 3.56 at 37 + 79, 37.3 / 34.6 at 1,270, 277 / 252 at 10,180; eight
  // block-sparse problems, 42 GFLOP in shorter sums, 2.007 / 2.017)
  bulk = !split && tile == TILE_64x48 && exec_flops >= 32e9;
  // Term lists are cut for 8 waves of CTAs (2 waves: 3.95 ms at 117 GFLOP; with 4 for the small
  // tile the longer chains of sums rounded 1.3 times as much at 1.2 GFLOP, in the same time),
  // those with bulk copies for 32: shorter chains round less, at the same time (8 / 32 waves, 2-norm
  // error in 1e-15: 1.19 / 1.09 in 3.55 / 3.50 ms at 117 GFLOP, 1.84 / 1.81 in 34.7 / 34.5 at 1,270),
  // while 242 us at 5 GFLOP became 258.
  if (waves <= 0) waves = split ? 4 : bulk ? 32 : 8;
  elementwise = !split && !any_gemm;
  if (elementwise) tile = TILE_32x32;
  const int TMt = split ? SPLIT_TILE_M : tile_rows(tile), TNt = split ? SPLIT_TILE_N : tile_cols(tile);
  if (!split) slots = slots / 2 * (tile == TILE_32x32 ? 4 : 2);   // resident CTAs per SM x SMs
  // Cost of a term in one tile.  Split form: its K steps of 16.  FP64 form, in cycles: a
  // chunk of 16 costs the busiest warp 12 DMMAs of 16 cycles per 8x8 sub-tile, and about
  // 150 cycles whatever its size.
  auto tile_cost = [&](int rows, int cols) -> long long {
    if (split) return 1;
    int wm, wn;
    const int mtot = (rows + 7) / 8, ntot = (cols + 7) / 8;
    warp_grid(mtot, ntot, TMt / 16, TNt / 16, wm, wn);
    return 192ll * ((mtot + wm - 1) / wm) * ((ntot + wn - 1) / wn) + 150;
  };
  const long long job_cost = split ? 3 : 1500;
  auto tcost = [&](const GTerm& t, long long per_chunk) -> long long {
    if (!is_gemm(t)) return split ? 1 : 100;
    const long long nk = (t.K + GEMM_TK - 1) / GEMM_TK;
    return split ? nk + 1 : nk * per_chunk;
  };
  auto step_m = [&](const GGroup& g) { return split ? TMt : tile_step(g.M, TMt); };
  auto step_n = [&](const GGroup& g) { return split ? TNt : tile_step(g.N, TNt); };
  // pass 2: cost of a whole tile of every group, and in all
  std::vector<long long> gcost(groups.size(), 0), gchunk(groups.size(), 0);
  long long total = 0;
  for (size_t gi = 0; gi < groups.size(); ++gi) {
    const GGroup& g = groups[gi];
    if (g.M <= 0 || g.N <= 0) continue;
    gchunk[gi] = tile_cost(std::min(g.M, step_m(g)), std::min(g.N, step_n(g)));
    long long c = job_cost;
    for (int t = g.t0; t < g.t1; ++t) c += tcost(terms[t], gchunk[gi]);
    gcost[gi] = c;
    total += c * (long long)((g.M + TMt - 1) / TMt) * ((g.N + TNt - 1) / TNt);
  }
  // Split form: accumulator segments of GEMM terms [a, b), SPLIT_SEG steps each over one
  // term when the epilogue applies its coefficient, over all of them otherwise.
  auto segments = [&](int a, int b) {
    int nseg = 0, steps = 0;
    for (int t = a; t < b; ++t) {
      steps += (terms[t].K + GEMM_TK - 1) / GEMM_TK;
      if (!term_alpha && t + 1 < b) continue;
      nseg += (steps + SPLIT_SEG - 1) / SPLIT_SEG;
      steps = 0;
    }
    return nseg;
  };
  // pass 3: jobs, splitting long groups into term chunks of about a wave's share of the work
  // (0 waves: none).  Aimed at no less than 3000 cycles a job: at m=40 (7 MFLOP in all) 15000
  // left the longest jobs to run alone (45 against 33 us), 6000 was no faster and summed longer
  // chains.  FP64 form: nor are more than `chain` products summed in one accumulator where the
  // terms allow it; at m=4000, where a wave's share is longer, the error of equal terms falls
  // from 8.5e-15 to 5.9e-15 at 16384 (4.5e-15 at 8192, with twice the partial tiles: 2 GB) in
  // the same time.
  auto cut_jobs = [&](int nwaves, long long chain) {
    const long long target =
        nwaves ? std::max<long long>(split ? 8 : 3000, total / std::max(1, slots * nwaves)) : LLONG_MAX / 4;
    chunks.clear();
    reds.clear();
    part_elems = max_red_elems = 0;
    for (size_t gi = 0; gi < groups.size(); ++gi) {
      const GGroup& g = groups[gi];
      if (g.M <= 0 || g.N <= 0) continue;
      const int tg = gemm_end[gi];
      long long want = gcost[gi] <= target + target / 2 ? 1 : (gcost[gi] + target - 1) / target, ksum = 0;
      if (!split) {
        for (int t = g.t0; t < tg; ++t) ksum += terms[t].K;
        want = std::max(want, (ksum + chain - 1) / chain);
      }
      const int nchunk = (int)std::min<long long>(want, std::max(1, g.t1 - g.t0));
      if (nchunk <= 1) {
        chunks.push_back({(int)gi, g.t0, tg, g.t1, -1, gcost[gi], split ? segments(g.t0, tg) : 0});
        continue;
      }
      // contiguous chunks of roughly equal cost
      const long long base = part_elems, mn = (long long)g.M * g.N;
      long long acc = 0, per = (gcost[gi] + nchunk - 1) / nchunk;
      int P = 0;
      for (int t = g.t0, c0 = g.t0; t < g.t1; ++t) {
        acc += tcost(terms[t], gchunk[gi]);
        if (t + 1 < g.t1 && (acc < per || P + 1 >= nchunk)) continue;
        const int cg = std::max(c0, std::min(tg, t + 1));
        chunks.push_back({(int)gi, c0, cg, t + 1, base + P * mn, acc + job_cost, split ? segments(c0, cg) : 0});
        ++P;
        c0 = t + 1;
        acc = 0;
      }
      part_elems += P * mn;
      reds.push_back(GReduce{(int)gi, P, base});
      max_red_elems = std::max(max_red_elems, mn);
    }
  };
  constexpr long long kChain = 16384, kAnyChain = LLONG_MAX / 4;
  cut_jobs(waves, kChain);
  // A list of the no-allocation entry whose partial tiles would pass its fixed scratch: cut for
  // at most 8 waves and, where those of the basic schedule would fit, for fewer until they do.
  // Where neither fits the entry refuses the superblock, and the list stays as it was.
  if (scratch_beside >= 0 && scratch_beside <= TSC_NOALLOC_SCRATCH_ELEMS) {
    const long long room = TSC_NOALLOC_SCRATCH_ELEMS - scratch_beside;
    if (part_elems > room) {
      int w = std::min(waves, 8);
      cut_jobs(w, kAnyChain);
      if (basic_part_elems() <= room)
        while (w && part_elems > room) cut_jobs(w /= 2, kAnyChain);
      if (part_elems > room) cut_jobs(waves, kChain);
    }
  }
  // longest jobs first: the persistent CTAs then approximate LPT balancing
  std::stable_sort(chunks.begin(), chunks.end(), [](const Chunk& a, const Chunk& b) { return a.cost > b.cost; });
  auto tiles_m = [&](const GGroup& g) { return (g.M + TMt - 1) / TMt; };
  auto tiles_n = [&](const GGroup& g) { return (g.N + TNt - 1) / TNt; };
  njobs = 0;
  for (const Chunk& c : chunks) njobs += tiles_m(groups[c.group]) * tiles_n(groups[c.group]);
  nreds = (int)reds.size();
  nterms = (long long)terms.size();
  std::vector<int> starts;
  std::vector<SJob> sjobs;
  std::vector<ZJob> zjobs;
  (split ? sjobs.reserve(njobs) : zjobs.reserve(njobs));
  for (const Chunk& c : chunks) {
    const GGroup& g = groups[c.group];
    const bool partial = c.part_off >= 0;
    const uint8_t c_base = partial ? (uint8_t)BASE_PART : g.c_base, beta = !partial && g.beta;
    const long long c_off = partial ? c.part_off : g.c_off;
    const int c_ld = partial ? g.M : g.c_ld, tm = tiles_m(g), tn = tiles_n(g);
    if (split) {
      SJob j{};
      j.c_off = c_off;
      j.s_off = partial ? -1 : g.s_off;
      j.c_ld = c_ld;
      j.M = g.M;
      j.N = g.N;
      j.t0 = c.t0;
      j.tg = c.tg;
      j.t1 = c.t1;
      j.nseg = c.nseg;
      j.c_base = c_base;
      j.beta = beta;
      for (j.tm = 0; j.tm < tm; ++j.tm)
        for (j.tn = 0; j.tn < tn; ++j.tn) sjobs.push_back(j);
    } else {
      ZJob z{};
      z.c_base = c_base;
      z.c_off = c_off;
      z.c_ld = c_ld;
      z.beta = beta;
      z.t0 = c.t0;
      z.tg = c.tg;
      z.t1 = c.t1;
      const int sm = step_m(g), sn = step_n(g);
      for (int a = 0; a < tm; ++a) {
        z.m0 = a * sm;
        z.mend = std::min(g.M, z.m0 + sm);
        for (int b = 0; b < tn; ++b) {
          z.n0 = b * sn;
          z.nend = std::min(g.N, z.n0 + sn);
          zjobs.push_back(z);
        }
      }
    }
  }
  // split form: dealt out to the CTAs, each job to the one with the least work so far
  if (split) {
    nctas = std::min(njobs, slots / 2);
    std::priority_queue<std::pair<long long, int>, std::vector<std::pair<long long, int>>, std::greater<>> load;
    for (int c = 0; c < nctas; ++c) load.push({0, c});
    std::vector<int> cta(njobs);
    starts.assign(nctas + 1, 0);
    int k = 0;
    for (const Chunk& c : chunks)
      for (int e = k + tiles_m(groups[c.group]) * tiles_n(groups[c.group]); k < e; ++k) {
        auto [w, to] = load.top();
        load.pop();
        cta[k] = to;
        ++starts[to + 1];
        load.push({w + c.cost, to});
      }
    for (int c = 0; c < nctas; ++c) starts[c + 1] += starts[c];
    std::vector<SJob> dealt(njobs);
    std::vector<int> at(starts.begin(), starts.end());
    for (k = 0; k < njobs; ++k) dealt[at[cta[k]]++] = sjobs[k];
    sjobs.swap(dealt);
  }
  size_t bj = sjobs.size() * sizeof(SJob) + zjobs.size() * sizeof(ZJob), bg = groups.size() * sizeof(GGroup),
         bt = terms.size() * sizeof(GTerm), br = reds.size() * sizeof(GReduce), bs = starts.size() * sizeof(int);
  auto al = [](size_t x) { return (x + 255) / 256 * 256; };
  size_t total_b = al(bj) + al(bg) + al(bt) + al(br) + al(bs) + 256;
  dev = std::make_shared<DevBuf>((total_b + 15) / 16, st, false);
  char* base = reinterpret_cast<char*>(dev->p);
  d_sjobs = reinterpret_cast<SJob*>(base);
  d_zjobs = reinterpret_cast<ZJob*>(base);
  d_groups = reinterpret_cast<GGroup*>(base + al(bj));
  d_terms = reinterpret_cast<GTerm*>(base + al(bj) + al(bg));
  d_reds = reinterpret_cast<GReduce*>(base + al(bj) + al(bg) + al(bt));
  d_starts = reinterpret_cast<int*>(base + al(bj) + al(bg) + al(bt) + al(br));
  d_next = reinterpret_cast<int*>(base + al(bj) + al(bg) + al(bt) + al(br) + al(bs));   // zero: the host copy is
  std::vector<char> host(total_b, 0);
  if (bj) std::memcpy(host.data(), split ? (const void*)sjobs.data() : (const void*)zjobs.data(), bj);
  if (bg) std::memcpy(host.data() + al(bj), groups.data(), bg);
  if (bt) std::memcpy(host.data() + al(bj) + al(bg), terms.data(), bt);
  if (br) std::memcpy(host.data() + al(bj) + al(bg) + al(bt), reds.data(), br);
  if (bs) std::memcpy(host.data() + al(bj) + al(bg) + al(bt) + al(br), starts.data(), bs);
  cuda_check(cudaMemcpyAsync(base, host.data(), total_b, cudaMemcpyHostToDevice, st), "task upload");
  part = part_elems ? std::make_shared<DevBuf>((size_t)part_elems, st, false) : nullptr;
  cuda_check(cudaStreamSynchronize(st), "task upload sync");
}

cudaError_t launch_tasks(const TaskList& tl, const Bases& b, int* fault, const WaitLimits& limits, cudaStream_t st) {
  cudaError_t e;
  if (tl.split)
    e = launch_grouped_zgemm_split(tl.d_sjobs, tl.d_starts, tl.nctas, tl.d_terms, b, tl.arenas, fault, limits.split,
                                   tl.term_alpha ? 1 : 0, st);
  else if (tl.elementwise)
    e = launch_grouped_axpy(tl.d_zjobs, tl.njobs, tl.d_terms, b, st);
  else
    e = launch_grouped_zgemm(tl.d_zjobs, tl.njobs, tl.d_terms, b, tl.d_next, fault, limits.fp64, st, tl.tile, tl.bulk);
  if (e == cudaSuccess && tl.nreds) e = launch_reduce_partials(tl.d_reds, tl.nreds, tl.d_groups, b, tl.max_red_elems, st);
  return e;
}

void Engine::run_tasks(TaskList& tl, double2* in, double2* out, double2* scr) {
  launch(tl, Bases{{nullptr, in, out, scr, tl.part ? tl.part->p : nullptr}});
}

void Engine::launch(TaskList& tl, const Bases& b) {
  if (tl.njobs > 0 && (tl.split || tl.bulk)) waits_unread_ = true;
  cuda_check(launch_tasks(tl, b, d_fault, wait_limits_, st), tl.split ? "grouped_zgemm_split" : "grouped_zgemm");
}

// ---- block transfer ----------------------------------------------------------------------
DBlock Engine::upload_block(const int*& ip, const cplx*& dp) {
  DBlock b;
  b.len = *ip++;
  b.num = *ip++;
  b.dim = *ip++;
  b.up_dif = *ip++;
  b.down_dif = *ip++;
  if (b.num < 0 || b.num > 1000000) throw Error(-1, "bad block descriptor");
  long long off = 0;
  for (int i = 0; i < b.num; ++i) {
    SubDesc s;
    s.num_up = *ip++;
    s.num_down = *ip++;
    s.down_dif = *ip++;
    s.row_dim = *ip++;
    s.sdim = *ip++;
    if (s.row_dim < 0 || s.sdim < 0) throw Error(-1, "bad sub-block dims");
    s.off = off;
    off += (long long)s.row_dim * s.sdim;
    b.sub.push_back(s);
  }
  b.buf = std::make_shared<DevBuf>((size_t)off, st, false);
  if (off) cuda_check(cudaMemcpyAsync(b.buf->p, dp, off * sizeof(double2), cudaMemcpyHostToDevice, st), "upload");
  dp += off;
  return b;
}

void Engine::download_block(const DBlock& b, std::vector<int>& ints, std::vector<cplx>& data) const {
  ints.insert(ints.end(), {b.len, b.num, b.dim, b.up_dif, b.down_dif});
  size_t d0 = data.size();
  for (const auto& s : b.sub) ints.insert(ints.end(), {s.num_up, s.num_down, s.down_dif, s.row_dim, s.sdim});
  long long tot = b.total();
  data.resize(d0 + tot);
  // one copy per run of sub-blocks that lie one after another (a block of the engine's own
  // is one run; 700 copies of a grown model took 10 ms)
  for (size_t i = 0; i < b.sub.size();) {
    const long long off = b.sub[i].off;
    long long n = 0;
    for (; i < b.sub.size() && b.sub[i].off == off + n; ++i) n += (long long)b.sub[i].row_dim * b.sub[i].sdim;
    if (n)
      cuda_check(cudaMemcpyAsync(&data[d0], b.buf->p + off, n * sizeof(double2), cudaMemcpyDeviceToHost, st),
                 "download");
    d0 += n;
  }
  cuda_check(cudaStreamSynchronize(st), "download sync");
}

// ---- stored models: device-resident under a byte limit, host memory beyond it ----
namespace {
template <class F>
void for_blocks(DModel& m, F&& f) {
  f(m.ham);
  for (auto& os : m.sub)
    for (auto& b : os.op) f(b);
}
long long model_bytes(DModel& m) {
  long long n = 0;
  for_blocks(m, [&](DBlock& b) {
    if (b.buf) n += (long long)b.buf->n * (long long)sizeof(double2);
  });
  return n;
}
}  // namespace

long long ModelStore::limit() const {
  if (limit_ >= 0) return limit_;
  size_t fr = 0, tot = 0;
  if (cudaMemGetInfo(&fr, &tot) != cudaSuccess) {
    cudaGetLastError();
    return 1ll << 62;
  }
  return (long long)(default_frac_ * (double)tot);
}

void ModelStore::spill(Entry& e) {
  if (e.spilled) return;
  auto t0 = std::chrono::steady_clock::now();
  e.host.clear();
  for_blocks(e.m, [&](DBlock& b) {
    e.host.emplace_back();
    if (!b.buf) return;
    auto& h = e.host.back();
    h.resize(b.buf->n);
    if (b.buf->n)
      cuda_check(cudaMemcpyAsync(h.data(), b.buf->p, b.buf->n * sizeof(double2), cudaMemcpyDeviceToHost, st_),
                 "spill d2h");
  });
  cuda_check(cudaStreamSynchronize(st_), "spill sync");
  for_blocks(e.m, [&](DBlock& b) { b.buf.reset(); });
  e.spilled = true;
  resident_ -= e.bytes;
  host_bytes_ += e.bytes;
  spills++;
  moved_bytes += (double)e.bytes;
  moved_seconds += std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
}

void ModelStore::restore(Entry& e) {
  if (!e.spilled) return;
  if (e.on_disk) from_disk(e);
  auto t0 = std::chrono::steady_clock::now();
  size_t k = 0;
  for_blocks(e.m, [&](DBlock& b) {
    auto& h = e.host[k++];
    if (h.empty()) return;
    b.buf = std::make_shared<DevBuf>(h.size(), st_, false);
    cuda_check(cudaMemcpyAsync(b.buf->p, h.data(), h.size() * sizeof(double2), cudaMemcpyHostToDevice, st_),
               "restore h2d");
  });
  cuda_check(cudaStreamSynchronize(st_), "restore sync");
  e.host.clear();
  e.host.shrink_to_fit();
  e.spilled = false;
  resident_ += e.bytes;
  host_bytes_ -= e.bytes;
  restores++;
  moved_bytes += (double)e.bytes;
  moved_seconds += std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
}

// spills least recently used models (never `keep`) until the resident ones fit
void ModelStore::enforce(long long keep) {
  const long long lim = limit();
  while (resident_ > lim) {
    Entry* victim = nullptr;
    for (auto& kv : map_)
      if (kv.first != keep && !kv.second.spilled && kv.second.bytes > 0 &&
          (!victim || kv.second.tick < victim->tick))
        victim = &kv.second;
    if (!victim) break;
    spill(*victim);
  }
  enforce_host(keep);
}

void ModelStore::put(int side, int len, const DModel& m) {
  const long long k = key(side, len);
  auto it = map_.find(k);
  if (it != map_.end()) {
    Entry& o = it->second;
    if (!o.spilled) resident_ -= o.bytes;
    else if (!o.on_disk) host_bytes_ -= o.bytes;
    if (o.on_disk) std::remove(o.file.c_str());
  }
  Entry& e = map_[k];
  e.m = m;
  e.host.clear();
  e.spilled = false;
  e.on_disk = false;
  e.file.clear();
  e.bytes = model_bytes(e.m);
  e.tick = ++clock_;
  resident_ += e.bytes;
  enforce(k);
}

DModel ModelStore::get(int side, int len) {
  const long long k = key(side, len);
  auto it = map_.find(k);
  if (it == map_.end()) throw Error(-4, "stored model not found (side " + std::to_string(side) + ", length " +
                                            std::to_string(len) + ")");
  Entry& e = it->second;
  e.tick = ++clock_;
  if (e.spilled) {
    restore(e);
    enforce(k);
  }
  return e.m;
}

// host copies of the least recently used spilled models to files until the
// spilled models' host bytes fit under the host limit
void ModelStore::enforce_host(long long keep) {
  if (host_limit_ < 0 || disk_dir_.empty()) return;
  while (host_bytes_ > host_limit_) {
    long long vk = 0;
    Entry* victim = nullptr;
    for (auto& kv : map_)
      if (kv.first != keep && kv.second.spilled && !kv.second.on_disk && kv.second.bytes > 0 &&
          (!victim || kv.second.tick < victim->tick)) {
        victim = &kv.second;
        vk = kv.first;
      }
    if (!victim) break;
    to_disk(vk, *victim);
  }
}

// one file per model: for every block, its element count (int64) and elements
void ModelStore::to_disk(long long k, Entry& e) {
  auto t0 = std::chrono::steady_clock::now();
  e.file = disk_dir_ + "/tsc_model_" + std::to_string(k >> 32) + "_" + std::to_string(k & 0xffffffff) + "_" +
           std::to_string(reinterpret_cast<uintptr_t>(this)) + ".bin";
  std::FILE* f = std::fopen(e.file.c_str(), "wb");
  if (!f) throw Error(-1, "model spill: cannot create " + e.file);
  bool ok = true;
  for (const auto& h : e.host) {
    const long long n = (long long)h.size();
    ok = ok && std::fwrite(&n, sizeof(n), 1, f) == 1;
    if (n) ok = ok && std::fwrite(h.data(), sizeof(double2), (size_t)n, f) == (size_t)n;
  }
  ok = (std::fclose(f) == 0) && ok;
  if (!ok) {
    std::remove(e.file.c_str());
    throw Error(-1, "model spill: cannot write " + e.file);
  }
  std::vector<std::vector<double2>>().swap(e.host);
  e.on_disk = true;
  host_bytes_ -= e.bytes;
  disk_writes++;
  disk_bytes += (double)e.bytes;
  disk_seconds += std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
}

void ModelStore::from_disk(Entry& e) {
  auto t0 = std::chrono::steady_clock::now();
  std::FILE* f = std::fopen(e.file.c_str(), "rb");
  if (!f) throw Error(-1, "model spill: cannot open " + e.file);
  e.host.clear();
  bool ok = true;
  size_t nb = 0;
  for_blocks(e.m, [&](DBlock&) { nb++; });
  for (size_t i = 0; i < nb && ok; ++i) {
    long long n = 0;
    ok = std::fread(&n, sizeof(n), 1, f) == 1 && n >= 0;
    e.host.emplace_back();
    if (ok && n) {
      e.host.back().resize((size_t)n);
      ok = std::fread(e.host.back().data(), sizeof(double2), (size_t)n, f) == (size_t)n;
    }
  }
  std::fclose(f);
  if (!ok) throw Error(-1, "model spill: cannot read " + e.file);
  std::remove(e.file.c_str());
  e.file.clear();
  e.on_disk = false;
  host_bytes_ += e.bytes;
  disk_reads++;
  disk_bytes += (double)e.bytes;
  disk_seconds += std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
}

void ModelStore::clear() {
  for (auto& kv : map_)
    if (kv.second.on_disk) std::remove(kv.second.file.c_str());
  map_.clear();
  resident_ = 0;
  host_bytes_ = 0;
}

DBlock Engine::copy_block(const DBlock& b) {
  DBlock c = b;
  long long off = 0;
  for (auto& s : c.sub) {
    s.off = off;
    off += (long long)s.row_dim * s.sdim;
  }
  c.buf = std::make_shared<DevBuf>((size_t)off, st, false);
  for (int i = 0; i < b.num; ++i) {
    long long n = (long long)b.sub[i].row_dim * b.sub[i].sdim;
    if (n)
      cuda_check(cudaMemcpyAsync(c.buf->p + c.sub[i].off, b.buf->p + b.sub[i].off, n * sizeof(double2),
                                 cudaMemcpyDeviceToDevice, st),
                 "copy");
  }
  return c;
}

double Engine::wave_norm2(const double2* d, long long n) {
  cuda_check(launch_multi_dot(d, 0, 1, d, n, d_red, d_scal + 1900, st), "wave norm");
  cuda_check(cudaMemcpyAsync(h_scal + 1900, d_scal + 1900, sizeof(double), cudaMemcpyDeviceToHost, st), "d2h");
  cuda_check(cudaStreamSynchronize(st), "sync");
  return h_scal[1900];
}

void Engine::normalize(double2* d, long long n) {
  if (n <= 0) return;
  cuda_check(launch_multi_dot(d, 0, 1, d, n, d_red, d_scal + 1901, st), "normalize norm");
  cuda_check(launch_scale(d, d_scal + 1901, n, 1, st), "scale");
}

// random_number stand-in (splitmix64 -> uniform [0,1)), block.f90:1154-1180
double Engine::rand01() {
  uint64_t z = (rng += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z = z ^ (z >> 31);
  return (double)(z >> 11) * (1.0 / 9007199254740992.0);
}

void Engine::wave_initialize(const WLayout& wl, double2* d) {
  std::vector<double2> h((size_t)wl.dim);
  for (const auto& s : wl.sec) {
    size_t n = (size_t)s.sys_dim * s.env_dim;
    for (size_t e = 0; e < n; ++e) h[s.off + e].x = rand01();
    for (size_t e = 0; e < n; ++e) h[s.off + e].y = rand01();
  }
  cuda_check(cudaMemcpyAsync(d, h.data(), h.size() * sizeof(double2), cudaMemcpyHostToDevice, st), "upload");
  normalize(d, wl.dim);
  cuda_check(cudaStreamSynchronize(st), "sync");
}

}  // namespace tsc
