// ixb_tridiag.cu -- batched tridiagonal solves over device arrays, the
// batched form of tridiagonal (source/mod_solucionador.f90:25-47).
//
// Hybrid solver, by layout and size:
//  layout 0 (each system contiguous, like the reference's x-lines)
//    n <= 4864: tri_stream_kernel, one system per CTA at a time, the next one
//               arriving by bulk copies (any alignment);
//    longer:    tri_contig_kernel, one system staged per CTA.
//  layout 1 (systems interleaved, row i of system s at i*nsys+s, like the
//  y-lines of a column-major field)
//    short:     tri_cols_kernel, whole systems in the registers of a CTA;
//    n <= 4096 in whole 16-byte granules: tri_strided_kernel, a group of
//               systems in a thread-block cluster;
//    others:    tri_block_kernel, blocks of 128 rows, each read twice (the
//               second time from L2) around the solve of the block ends.
// The exact solver stages contiguous systems (tri_contig_kernel) and walks
// interleaved ones with one thread each (tri_inter_kernel), in the
// reference's operation order.
#include <cooperative_groups.h>
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <mutex>

#include "ixb_internal.h"

namespace ixb {

template <class R, int SOLVER, int TL, int G>
__global__ void __launch_bounds__(TL * G) tri_contig_kernel(const R* __restrict__ a, const R* __restrict__ b,
                                                            const R* __restrict__ c, const R* __restrict__ d,
                                                            R* x, int n, int nsys, int m, int mp) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  R* sm = reinterpret_cast<R*>(smem_raw);
  const int npad = G * m;
  const size_t LS = line_smem_elems(G, mp), arr = (size_t)G * mp;
  const long long s0 = (long long)blockIdx.x * TL;
  for (int idx = threadIdx.x; idx < TL * npad; idx += TL * G) {
    const int l = idx / npad, r = idx - l * npad;
    const long long s = s0 + l;
    if (s >= nsys) continue;
    R ra = R(0), rb = R(1), rc = R(0), rd = R(0);
    if (r < n) {
      const size_t g = (size_t)s * n + r;
      ra = r == 0 ? R(0) : a[g];
      rb = b[g];
      rc = r == n - 1 ? R(0) : c[g];
      rd = d[g];
    }
    const int ch = r / m;
    const size_t o = (size_t)l * LS + (size_t)ch * mp + (r - ch * m);
    sm[o] = ra; sm[o + arr] = rb; sm[o + 2 * arr] = rc; sm[o + 3 * arr] = rd;
  }
  __syncthreads();
  {
    const int l = threadIdx.x / G;
    const bool active = s0 + l < nsys;
    R* line = sm + (size_t)l * LS;
    if (SOLVER == IXB_SOLVER_EXACT) {
      if (active && threadIdx.x % G == 0) thomas_exact(line, line + arr, line + 2 * arr, line + 3 * arr, n, m, mp);
    } else {
      chunk_solve<R, G>(line, m, mp, active);
    }
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < TL * n; idx += TL * G) {
    const int l = idx / n, r = idx - l * n;
    const long long s = s0 + l;
    if (s >= nsys) continue;
    const int ch = r / m;
    x[(size_t)s * n + r] = sm[(size_t)l * LS + 3 * arr + (size_t)ch * mp + (r - ch * m)];
  }
}

// One thread per interleaved system, the reference's operation order
// (modified diagonal in `work`, modified right-hand side in x).
template <class R>
__global__ void __launch_bounds__(128) tri_inter_kernel(const R* __restrict__ a, const R* __restrict__ b,
                                                        const R* __restrict__ c, const R* d, R* x,
                                                        R* __restrict__ work, int n, int nsys) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nsys) return;
  const size_t S = (size_t)nsys;
  R bp = b[s], dp = d[s];
  work[s] = bp;
  x[s] = dp;
  for (int i = 1; i < n; ++i) {
    const size_t g = (size_t)i * S + s;
    const R q = a[g] / bp;
    dp = d[g] - q * dp;
    bp = b[g] - q * c[g - S];
    x[g] = dp;
    work[g] = bp;
  }
  R xn = dp / bp;
  x[(size_t)(n - 1) * S + s] = xn;
  for (int i = n - 2; i >= 0; --i) {
    const size_t g = (size_t)i * S + s;
    xn = (x[g] - c[g] * xn) / work[g];
    x[g] = xn;
  }
}

// ---------------------------------------------------------------------------
// Streamed contiguous solve (hybrid solver): CTAs of T threads walk their
// systems; while one is solved from registers, the bulk-copy engine is
// already loading the CTA's next one into shared memory, and the solution
// leaves through a bulk shared->global copy.  Thread t owns rows t*M ..
// t*M+M-1 (M odd, so the threads of a warp reading their own row j hit
// different banks); it eliminates them in registers (Chunk), the reduced rows
// go through reduced_pcr, and each thread back-substitutes its rows.
// Long lines are bound by HBM (4096 x 4096 binary64: 105 us, 6.4 TB/s, 98 % of
// the measured copy rate; 135.2 us before the reduced system's shared-memory
// traffic was cut), short ones by the latency of one system.
//
// Bulk copies move whole 16-byte granules.  A system that starts or ends
// inside one (odd n, or an array that is not 16-byte aligned) keeps its
// alignment in shared memory (a shift of up to 16 bytes), the bulk copy takes
// the whole granules, and the up to 16 / sizeof(R) - 1 elements on each side
// go by ordinary loads and stores, so nothing outside the system is touched.
// (701-row systems, 302 of them, binary64: 22.5 us by the staged kernel
// before, 9.8 us here.)  RAG picks that form; where every system fills whole
// granules the fixed addresses save 5 % at 4096 x 4096 (113.0 against 107.3 us, both before this solve
// reached 105).
//
// Every wait on the copy engine is bounded: on a timeout the CTA records it
// in g_tri_timeout, waits (bounded) for its copies still in flight and
// leaves without writing.
// ---------------------------------------------------------------------------
namespace {

constexpr int kSpinLimit = 1 << 22;  // bounded mbarrier polls (a hang guard)
__device__ int g_tri_timeout = 0;
// Poll limit of the first wait of every CTA of the streamed and the cluster
// kernel (their other waits, and the drain after a timeout, keep kSpinLimit); lowered only by
// ixb_tridiag_set_first_wait_limit, for failure-detection tests.
__device__ int g_tri_first_wait_polls = kSpinLimit;

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void bulk_load(void* dst, const void* src, unsigned bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ void bulk_store(void* dst, const void* src, unsigned bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem_u32(src)),
               "r"(bytes)
               : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

__device__ __forceinline__ void bulk_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_store_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// At most `limit` polls, and no longer than about two seconds (%globaltimer).
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, unsigned parity, int limit = kSpinLimit) {
  unsigned long long t0;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  for (int i = 0; i < limit; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 255) == 255) {
      unsigned long long t;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
      if (t - t0 > 2000000000ull) return false;
    }
  }
  return false;
}

// elements per 16-byte granule
template <class R>
constexpr int kGran = 16 / (int)sizeof(R);

// a system's rows at p: elements before the first whole granule (`head`),
// in whole granules (`body`), and the shift that keeps p's alignment
template <class R, bool RAG>
struct Granules {
  int shift, head, body;
  __device__ __forceinline__ Granules(const R* p, int n) {
    constexpr int E = kGran<R>;
    if constexpr (!RAG) {  // every system starts and ends on a granule
      shift = head = 0;
      body = n;
      return;
    }
    shift = (int)((reinterpret_cast<uintptr_t>(p) / sizeof(R)) & (E - 1));
    head = min((E - shift) & (E - 1), n);
    body = (n - head) & ~(E - 1);
  }
  // element of edge slot i (0 .. 2*kGran-1: head, then tail), -1: none
  __device__ __forceinline__ int edge(int i, int n) const {
    constexpr int E = kGran<R>;
    if (i < E) return i < head ? i : -1;
    const int r = head + body + i - E;
    return r < n ? r : -1;
  }
};

// Shared memory of the streamed kernel: 4 row arrays (the copy target) and
// the solution, each T*M elements and room for the shift, the reduced
// system (9*T) and the mbarrier.
template <class R, int T, int M>
__host__ __device__ constexpr size_t stream_smem_bytes() {
  return ((size_t)5 * (T * M + kGran<R>) + 9 * T) * sizeof(R) + 16;
}

template <class R, int T, int M, bool RAG>
__global__ void __launch_bounds__(T) tri_stream_kernel(const R* a, const R* b, const R* c, const R* d, R* x, int n,
                                                       int nsys) {
  constexpr int E = kGran<R>, NS = T * M + E;
  static_assert(8 * E <= T, "one thread per edge element of the four arrays");
  extern __shared__ __align__(128) unsigned char smem_raw[];
  R* buf = reinterpret_cast<R*>(smem_raw);  // a | b | c | d, NS each
  R* xbuf = buf + 4 * NS;
  R* red = xbuf + NS;
  uint64_t* bar = reinterpret_cast<uint64_t*>(red + 9 * T);
  const int tid = threadIdx.x;
  auto row_of = [&](int q) { return q == 0 ? a : q == 1 ? b : q == 2 ? c : d; };
  if constexpr (!RAG) {  // identity rows pad every system to T*M rows; the copies never touch them
    for (int r = n + tid; r < T * M; r += T) {
      buf[r] = R(0); buf[NS + r] = R(1); buf[2 * NS + r] = R(0); buf[3 * NS + r] = R(0);
    }
  }
  if (tid == 0) mbar_init(bar);
  __syncthreads();
  auto issue = [&](unsigned s) {
    const size_t off = (size_t)s * n;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // earlier reads of buf precede the copies
    unsigned bytes = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) bytes += (unsigned)(Granules<R, RAG>(row_of(q) + off, n).body * sizeof(R));
    mbar_expect_tx(bar, bytes);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const R* p = row_of(q) + off;
      const Granules<R, RAG> gr(p, n);
      if (gr.body)
        bulk_load(buf + q * NS + gr.shift + gr.head, p + gr.head, (unsigned)(gr.body * sizeof(R)), bar);
    }
  };
  // this thread's edge element of system s: its slot in buf (or -1) and value
  auto edge_load = [&](unsigned s, R& v) -> int {
    if (!RAG || tid >= 8 * E) return -1;
    const int q = tid / (2 * E);
    const R* p = row_of(q) + (size_t)s * n;
    const Granules<R, RAG> gr(p, n);
    const int r = gr.edge(tid % (2 * E), n);
    if (r < 0) return -1;
    v = p[r];
    return q * NS + gr.shift + r;
  };
  // systems are counted in unsigned: one past the last of 2^31 - 1 by a grid still fits
  const unsigned systems = (unsigned)nsys;
  if (blockIdx.x < systems) {
    if (tid == 0) issue(blockIdx.x);
    R v;
    const int slot = edge_load(blockIdx.x, v);
    if (slot >= 0) buf[slot] = v;
  }
  const int first_limit = *(volatile int*)&g_tri_first_wait_polls;
  unsigned parity = 0;
  bool failed = false;
  for (unsigned s = blockIdx.x; s < systems; s += gridDim.x) {
    const bool ok = mbar_wait_bounded(bar, parity, s == blockIdx.x ? first_limit : kSpinLimit);
    if (__syncthreads_or(!ok)) { failed = true; break; }
    parity ^= 1;
    // own rows into registers (row 0 has no a, row n-1 no c; identity rows past n)
    Chunk<R, M> ch;
    {
      const size_t off = (size_t)s * n;
      const R* ba = buf + Granules<R, RAG>(a + off, n).shift;
      const R* bb = buf + NS + Granules<R, RAG>(b + off, n).shift;
      const R* bc = buf + 2 * NS + Granules<R, RAG>(c + off, n).shift;
      const R* bd = buf + 3 * NS + Granules<R, RAG>(d + off, n).shift;
#pragma unroll
      for (int j = 0; j < M; ++j) {
        const int r = tid * M + j;
        if constexpr (RAG) {
          const bool in = r < n;
          ch.a[j] = in && r > 0 ? ba[r] : R(0);
          ch.b[j] = in ? bb[r] : R(1);
          ch.c[j] = r < n - 1 ? bc[r] : R(0);
          ch.d[j] = in ? bd[r] : R(0);
        } else {
          ch.a[j] = r == 0 ? R(0) : ba[r];
          ch.b[j] = bb[r];
          ch.c[j] = r == n - 1 ? R(0) : bc[r];
          ch.d[j] = bd[r];
        }
      }
    }
    __syncthreads();  // the row buffers are free: start loading the next system
    const unsigned next = s + gridDim.x;
    R ev = R(0);
    int eslot = -1;
    if (next < systems) {
      if (tid == 0) issue(next);
      eslot = edge_load(next, ev);
    }
    ch.eliminate();
    R x0, xl;
    reduced_pcr<R, true>(red, T, 1, T, tid, tid, true, ch.eA, ch.eC, ch.eD, ch.oA, ch.oC, ch.oD, x0, xl,
                         [](bool q) { return (bool)__syncthreads_or(q); });
    ch.substitute(x0, xl);
    // the previous solution must have left xbuf before it is overwritten
    if (tid == 0) bulk_store_wait_read();
    __syncthreads();
    R* xs = x + (size_t)s * n;
    const Granules<R, RAG> gx(xs, n);
#pragma unroll
    for (int j = 0; j < M; ++j) xbuf[gx.shift + tid * M + j] = ch.d[j];
    if (eslot >= 0) buf[eslot] = ev;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // generic writes -> copy engine
    __syncthreads();
    if (tid == 0 && gx.body) bulk_store(xs + gx.head, xbuf + gx.shift + gx.head, (unsigned)(gx.body * sizeof(R)));
    if (RAG && tid < 2 * E) {
      const int r = gx.edge(tid, n);
      if (r >= 0) xs[r] = xbuf[gx.shift + r];
    }
  }
  if (failed) {
    if (tid == 0) {
      atomicExch(&g_tri_timeout, 1);
      mbar_wait_bounded(bar, parity);  // copies still in flight land before the CTA leaves
    }
  }
  if (tid == 0) bulk_store_wait_all();
}

template <class R, int T, int M>
cudaError_t stream_launch(const R* a, const R* b, const R* c, const R* d, R* x, int n, int nsys, int nsm,
                          cudaStream_t st) {
  const uintptr_t all = (uintptr_t)a | (uintptr_t)b | (uintptr_t)c | (uintptr_t)d | (uintptr_t)x;
  const bool ragged = (all & 15) != 0 || ((size_t)n * sizeof(R)) % 16 != 0;
  auto k = ragged ? tri_stream_kernel<R, T, M, true> : tri_stream_kernel<R, T, M, false>;
  constexpr size_t smem = stream_smem_bytes<R, T, M>();
  if (smem > 48 * 1024) {
    const cudaError_t e = allow_smem(k, 0);
    if (e != cudaSuccess) return e;
  }
  // about one wave: by shared memory (227 KB per SM, 1 KB reserved per CTA)
  // and threads; the CTAs do not depend on one another
  const int per_sm = std::max(1, std::min((int)(227 * 1024 / (smem + 1024)), 1024 / T));
  k<<<std::min(nsys, nsm * per_sm), T, smem, st>>>(a, b, c, d, x, n, nsys);
  return cudaGetLastError();
}

// Lines of up to 32, 64, 128 and 256 threads' worth of three to seven rows:
// short chunks keep a lone system's latency down, and below 256 threads
// more systems share an SM.  From 256 threads on, longer chunks.
constexpr int kStreamMaxN = 256 * 19;

template <class R>
cudaError_t stream_solve(const R* a, const R* b, const R* c, const R* d, R* x, int n, int nsys, cudaStream_t st) {
  int dev = 0, nsm = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
#define IXB_STREAM_(T_, M_) \
  if (n <= T_ * M_) return stream_launch<R, T_, M_>(a, b, c, d, x, n, nsys, nsm, st);
  IXB_STREAM_(32, 3) IXB_STREAM_(32, 5)
  IXB_STREAM_(64, 3) IXB_STREAM_(64, 5)
  IXB_STREAM_(128, 3) IXB_STREAM_(128, 5)
  IXB_STREAM_(256, 3) IXB_STREAM_(256, 5) IXB_STREAM_(256, 7) IXB_STREAM_(256, 9) IXB_STREAM_(256, 11)
  IXB_STREAM_(256, 13) IXB_STREAM_(256, 15) IXB_STREAM_(256, 17) IXB_STREAM_(256, 19)
#undef IXB_STREAM_
  return cudaErrorInvalidValue;
}

}  // namespace

// ---------------------------------------------------------------------------
// Interleaved systems (row i of system s at i*nsys + s), hybrid solver.
// A CTA holds W adjacent systems: thread t the M consecutive rows of chunk
// t / W of system t % W, loaded straight into registers, so that every load
// of a warp covers W adjacent elements of 32 / W rows and no alignment is
// asked of the arrays or of nsys.
// ---------------------------------------------------------------------------
namespace {

// rows k*M .. k*M+M-1 past row0 of system s; identity rows outside
template <class R, int M, class Ld>
__device__ __forceinline__ void load_chunk(Chunk<R, M>& ch, const R* a, const R* b, const R* c, const R* d,
                                           size_t row0, int n, size_t s, int nsys, Ld ld) {
#pragma unroll
  for (int j = 0; j < M; ++j) {
    const size_t r = row0 + j;
    const bool in = s < (size_t)nsys && r < (size_t)n;
    const size_t g = in ? r * nsys + s : 0;
    ch.a[j] = in && r > 0 ? ld(a + g) : R(0);
    ch.b[j] = in ? ld(b + g) : R(1);
    ch.c[j] = in && r < (size_t)n - 1 ? ld(c + g) : R(0);
    ch.d[j] = in ? ld(d + g) : R(0);
  }
}

// Whole systems: n <= M * G rows on the G chunks of a CTA.
template <class R, int W, int M>
__global__ void __launch_bounds__(512) tri_cols_kernel(const R* a, const R* b, const R* c, const R* d, R* x, int n,
                                                       int nsys, int G) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  R* red = reinterpret_cast<R*>(smem_raw);
  const int w = threadIdx.x % W, k = threadIdx.x / W;
  const size_t s = (size_t)blockIdx.x * W + w;
  const bool active = s < (size_t)nsys;
  Chunk<R, M> ch;
  load_chunk(ch, a, b, c, d, (size_t)k * M, n, s, nsys, [](const R* p) { return *p; });
  ch.eliminate();
  R x0, xl;
  reduced_pcr<R, true>(red, W * G, W, G, threadIdx.x, k, active, ch.eA, ch.eC, ch.eD, ch.oA, ch.oC, ch.oD, x0, xl,
                       [](bool q) { return (bool)__syncthreads_or(q); });
  ch.substitute(x0, xl);
#pragma unroll
  for (int j = 0; j < M; ++j) {
    const int r = k * M + j;
    if (active && r < n) x[(size_t)r * nsys + s] = ch.d[j];
  }
}

// Blocks of 128 rows of 128 bytes' worth of systems, for lines that fit
// neither one CTA nor the cluster kernel's copies (odd nsys, n > 4096).  Two items per block, handed out in order by a ticket:
//   A: eliminate the block to its first and last rows as functions of the
//      neighbouring blocks' ends; the last A of a system group then solves
//      the group's block ends (block_ends) and raises its flag;
//   C: the same elimination from the same inputs (mostly L2 hits: C of group
//      g follows A of group g + lag), then, with the block's outer
//      neighbours known, its rows.
// DRAM sees the inputs and the solution once; nothing waits on a cluster or
// a launch boundary.  Items wait only on items with lower tickets, which
// running CTAs hold, and the wait is bounded (g_tri_timeout).  Bound by the
// latency of an item (64 KB in registers, two items per SM): 4095 x 4095
// binary64 307 us (2.19 TB/s), against 5057 us for one thread per system;
// where the cluster kernel applies it is faster (4096 x 4096: 156 against
// 305 us).
template <class R>
struct BlockCfg {
  static constexpr int T = 256;
  static constexpr int W = 128 / (int)sizeof(R);  // systems per group
  static constexpr int G = T / W;                 // chunks per block
  static constexpr int ROWS = 128;
  static constexpr int M = ROWS / G;              // rows per chunk
};

struct BlockPlan {
  int groups, blocks, lag;
  long long items;
  size_t ends, outer, ctr;  // scratch: elements of block ends and outer values, ints of counters
};

template <class R>
BlockPlan block_plan(int n, int nsys, int resident) {
  using B = BlockCfg<R>;
  BlockPlan p{};
  p.groups = (nsys + B::W - 1) / B::W;
  p.blocks = (n + B::ROWS - 1) / B::ROWS;
  // A runs ahead of C by the groups a full GPU has in flight, and two more
  p.lag = std::min(p.groups, resident / p.blocks + 2);
  p.items = 2LL * p.groups * p.blocks;
  p.ends = (size_t)p.groups * p.blocks * 6 * B::W;
  p.outer = (size_t)p.groups * p.blocks * 2 * B::W;
  p.ctr = 2 + 2 * (size_t)p.groups;
  return p;
}

template <class R>
size_t block_scratch_bytes(const BlockPlan& p) {
  return (p.ends + p.outer) * sizeof(R) + p.ctr * sizeof(unsigned);
}

// item t: group, block and whether it is a C item
__device__ __forceinline__ void block_item(long long t, int groups, int blocks, int lag, int& g, int& blk, bool& c) {
  const long long head = (long long)lag * blocks, mid = 2LL * (groups - lag) * blocks;
  if (t < head) {
    g = (int)(t / blocks); blk = (int)(t % blocks); c = false;
  } else if (t < head + mid) {
    const long long u = t - head, pos = u / (2 * blocks), v = u % (2 * blocks);
    c = v >= blocks;
    g = (int)pos + (c ? 0 : lag);
    blk = (int)(v % blocks);
  } else {
    const long long u = t - head - mid;
    g = groups - lag + (int)(u / blocks); blk = (int)(u % blocks); c = true;
  }
}

// Odd rows of a block's chunks as functions of the outer unknowns:
//   xl_k + A XL + C XF = D, XL the last unknown before the block, XF the first
// after it.  reduced_pcr with open ends: a row without a neighbour keeps its
// coupling to the outer unknown (the neighbour "row" is -x_outer).
template <class R>
__device__ __forceinline__ void block_pcr(R* red, int W, int G, int k, const R eA, const R eC, const R eD, R& oA,
                                          R& oC, R& oD) {
  const int N = W * G, pos = threadIdx.x;
  red[pos] = eA; red[N + pos] = eC; red[2 * N + pos] = eD;
  __syncthreads();
  R hA = R(0), hC = R(-1), hD = R(0);
  if (k + 1 < G) { hA = red[pos + W]; hC = red[N + pos + W]; hD = red[2 * N + pos + W]; }
  pcr_row(oA, oC, oD, eA, eC, eD, hA, hC, hD);
  R* cur = red + 3 * N;
  R* nxt = red + 6 * N;
#pragma unroll 1
  for (int h = 1; h < G; h <<= 1) {
    cur[pos] = oA; cur[N + pos] = oC; cur[2 * N + pos] = oD;
    __syncthreads();
    R lA = R(-1), lC = R(0), lD = R(0);
    hA = R(0); hC = R(-1); hD = R(0);
    if (k >= h) { const int q = pos - h * W; lA = cur[q]; lC = cur[N + q]; lD = cur[2 * N + q]; }
    if (k + h < G) { const int q = pos + h * W; hA = cur[q]; hC = cur[N + q]; hD = cur[2 * N + q]; }
    pcr_row(oA, oC, oD, lA, lC, lD, hA, hC, hD);
    R* t = cur; cur = nxt; nxt = t;
  }
  __syncthreads();  // red is free again
}

// Block ends of one system (thread w of a group): per block, first row
// f + al XL + be XF = de and last row l + A XL + C XF = D, with XL the previous
// block's l and XF the next block's f.  Forward: l_b = P_b - Q_b f_{b+1} and
// f_b = F0_b - F1_b f_{b+1}, one reciprocal per block; backward: the values,
// and each block's XL, XF.  `ends` is overwritten by (F0, F1, P, Q).
template <class R>
__device__ void block_ends(R* ends, R* outer, int W, int blocks) {
  R P = R(0), Q = R(0);
  constexpr int U = 4;  // blocks whose ends are loaded together
  for (int b0 = 0; b0 < blocks; b0 += U) {
    R v[U][6];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int q = 0; q < 6; ++q) v[u][q] = b0 + u < blocks ? __ldcg(ends + ((size_t)(b0 + u) * 6 + q) * W) : R(0);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (b0 + u >= blocks) break;
      const R al = v[u][0], be = v[u][1], de = v[u][2], A = v[u][3], Cc = v[u][4], D = v[u][5];
      const R r = fast_rcp(fmaT(-al, Q, R(1)));
      const R F0 = fmaT(-al, P, de) * r, F1 = be * r;
      const R AQ = A * Q;
      const R Pn = fmaT(AQ, F0, fmaT(-A, P, D)), Qn = fmaT(AQ, F1, Cc);
      R* e = ends + (size_t)(b0 + u) * 6 * W;
      __stcg(e, F0); __stcg(e + W, F1); __stcg(e + 2 * W, Pn); __stcg(e + 3 * W, Qn);
      P = Pn; Q = Qn;
    }
  }
  R fn = R(0);
  for (int b1 = blocks - 1; b1 >= 0; b1 -= U) {
    R v[U][4];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int b = b1 - u;
      v[u][0] = b >= 0 ? __ldcg(ends + (size_t)b * 6 * W) : R(0);
      v[u][1] = b >= 0 ? __ldcg(ends + ((size_t)b * 6 + 1) * W) : R(0);
      v[u][2] = b > 0 ? __ldcg(ends + ((size_t)(b - 1) * 6 + 2) * W) : R(0);
      v[u][3] = b > 0 ? __ldcg(ends + ((size_t)(b - 1) * 6 + 3) * W) : R(0);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int b = b1 - u;
      if (b < 0) break;
      const R f = fmaT(-v[u][1], fn, v[u][0]);
      __stcg(outer + (size_t)b * 2 * W, fmaT(-v[u][3], f, v[u][2]));
      __stcg(outer + ((size_t)b * 2 + 1) * W, fn);
      fn = f;
    }
  }
}

// Bounded wait for a flag another CTA of this launch raises.
__device__ __forceinline__ bool flag_wait_bounded(const unsigned* flag) {
  unsigned long long t0;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  for (int i = 0; i < kSpinLimit; ++i) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
    if (v) return true;
    if ((i & 63) == 63) {
      unsigned long long t;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
      if (t - t0 > 2000000000ull) return false;
    }
  }
  return false;
}

template <class R>
__global__ void __launch_bounds__(BlockCfg<R>::T, 2)
    tri_block_kernel(const R* a, const R* b, const R* c, const R* d, R* x, int n, int nsys, int groups, int blocks,
                     int lag, R* ends, R* outer, unsigned* ctr) {
  using B = BlockCfg<R>;
  constexpr int W = B::W, G = B::G, M = B::M;
  __shared__ R red[9 * B::T];
  __shared__ long long s_item;
  __shared__ int s_last;
  const int tid = threadIdx.x, w = tid % W, k = tid / W;
  unsigned long long* ticket = reinterpret_cast<unsigned long long*>(ctr);
  unsigned* done = ctr + 2;
  unsigned* flag = done + groups;
  const long long items = 2LL * groups * blocks;
  if (tid == 0) s_item = (long long)atomicAdd(ticket, 1ull);
  __syncthreads();
  long long t = s_item;
  while (t < items) {
    long long nt = 0;
    if (tid == 0) nt = (long long)atomicAdd(ticket, 1ull);  // the next ticket, while this item runs
    int g, blk;
    bool second;
    block_item(t, groups, blocks, lag, g, blk, second);
    const size_t s = (size_t)g * W + w;
    const size_t row0 = (size_t)blk * B::ROWS + k * M;
    Chunk<R, M> ch;
    if (second) load_chunk(ch, a, b, c, d, row0, n, s, nsys, [](const R* p) { return __ldcs(p); });
    else load_chunk(ch, a, b, c, d, row0, n, s, nsys, [](const R* p) { return __ldcg(p); });
    ch.eliminate();
    const R eA = ch.eA, eC = ch.eC, eD = ch.eD;
    R oA = ch.oA, oC = ch.oC, oD = ch.oD;
    block_pcr(red, W, G, k, eA, eC, eD, oA, oC, oD);
    R* my_ends = ends + ((size_t)g * blocks + blk) * 6 * W + w;
    R* my_outer = outer + ((size_t)g * blocks + blk) * 2 * W + w;
    if (!second) {
      if (k == 0) {
        __stcg(my_ends, fmaT(-eC, oA, eA));
        __stcg(my_ends + W, -eC * oC);
        __stcg(my_ends + 2 * W, fmaT(-eC, oD, eD));
      }
      if (k == G - 1) { __stcg(my_ends + 3 * W, oA); __stcg(my_ends + 4 * W, oC); __stcg(my_ends + 5 * W, oD); }
      __threadfence();
      __syncthreads();
      if (tid == 0) s_last = atomicAdd(done + g, 1u) == (unsigned)blocks - 1;
      __syncthreads();
      if (s_last) {
        __threadfence();
        if (tid < W)
          block_ends(ends + (size_t)g * blocks * 6 * W + tid, outer + (size_t)g * blocks * 2 * W + tid, W, blocks);
        __threadfence();
        __syncthreads();
        if (tid == 0) asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(flag + g), "r"(1u) : "memory");
      }
    } else {
      bool ok = true;
      if (tid == 0) ok = flag_wait_bounded(flag + g);
      if (__syncthreads_or(!ok)) {
        if (tid == 0) atomicExch(&g_tri_timeout, 1);
        return;
      }
      const R XL = __ldcg(my_outer), XF = __ldcg(my_outer + W);
      const R xl = fmaT(-oC, XF, fmaT(-oA, XL, oD));
      red[tid] = xl;
      __syncthreads();
      const R xm = k > 0 ? red[tid - W] : XL;
      const R x0 = fmaT(-eC, xl, fmaT(-eA, xm, eD));
      ch.substitute(x0, xl);
      if (s < (size_t)nsys) {
#pragma unroll
        for (int j = 0; j < M; ++j)
          if (row0 + j < (size_t)n) __stcs(x + (row0 + j) * nsys + s, ch.d[j]);
      }
    }
    if (tid == 0) s_item = nt;
    __syncthreads();
    t = s_item;
    __syncthreads();
  }
}

template <class R, int W, int M>
cudaError_t cols_launch(const R* a, const R* b, const R* c, const R* d, R* x, int n, int nsys, cudaStream_t st) {
  constexpr int Q = W < 32 ? 32 / W : 1;  // chunks that fill a warp
  const int G = ((n + M - 1) / M + Q - 1) / Q * Q;
  const size_t smem = (size_t)9 * W * G * sizeof(R);
  tri_cols_kernel<R, W, M><<<(nsys + W - 1) / W, W * G, smem, st>>>(a, b, c, d, x, n, nsys, G);
  return cudaGetLastError();
}

// Whole systems in one CTA's registers (up to 512 threads).  64-byte row
// pieces stream from HBM, 32-byte ones at under half its rate, but they put
// twice as many CTAs on a GPU that 64-byte ones leave idle: used below two
// CTAs per SM, and up to 1024 rows.
template <class R>
bool cols_fit(int n, int nsys, int nsm) {
  const int W = 64 / (int)sizeof(R);
  return n <= 512 || (n <= 1024 && (nsys + W - 1) / W < 4 * nsm);
}

template <class R>
cudaError_t cols_solve(const R* a, const R* b, const R* c, const R* d, R* x, int n, int nsys, int nsm,
                       cudaStream_t st) {
  constexpr int W1 = 64 / (int)sizeof(R), W2 = W1 / 2;  // systems per 64- and 32-byte piece
  if (n <= 512 && (nsys + W1 - 1) / W1 >= 2 * nsm) {
    if constexpr (sizeof(R) == 8) {
      return n <= 256 ? cols_launch<R, W1, 4>(a, b, c, d, x, n, nsys, st)
                      : cols_launch<R, W1, 8>(a, b, c, d, x, n, nsys, st);
    } else {
      return n <= 256 ? cols_launch<R, W1, 8>(a, b, c, d, x, n, nsys, st)
                      : cols_launch<R, W1, 16>(a, b, c, d, x, n, nsys, st);
    }
  }
  if (n <= 2048 / W2) return cols_launch<R, W2, 4>(a, b, c, d, x, n, nsys, st);
  if (sizeof(R) == 8 || n <= 4096 / W2) return cols_launch<R, W2, 8>(a, b, c, d, x, n, nsys, st);
  if constexpr (sizeof(R) == 4) return cols_launch<R, W2, 16>(a, b, c, d, x, n, nsys, st);
  return cudaErrorInvalidValue;
}

// Resident CTAs of tri_block_kernel at two per SM (its launch bound).
template <class R>
cudaError_t block_solve(const R* a, const R* b, const R* c, const R* d, R* x, int n, int nsys, int nsm,
                        const BlockPlan& p, void* scratch, cudaStream_t st) {
  R* ends = static_cast<R*>(scratch);
  R* outer = ends + p.ends;
  unsigned* ctr = reinterpret_cast<unsigned*>(outer + p.outer);  // W is even: 8-byte aligned
  cudaError_t e = cudaMemsetAsync(ctr, 0, p.ctr * sizeof(unsigned), st);
  if (e != cudaSuccess) return e;
  const int grid = (int)std::min<long long>(p.items, 2LL * nsm);
  tri_block_kernel<R><<<grid, BlockCfg<R>::T, 0, st>>>(a, b, c, d, x, n, nsys, p.groups, p.blocks, p.lag, ends, outer,
                                                       ctr);
  return cudaGetLastError();
}

// Stream-ordered scratch from pools of the library's own (one of each kind per
// device context), so that memory freed after a call is still mapped at the
// next one: with the device's default pool every synchronisation unmapped it,
// and a 0.2 ms solve that the host waits for took 4.2 ms.  What a pool keeps
// mapped across synchronisations is bounded:
//  * line solves 32 MB (the block kernel's scratch takes 8.4 MB at 4095x4095
//    binary64); larger requests, those of the exact interleaved solve, go to
//    the default pool and back to the device at the next synchronisation;
//  * a handle's gradients and energy passes 256 MB (a 128x128 gradient of the
//    coupled iteration with a checkpoint every 10 holds 21 MB: as thirty
//    cudaMalloc / cudaFree pairs its workspace cost 2 to 10 ms per call), given
//    back when the handle is destroyed.
// ixb_release_scratch gives back what is idle of both.  While `st` is captured,
// or if the pool cannot be had, the default allocator serves.
constexpr unsigned long long kPoolKeep[SCRATCH_KINDS] = {32ull << 20, 256ull << 20};
constexpr int kPoolDevices = 64;

// the pool of the current device's context; made on first use with `make`,
// else null if there is none
cudaMemPool_t scratch_pool(ScratchKind kind, int dev, bool make) {
  static std::mutex mu;
  static cudaMemPool_t pools[SCRATCH_KINDS][kPoolDevices] = {};
  static unsigned long long owners[SCRATCH_KINDS][kPoolDevices] = {};  // context the pool belongs to (0: none)
  cudaMemPool_t* const pool = pools[kind];
  unsigned long long* const owner = owners[kind];
  using CtxIdFn = CUresult (*)(CUcontext, unsigned long long*);
  static CtxIdFn ctx_id = nullptr;
  if (dev < 0 || dev >= kPoolDevices) return nullptr;
  std::lock_guard<std::mutex> lock(mu);
  if (!ctx_id) {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      ctx_id = reinterpret_cast<CtxIdFn>(f);
  }
  unsigned long long id = 0;
  if (!ctx_id || ctx_id(nullptr, &id) != CUDA_SUCCESS) return nullptr;
  if (owner[dev] != id + 1 && make) {  // first use, or the context was re-created (cudaDeviceReset)
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t made = nullptr;
    unsigned long long keep = kPoolKeep[kind];
    if (cudaMemPoolCreate(&made, &props) == cudaSuccess &&
        cudaMemPoolSetAttribute(made, cudaMemPoolAttrReleaseThreshold, &keep) == cudaSuccess) {
      pool[dev] = made;
      owner[dev] = id + 1;
    } else {
      cudaGetLastError();
    }
  }
  return owner[dev] == id + 1 ? pool[dev] : nullptr;
}
}  // namespace

cudaError_t scratch_alloc(ScratchKind kind, void** p, size_t bytes, cudaStream_t st) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if ((e = cudaStreamIsCapturing(st, &cap)) != cudaSuccess) return e;
  const bool own = cap == cudaStreamCaptureStatusNone && (kind != SCRATCH_LINES || bytes <= kPoolKeep[kind]);
  cudaMemPool_t use = own ? scratch_pool(kind, dev, true) : nullptr;
  return use ? cudaMallocFromPoolAsync(p, bytes, use, st) : cudaMallocAsync(p, bytes, st);
}

cudaError_t scratch_trim(ScratchKind kind) {
  int dev = 0;
  const cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  cudaMemPool_t pool = scratch_pool(kind, dev, false);
  return pool ? cudaMemPoolTrimTo(pool, 0) : cudaSuccess;
}

// ---------------------------------------------------------------------------
// Interleaved systems in a thread-block cluster (hybrid solver; rows of whole
// 16-byte granules, up to 4096 of them).
// A group of W adjacent systems occupies SEG = W*sizeof(R) contiguous bytes
// of every row: 128-byte segments stream from HBM at full rate, 64-byte ones
// a little below it and 32-byte ones (4 binary64 systems) at under 40 % of
// it.  A thread-block cluster of Q CTAs (one per SM) solves one group at a
// time, CTA q holding rows q*ROWS .. q*ROWS+ROWS-1 of all W systems: thread
// t owns rows k*16 .. k*16+15 (k = t / W) of system w = t % W.  Each group
// arrives as four tiles (a, b, c, d; boxes of W x 256 rows, copied by the
// tensor engine without multicast) in shared memory while the CTA is still
// solving the previous group from registers.  Every thread eliminates its
// rows (modified Thomas) to two rows coupled to the neighbouring chunks; the
// CTA sends the reduced rows of each system to its owner, cluster rank w % Q,
// by one bulk shared-to-shared copy that completes on the owner's mbarrier.
// All threads of every CTA solve the systems it owns (reduced_pcr: as many
// chunks as threads) and each CTA of the cluster gets the solutions of its
// chunks the same way; every thread back-substitutes into a solution tile
// that the tensor engine stores.  No cluster barrier: rows of the next group
// are sent only after the solutions of this one have come, so every buffer
// has been read before it is written again (each wait follows from the one
// before it).  Bound by this chain of some 7,000 cycles per group, one group
// per SM at a time, with the tile copies under it.  Every wait on a copy is bounded
// (g_tri_timeout, as above).  (SEG, ROWS) = (128, 256) for lines of up to
// 1024 rows; (64, 512) above, which halves W and so the cluster size that
// holds a group (4096 rows: 8 instead of 16 CTAs; more clusters fit the GPU).
// 4096 x 4096 binary64: 154 us, 4.4 TB/s on the 120 SMs that clusters of 8
// fill; with each owned system on one warp and the solutions read across the
// cluster between two barriers 213 us (2048 x 2048: 43.8 against 55.8).
// ---------------------------------------------------------------------------
namespace {

namespace cg = cooperative_groups;

constexpr int kStrM = 16;    // rows per thread
constexpr int kStrBox = 256;  // rows per 2-D tile box (the tensor-copy limit)

// A configuration: SEG bytes of every row per group (W = SEG / sizeof(R)
// systems) and ROWS rows per CTA, so that a cluster of Q CTAs covers
// Q * ROWS rows.  (128, 256): W = 16 / 32, clusters of up to 16 CTAs;
// (64, 512): W = 8 / 16, clusters of up to 8 (n <= 4096 in both).
template <class R, int SEG, int ROWS>
struct StridedCfg {
  static constexpr int W = SEG / (int)sizeof(R);  // systems per group
  static constexpr int C = ROWS / kStrM;          // chunks per CTA per system
  static constexpr int T = W * C;                 // threads per CTA
  static constexpr int TILE = W * ROWS;           // elements per tile
  static constexpr int BOXES = ROWS / kStrBox;    // tile boxes per array
  static constexpr int QMAX = W < 16 ? W : 16;  // every CTA of a cluster owns W / Q systems
  // an owner's reduced rows (W / Q systems of 2*C*Q rows, a | c | d per
  // sender), and in their place the working arrays of reduced_pcr once read
  static constexpr int RED = (sizeof(R) == 8 ? 9 : 12) * T;
  static constexpr int RUN = 6 * C;  // what a CTA sends of one system: a | c | d of its C chunks
};

// shared memory (bytes): 4 input tiles, the solution tile, the reduced
// systems, outgoing rows (later outgoing solutions), incoming solutions,
// 3 mbarriers (tiles, reduced rows, solutions)
template <class R, int SEG, int ROWS>
__host__ __device__ constexpr size_t strided_smem_bytes() {
  using SC = StridedCfg<R, SEG, ROWS>;
  return ((size_t)5 * SC::TILE + SC::RED + (6 + 2 + 2) * (size_t)SC::T) * sizeof(R) + 32;
}

__device__ __forceinline__ void tile_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::
          "r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ void tile_store_2d(const CUtensorMap* map, int x, int y, const void* src) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(x), "r"(y), "r"(smem_u32(src))
               : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

// shared::cluster address of `local`'s counterpart in cluster rank `rank`
__device__ __forceinline__ unsigned cluster_smem_addr(const void* local, int rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(local)), "r"(rank));
  return r;
}

// bulk copy from this CTA's shared memory to cluster shared memory,
// completing on the destination's mbarrier
__device__ __forceinline__ void bulk_send(unsigned dst, const void* src, unsigned bytes, unsigned bar) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   dst),
               "r"(smem_u32(src)), "r"(bytes), "r"(bar)
               : "memory");
}

// pairs of adjacent elements (16 bytes in binary64, 8 in binary32)
template <class R>
struct Pair2;
template <>
struct Pair2<double> { using type = double2; };
template <>
struct Pair2<float> { using type = float2; };

template <class R, int SEG, int ROWS>
__global__ void __launch_bounds__(StridedCfg<R, SEG, ROWS>::T, 1)
    tri_strided_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                       const __grid_constant__ CUtensorMap mapC, const __grid_constant__ CUtensorMap mapD,
                       const __grid_constant__ CUtensorMap mapX, int n, int nsys) {
  using SC = StridedCfg<R, SEG, ROWS>;
  using P2 = typename Pair2<R>::type;
  constexpr int W = SC::W, T = SC::T, M = kStrM, CH = SC::C;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  R* tile = reinterpret_cast<R*>(smem_raw);  // a | b | c | d, [row][system] each
  R* xt = tile + 4 * SC::TILE;               // solution tile
  R* red = xt + SC::TILE;                    // owned systems: a | c | d, 2*T each; then reduced_pcr's
  R* outr = red + SC::RED;                   // outgoing reduced rows: [system][a | c | d][chunk]
  R* outx = outr + 6 * T;                    // outgoing solutions: [owned system][chunk]
  R* xs = outx + 2 * T;                      // incoming solutions: [system][own chunk]
  uint64_t* bar = reinterpret_cast<uint64_t*>(xs + 2 * T);  // tiles
  uint64_t* rbar = bar + 1;                                 // reduced rows
  uint64_t* xbar = bar + 2;                                 // solutions
  cg::cluster_group cluster = cg::this_cluster();
  const int Q = (int)cluster.num_blocks();  // 4 .. SC::QMAX, a power of two
  const int rank = (int)cluster.block_rank();
  const int tid = threadIdx.x;
  const int w = tid % W, k = tid / W;
  const int row0 = rank * ROWS + k * M;
  const int nclusters = gridDim.x / Q;
  const int cl = blockIdx.x / Q;
  const int ngroups = (nsys + W - 1) / W;
  const bool stores = rank * ROWS < n;  // CTAs wholly past the last row store nothing
  const int G = CH * Q;  // chunks per system; the W / Q owned systems have T
  const int c = tid % G, slot = tid / G;  // the chunk this thread solves for
  P2* const my_rows = reinterpret_cast<P2*>(outr + w * SC::RUN) + k;
  const P2* const my_red = reinterpret_cast<const P2*>(red + (slot * Q + c / CH) * SC::RUN) + c % CH;
  const unsigned rows_bytes = (unsigned)(6 * T * sizeof(R)), xs_bytes = (unsigned)(2 * T * sizeof(R));
  constexpr unsigned kTileBytes = (unsigned)(SC::TILE * sizeof(R));
  auto issue = [&](int g) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // earlier reads of the tiles precede the copies
    mbar_expect_tx(bar, 4 * kTileBytes);
#pragma unroll
    for (int bx = 0; bx < SC::BOXES; ++bx) {
      const int y = rank * ROWS + bx * kStrBox, o = bx * kStrBox * W;
      tile_load_2d(tile + o, &mapA, g * W, y, bar);
      tile_load_2d(tile + SC::TILE + o, &mapB, g * W, y, bar);
      tile_load_2d(tile + 2 * SC::TILE + o, &mapC, g * W, y, bar);
      tile_load_2d(tile + 3 * SC::TILE + o, &mapD, g * W, y, bar);
    }
  };
  if (tid == 0) {
    mbar_init(bar);
    mbar_init(rbar);
    mbar_init(xbar);
    mbar_expect_tx(rbar, rows_bytes);
    mbar_expect_tx(xbar, xs_bytes);
  }
  cluster.sync();  // every CTA of the cluster runs and its mbarriers are set up
  if (tid == 0 && cl < ngroups) issue(cl);
  const int first_limit = *(volatile int*)&g_tri_first_wait_polls;
  // phase of each mbarrier that is waited for next (a wait that ran out leaves it), tiles on their way
  unsigned parity = 0, rpar = 0, xpar = 0;
  bool loading = cl < ngroups, failed = false;
  for (int g = cl; g < ngroups; g += nclusters) {
    const int sys = g * W + w;
    const bool live = sys < nsys;
    {
      const bool ok = mbar_wait_bounded(bar, parity, g == cl ? first_limit : kSpinLimit);
      if (__syncthreads_or(!ok)) { failed = true; break; }
      parity ^= 1;
    }
    // own rows into registers; row 0 has no a, row n-1 no c, and rows or
    // systems outside the problem (zeros in the tiles) become identity rows
    R ra[M], rb[M], rc[M], rd[M];
    // (64-byte rows: chunks of odd k take each pair of rows in the other
    // order, or the chunks of a warp would meet in one half of the banks; at
    // 4096 rows binary64 the loads of a group took 2490 cycles without)
    const bool swap = SEG == 64 && (k & 1);
    const int o0 = (k * M + (swap ? 1 : 0)) * W + w, o1 = (k * M + (swap ? 0 : 1)) * W + w;
    auto pair = [&](const R* t, R& first, R& second, int j) {
      const R p = t[o0 + j * W], q = t[o1 + j * W];
      first = swap ? q : p;
      second = swap ? p : q;
    };
#pragma unroll
    for (int j = 0; j < M; j += 2) {
      pair(tile, ra[j], ra[j + 1], j);
      pair(tile + SC::TILE, rb[j], rb[j + 1], j);
      pair(tile + 2 * SC::TILE, rc[j], rc[j + 1], j);
      pair(tile + 3 * SC::TILE, rd[j], rd[j + 1], j);
    }
    if (!(live && row0 >= 1 && row0 + M <= n - 1)) {
#pragma unroll
      for (int j = 0; j < M; ++j) {
        const int r = row0 + j;
        if (!(live && r < n)) {
          ra[j] = R(0); rb[j] = R(1); rc[j] = R(0); rd[j] = R(0);
        } else {
          if (r == 0) ra[j] = R(0);
          if (r == n - 1) rc[j] = R(0);
        }
      }
    }
    __syncthreads();  // the tiles are free: start loading the cluster's next group
    loading = g + nclusters < ngroups;
    if (tid == 0 && loading) issue(g + nclusters);
    // modified Thomas on the own rows (as in the contiguous kernels)
    R inv = fast_rcp(rb[1]);
    R ap = ra[1] * inv, cp = rc[1] * inv, dp = rd[1] * inv;
    ra[1] = ap; rc[1] = cp; rd[1] = dp;
#pragma unroll
    for (int j = 2; j < M; ++j) {
      const R aj = ra[j];
      const R r = fast_rcp(fmaT(-aj, cp, rb[j]));
      ap = -aj * ap * r;
      dp = fmaT(-aj, dp, rd[j]) * r;
      cp = rc[j] * r;
      ra[j] = ap; rc[j] = cp; rd[j] = dp;
    }
    R an = ra[M - 2], cn = rc[M - 2], dn = rd[M - 2];
#pragma unroll
    for (int j = M - 3; j >= 1; --j) {
      const R cj = rc[j];
      dn = fmaT(-cj, dn, rd[j]);
      an = fmaT(-cj, an, ra[j]);
      cn = -cj * cn;
      ra[j] = an; rc[j] = cn; rd[j] = dn;
    }
    const R r0 = fast_rcp(fmaT(-rc[0], an, rb[0]));
    const R eA = ra[0] * r0, eC = -rc[0] * cn * r0, eD = fmaT(-rc[0], dn, rd[0]) * r0;
    my_rows[0] = P2{eA, ap};
    my_rows[CH] = P2{eC, cp};
    my_rows[2 * CH] = P2{eD, dp};
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // generic accesses -> copy engine
    __syncthreads();
    if (tid < W)
      bulk_send(cluster_smem_addr(red + ((tid / Q) * Q + rank) * SC::RUN, tid % Q), outr + tid * SC::RUN,
                (unsigned)(SC::RUN * sizeof(R)), cluster_smem_addr(rbar, tid % Q));
    {
      const bool ok = mbar_wait_bounded(rbar, rpar);
      if (__syncthreads_or(!ok)) { failed = true; break; }
      rpar ^= 1;
    }
    {
      const P2 A = my_red[0], C = my_red[CH], D = my_red[2 * CH];
      __syncthreads();
      R x0, xl;
      reduced_pcr<R, sizeof(R) == 8>(red, T, 1, G, tid, c, true, A.x, C.x, D.x, A.y, C.y, D.y, x0, xl,
                                     [](bool q) { return (bool)__syncthreads_or(q); });
      reinterpret_cast<P2*>(outx)[tid] = P2{x0, xl};
    }
    if (tid == 0) {
      mbar_expect_tx(rbar, rows_bytes);  // the next group's rows come only after these solutions
      bulk_store_wait_read();            // the previous solution tile has been read out
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // generic accesses -> copy engine
    __syncthreads();
    if (tid < W)  // owned system tid / Q, the chunks of rank tid % Q
      bulk_send(cluster_smem_addr(xs + ((tid / Q) * Q + rank) * 2 * CH, tid % Q),
                outx + 2 * ((tid / Q) * G + (tid % Q) * CH), (unsigned)(2 * CH * sizeof(R)),
                cluster_smem_addr(xbar, tid % Q));
    {
      const bool ok = mbar_wait_bounded(xbar, xpar);
      if (__syncthreads_or(!ok)) { failed = true; break; }
      xpar ^= 1;
    }
    if (tid == 0) mbar_expect_tx(xbar, xs_bytes);  // the next ones come only after the rows sent below
    const P2 sol = reinterpret_cast<const P2*>(xs)[w * CH + k];
    const R x0 = sol.x, xl = sol.y;
    auto row = [&](int j) { return j == 0 ? x0 : (j == M - 1 ? xl : fmaT(-rc[j], xl, fmaT(-ra[j], x0, rd[j]))); };
#pragma unroll
    for (int j = 0; j < M; j += 2) {
      const R p = row(j), q = row(j + 1);
      xt[o0 + j * W] = swap ? q : p;
      xt[o1 + j * W] = swap ? p : q;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // generic writes -> tensor engine
    __syncthreads();
    // rows past n and systems past nsys fall outside the map and are not written
    if (tid == 0 && stores) {
#pragma unroll
      for (int bx = 0; bx < SC::BOXES; ++bx)
        if (rank * ROWS + bx * kStrBox < n) tile_store_2d(&mapX, g * W, rank * ROWS + bx * kStrBox, xt + bx * kStrBox * W);
    }
  }
  cluster.sync();  // no CTA of the cluster sends any more
  if (tid == 0) {
    if (failed) {
      atomicExch(&g_tri_timeout, 1);
      // copies still in flight land before the CTA leaves (the last two waits
      // run out if nothing more was sent)
      if (loading) mbar_wait_bounded(bar, parity);
      mbar_wait_bounded(rbar, rpar);
      mbar_wait_bounded(xbar, xpar);
    }
    bulk_store_wait_all();
  }
  cluster.sync();  // no CTA leaves while the copy engine may still read its shared memory
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no
// link-time dependence on the driver library)
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

// [n rows][nsys systems] in boxes of W systems x 256 rows; rows and systems
// past the ends read as zeros and are not written
template <class R>
bool strided_map(CUtensorMap* map, const R* p, int n, int nsys, int W) {
  const EncodeTiledFn fn = encode_tiled();
  if (!fn) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)nsys, (cuuint64_t)n};
  const cuuint64_t strides[1] = {(cuuint64_t)nsys * sizeof(R)};
  const cuuint32_t box[2] = {(cuuint32_t)W, (cuuint32_t)kStrBox};
  const cuuint32_t estr[2] = {1, 1};
  const CUtensorMapDataType dt = sizeof(R) == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  return fn(map, dt, 2, const_cast<R*>(p), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// cudaErrorInvalidValue: outside the configuration's range (n above
// QMAX * ROWS rows, or no room for a cluster of Q CTAs)
template <class R, int SEG, int ROWS>
cudaError_t strided_launch(const R* a, const R* b, const R* c, const R* d, R* x, int n, int nsys, cudaStream_t st) {
  using SC = StridedCfg<R, SEG, ROWS>;
  int Q = 4;  // CTAs per cluster: a power of two >= 4; each owns W / Q systems of a group
  while (Q * ROWS < n) Q <<= 1;
  if (Q > SC::QMAX) return cudaErrorInvalidValue;
  CUtensorMap maps[5];
  if (!strided_map(&maps[0], a, n, nsys, SC::W) || !strided_map(&maps[1], b, n, nsys, SC::W) ||
      !strided_map(&maps[2], c, n, nsys, SC::W) || !strided_map(&maps[3], d, n, nsys, SC::W) ||
      !strided_map(&maps[4], static_cast<const R*>(x), n, nsys, SC::W))
    return cudaErrorInvalidValue;
  auto k = tri_strided_kernel<R, SEG, ROWS>;
  const size_t smem = strided_smem_bytes<R, SEG, ROWS>();
  cudaError_t e = allow_smem(k, 0);
  if (e != cudaSuccess) return e;
  if (Q > 8 && (e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)) != cudaSuccess)
    return e;
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = Q;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.blockDim = dim3(SC::T);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cfg.gridDim = dim3(Q);
  int max_clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&max_clusters, k, &cfg) != cudaSuccess || max_clusters < 1) {
    cudaGetLastError();
    return cudaErrorInvalidValue;
  }
  const int ngroups = (nsys + SC::W - 1) / SC::W;
  cfg.gridDim = dim3(Q * std::min(ngroups, max_clusters));
  e = cudaLaunchKernelEx(&cfg, k, maps[0], maps[1], maps[2], maps[3], maps[4], n, nsys);
  if (e != cudaSuccess) return e;
  return cudaGetLastError();
}

// IXB_STRIDED_SEG=64 or 128 forces one configuration; otherwise lines of
// more than 1024 rows use 64-byte segments with 512-row CTAs (half the CTAs
// per cluster, so more clusters fit the GPU at once: binary64 1500 x 1500
// 33.2 against 39.3 us, 4096 x 4096 153 against 167), shorter lines 128-byte
// segments with 256-row CTAs (less padding).
int strided_seg_choice() {
  static const int v = [] {
    const char* e = std::getenv("IXB_STRIDED_SEG");
    return e ? std::atoi(e) : 0;
  }();
  return v;
}

// cudaErrorInvalidValue: outside the kernels' range (n > 4096 rows, a row
// pitch or base address the tensor copies cannot take, or no room for a
// cluster); the caller then uses the general interleaved kernel
template <class R>
cudaError_t strided_solve(const R* a, const R* b, const R* c, const R* d, R* x, int n, int nsys, cudaStream_t st) {
  if (n < 1 || n > 16 * kStrBox || nsys < 1) return cudaErrorInvalidValue;
  const uintptr_t all = (uintptr_t)a | (uintptr_t)b | (uintptr_t)c | (uintptr_t)d | (uintptr_t)x;
  if ((all & 15) != 0 || ((size_t)nsys * sizeof(R)) % 16 != 0) return cudaErrorInvalidValue;
  const int seg = strided_seg_choice();
  if (seg == 64 || (seg != 128 && n > 4 * kStrBox)) {
    const cudaError_t e = strided_launch<R, 64, 512>(a, b, c, d, x, n, nsys, st);
    if (e != cudaErrorInvalidValue) return e;
  }
  return strided_launch<R, 128, 256>(a, b, c, d, x, n, nsys, st);
}

}  // namespace

template <class R, int SOLVER, int TL>
static cudaError_t contig_tl(const R* a, const R* b, const R* c, const R* d, R* x, int n, int nsys, int m, int mp,
                             size_t smem, cudaStream_t st) {
  auto k = tri_contig_kernel<R, SOLVER, TL, 256 / TL>;
  cudaError_t e = allow_smem(k, 0);
  if (e != cudaSuccess) return e;
  const int grid = (nsys + TL - 1) / TL;
  k<<<grid, 256, smem, st>>>(a, b, c, d, x, n, nsys, m, mp);
  return cudaGetLastError();
}

template <class R, int SOLVER>
static cudaError_t tridiag_contig(const R* a, const R* b, const R* c, const R* d, R* x, int n, int nsys,
                                  cudaStream_t st) {
  if (SOLVER == IXB_SOLVER_HYBRID && n <= kStreamMaxN) return stream_solve(a, b, c, d, x, n, nsys, st);
  int g = 32;
  while (g < 256 && 3 * g < n) g <<= 1;
  const int tl = 256 / g;
  const int m = std::max(3, (n + g - 1) / g);
  const int mp = m | 1;
  const size_t smem = line_smem_elems(g, mp) * sizeof(R) * tl;
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (smem > (size_t)optin) return cudaErrorInvalidValue;  // line too long for one CTA
  if constexpr (SOLVER == IXB_SOLVER_EXACT) {
    switch (tl) {
      case 2: return contig_tl<R, SOLVER, 2>(a, b, c, d, x, n, nsys, m, mp, smem, st);
      case 4: return contig_tl<R, SOLVER, 4>(a, b, c, d, x, n, nsys, m, mp, smem, st);
      case 8: return contig_tl<R, SOLVER, 8>(a, b, c, d, x, n, nsys, m, mp, smem, st);
      default: break;
    }
  }
  return contig_tl<R, SOLVER, 1>(a, b, c, d, x, n, nsys, m, mp, smem, st);
}

// Interleaved systems.  fixed: scratch of at least fixed_bytes the caller
// owns (the allocation-free entry point), or null to allocate what is needed.
template <class R, int SOLVER>
static cudaError_t tridiag_inter(const R* a, const R* b, const R* c, const R* d, R* x, int n, int nsys,
                                 cudaStream_t st, void* fixed = nullptr, size_t fixed_bytes = 0) {
  int dev = 0, nsm = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  BlockPlan plan{};
  size_t bytes = (size_t)n * nsys * sizeof(R);
  if (SOLVER == IXB_SOLVER_HYBRID) {
    if (cols_fit<R>(n, nsys, nsm)) return cols_solve(a, b, c, d, x, n, nsys, nsm, st);
    const cudaError_t es = strided_solve(a, b, c, d, x, n, nsys, st);
    if (es != cudaErrorInvalidValue) return es;  // otherwise: outside the cluster kernel's range
    plan = block_plan<R>(n, nsys, 2 * nsm);
    bytes = block_scratch_bytes<R>(plan);
  }
  void* work = fixed;
  // a few very long systems: the block ends, padded to whole groups, can
  // exceed the fixed array, which always holds the sequential solve's scratch
  const bool sequential = SOLVER == IXB_SOLVER_EXACT || (fixed && bytes > fixed_bytes);
  if (!fixed && (e = scratch_alloc(SCRATCH_LINES, &work, bytes, st)) != cudaSuccess) return e;
  if (!sequential) {
    e = block_solve(a, b, c, d, x, n, nsys, nsm, plan, work, st);
  } else {
    tri_inter_kernel<R><<<(nsys + 127) / 128, 128, 0, st>>>(a, b, c, d, x, static_cast<R*>(work), n, nsys);
    e = cudaGetLastError();
  }
  if (fixed) return e;
  const cudaError_t e2 = cudaFreeAsync(work, st);
  return e != cudaSuccess ? e : e2;
}

template <class R, int SOLVER>
static cudaError_t tridiag_impl(const R* a, const R* b, const R* c, const R* d, R* x, int n, int nsys, int layout,
                                cudaStream_t st) {
  return layout == 0 ? tridiag_contig<R, SOLVER>(a, b, c, d, x, n, nsys, st)
                     : tridiag_inter<R, SOLVER>(a, b, c, d, x, n, nsys, st);
}

// Reads and clears the timeout flag the streamed and interleaved kernels set
// when a bounded wait on their copies expires (synchronous).
cudaError_t tridiag_take_timeout(int* flag) {
  int v = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&v, g_tri_timeout, sizeof(int));
  if (e != cudaSuccess) return e;
  if (v) {
    const int zero = 0;
    if ((e = cudaMemcpyToSymbol(g_tri_timeout, &zero, sizeof(int))) != cudaSuccess) return e;
  }
  *flag = v;
  return cudaSuccess;
}

cudaError_t tridiag_set_first_wait_polls(int polls) {
  const int v = polls < 0 ? kSpinLimit : polls;
  return cudaMemcpyToSymbol(g_tri_first_wait_polls, &v, sizeof(int));
}

cudaError_t tridiag_f64(const double* a, const double* b, const double* c, const double* d, double* x, int n,
                        int nsys, int layout, int solver, cudaStream_t st) {
  if (solver == IXB_SOLVER_EXACT) return tridiag_impl<double, IXB_SOLVER_EXACT>(a, b, c, d, x, n, nsys, layout, st);
  return tridiag_impl<double, IXB_SOLVER_HYBRID>(a, b, c, d, x, n, nsys, layout, st);
}

cudaError_t tridiag_f32(const float* a, const float* b, const float* c, const float* d, float* x, int n, int nsys,
                        int layout, int solver, cudaStream_t st) {
  if (solver == IXB_SOLVER_EXACT) return tridiag_impl<float, IXB_SOLVER_EXACT>(a, b, c, d, x, n, nsys, layout, st);
  return tridiag_impl<float, IXB_SOLVER_HYBRID>(a, b, c, d, x, n, nsys, layout, st);
}

}  // namespace ixb

// ===========================================================================
// Allocation-free variant of ixb_tridiag_f64.
//
// Some callers cannot let a library allocate device memory while they run:
// a Fortran driver whose GPU memory is owned by its OpenACC runtime or by a
// pool it reserved at start-up, a solver sharing a GPU under a fixed memory
// budget where an allocation in mid-run can fail, or a loop that must not
// pay the implicit synchronisation that cudaMalloc/cudaFree may cause.  For
// them, the interleaved layout keeps its scratch in a fixed array that is
// part of this library's device image (allocated by the driver together
// with the library's code, once per GPU, and held until the process exits).
// ===========================================================================
namespace ixb {
namespace {

// Scratch of the interleaved solve: IXB_NOALLOC_MAX_ELEMS doubles (8 MiB).
__device__ __align__(256) double g_noalloc_scratch[IXB_NOALLOC_MAX_ELEMS];

constexpr int kMaxDevices = 64;
double* g_noalloc_ptr[kMaxDevices] = {};
std::mutex g_noalloc_mutex;

// Device address of the scratch array for the current device.  In host code
// the name g_noalloc_scratch denotes a host-side shadow, not device memory,
// so the address is looked up with that device current.  Outside stream
// capture it is looked up on every call (a context destroyed and re-created,
// e.g. after cudaDeviceReset, reloads the module at another address); while
// `st` is capturing, the address of the last uncaptured call on this device
// is used, so the first call on a device must come before any capture.
cudaError_t noalloc_scratch(cudaStream_t st, double** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  e = cudaStreamIsCapturing(st, &cap);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (cap == cudaStreamCaptureStatusNone) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return e;
    g_noalloc_ptr[dev] = static_cast<double*>(p);
  } else if (!g_noalloc_ptr[dev]) {
    return cudaErrorStreamCaptureUnsupported;
  }
  *out = g_noalloc_ptr[dev];
  return cudaSuccess;
}

}  // namespace
}  // namespace ixb

extern "C" int ixb_tridiag_f64_noalloc(const double* a, const double* b, const double* c, const double* d, double* x,
                                       int n, int nsys, int layout, int solver, void* stream) {
  using namespace ixb;
  if (!a || !b || !c || !d || !x || n < 1 || nsys < 1 || (layout != 0 && layout != 1)) return IXB_EINVAL;
  if (solver != IXB_SOLVER_HYBRID && solver != IXB_SOLVER_EXACT) return IXB_EINVAL;
  cudaStream_t st = (cudaStream_t)stream;
  cudaError_t e;
  if (layout == 0) {
    // contiguous systems are staged in shared memory: no scratch at all
    e = solver == IXB_SOLVER_EXACT ? tridiag_impl<double, IXB_SOLVER_EXACT>(a, b, c, d, x, n, nsys, 0, st)
                                   : tridiag_impl<double, IXB_SOLVER_HYBRID>(a, b, c, d, x, n, nsys, 0, st);
  } else {
    if ((size_t)n * (size_t)nsys > (size_t)IXB_NOALLOC_MAX_ELEMS) return IXB_EINVAL;
    double* work = nullptr;
    e = noalloc_scratch(st, &work);
    if (e == cudaSuccess) {
      // every element is written (or cleared) before it is read
      const size_t bytes = (size_t)IXB_NOALLOC_MAX_ELEMS * sizeof(double);
      e = solver == IXB_SOLVER_EXACT
              ? tridiag_inter<double, IXB_SOLVER_EXACT>(a, b, c, d, x, n, nsys, st, work, bytes)
              : tridiag_inter<double, IXB_SOLVER_HYBRID>(a, b, c, d, x, n, nsys, st, work, bytes);
    }
  }
  if (e == cudaErrorInvalidValue) return IXB_EINVAL;
  return e == cudaSuccess ? IXB_OK : IXB_ECUDA;
}

// The memory of work still in flight is not idle, hence the wait.
extern "C" int ixb_release_scratch(void) {
  if (cudaDeviceSynchronize() != cudaSuccess) return IXB_ECUDA;
  for (int k = 0; k < ixb::SCRATCH_KINDS; ++k)
    if (ixb::scratch_trim((ixb::ScratchKind)k) != cudaSuccess) return IXB_ECUDA;
  return IXB_OK;
}

// Failure-detection hook (no counterpart in the reference): the poll limit of
// the first copy wait of every CTA of the streamed contiguous solve and of the
// interleaved solve in clusters.
extern "C" int ixb_tridiag_set_first_wait_limit(int polls) {
  return ixb::tridiag_set_first_wait_polls(polls) == cudaSuccess ? IXB_OK : IXB_ECUDA;
}
