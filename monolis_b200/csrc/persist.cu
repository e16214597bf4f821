// persist.cu -- CG (FP64, and FP32 with FP64 refresh) and FP64 BiCGSTAB as ONE
// cooperative kernel for the whole solve.
//
// A kernel per phase (solve.cu) costs 7 to 8 us a phase however small the
// system is (launch, entry, two-level reduction, drain); here the blocks stay
// resident, one per SM, and a phase ends in a grid exchange (grid_exchange).
// Block b owns a contiguous run of slices for the whole solve, so every vector
// entry is written by one block only. CG keeps its search direction in the
// block's shared memory over the band of columns the block's rows reach (the
// window) and forms p = z + beta p there from the z that the other blocks have
// written, so p never goes through memory; where the window does not fit, and
// in BiCGSTAB, products gather from global memory. The block's parts of the
// other vectors, and slices of the matrix, stay in shared memory as far as
// they fit.
//
// Arithmetic is that of solve.cu, expression by expression: FP64 row sums in
// CSR order, two roundings per a*b + c, dot products in double-double. The
// partial sums are grouped otherwise and renormalised less often, so a dot
// product rounds to the same bits unless its exact value lies within a few n
// eps^2 sum |x_i y_i| of a rounding boundary; every solve compared had the bits
// of the kernels per phase.
#include <algorithm>
#include <cstdio>

#include "krylov.cuh"
#include "spmv.cuh"

namespace mb {
namespace {

// ---------------------------------------------------------------------------
// Grid exchange
// ---------------------------------------------------------------------------
constexpr int kMaxBlocks = 160;  // one block per SM
constexpr int kMaxWords = 4;     // two double-double sums

// Partial sums [parity][word][block]: a block reaches exchange k + 2 only after
// every block has arrived at k + 1, so after every block has read k.
struct ExchangeSlots {
  double w[2][kMaxWords][kMaxBlocks];
  unsigned long long arrived;
  unsigned int finished;  // blocks that have written their part of X
};
struct ExchangeShared {
  double warp[32][kMaxWords];  // partial sums of this block's warps
  int ok;
};
struct Exchange {
  ExchangeSlots* slots;
  unsigned long long limit;     // polls before a wait gives up
  unsigned long long delay_at;  // testing that: block 0 arrives delay_ns late where target is this (0: nowhere)
  unsigned int delay_ns;
  unsigned long long target = 0;
  int parity = 0;
};

// release / acquire at GPU scope (__threadfence is the costlier sequentially
// consistent fence)
__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// (hi, lo) += (h2, l2) without renormalising: the error of the leading sum is
// exact (TwoSum) and the low parts are added in double, so a tree of a few
// levels loses a few eps^2 of the sum of the absolute partial sums (under
// cancellation that is more of the result than dd_merge loses); its chain is
// one addition a level where dd_merge's is ten, which is what a reduction over
// lanes waits for.
__device__ __forceinline__ void dd_merge_raw(double& hi, double& lo, double h2, double l2) {
  double s, e;
  two_sum(hi, h2, s, e);
  lo = __dadd_rn(__dadd_rn(lo, l2), e);
  hi = s;
}
__device__ __forceinline__ void dd_renorm(double& hi, double& lo) {
  double s, e;
  two_sum(hi, lo, s, e);
  hi = s;
  lo = e;
}
// sums over groups of n lanes (a power of two), in every lane
template <int K>
__device__ __forceinline__ void warp_total(PlainAcc<K>& v, int n = 32) {
  for (int o = n >> 1; o > 0; o >>= 1)
#pragma unroll
    for (int k = 0; k < K; k++) v.s[k] += __shfl_xor_sync(0xffffffffu, v.s[k], o);
}
template <int K>
__device__ __forceinline__ void warp_total(DDAcc<K>& v, int n = 32) {
  for (int o = n >> 1; o > 0; o >>= 1)
#pragma unroll
    for (int k = 0; k < K; k++) {
      const double h = __shfl_xor_sync(0xffffffffu, v.hi[k], o), l = __shfl_xor_sync(0xffffffffu, v.lo[k], o);
      dd_merge_raw(v.hi[k], v.lo[k], h, l);
    }
#pragma unroll
  for (int k = 0; k < K; k++) dd_renorm(v.hi[k], v.lo[k]);
}
template <class A>
struct AccWords;
template <int K>
struct AccWords<PlainAcc<K>> {
  static constexpr int n = K;
  static __device__ __forceinline__ double get(const PlainAcc<K>& v, int i) { return v.s[i]; }
  static __device__ __forceinline__ void set(PlainAcc<K>& v, int i, double x) { v.s[i] = x; }
  static __device__ __forceinline__ void add(PlainAcc<K>& v, const PlainAcc<K>& o) {
#pragma unroll
    for (int k = 0; k < K; k++) v.s[k] += o.s[k];
  }
  static __device__ __forceinline__ double total(const PlainAcc<K>& v, int k) { return v.s[k]; }
};
template <int K>
struct AccWords<DDAcc<K>> {
  static constexpr int n = 2 * K;
  static __device__ __forceinline__ double get(const DDAcc<K>& v, int i) { return i & 1 ? v.lo[i >> 1] : v.hi[i >> 1]; }
  static __device__ __forceinline__ void set(DDAcc<K>& v, int i, double x) {
    if (i & 1) v.lo[i >> 1] = x;
    else v.hi[i >> 1] = x;
  }
  static __device__ __forceinline__ void add(DDAcc<K>& v, const DDAcc<K>& o) {
#pragma unroll
    for (int k = 0; k < K; k++) dd_merge_raw(v.hi[k], v.lo[k], o.hi[k], o.lo[k]);
  }
  static __device__ __forceinline__ double total(const DDAcc<K>& v, int k) { return __dadd_rn(v.hi[k], v.lo[k]); }
};

// Arrival and wait of warp 0's lane 0: everything the block has written (its
// threads have met at a block barrier) is visible to every block that passes.
__device__ __forceinline__ bool arrive_and_wait(Exchange& x) {
  unsigned long long v, n = 0;
  // (compared whole, the words cost up to 1 us an iteration, by the code laid
  // out around them: 8^3 refined 11.8 against 10.7)
  if ((unsigned int)x.target == (unsigned int)x.delay_at && blockIdx.x == 0) {
#pragma unroll 1
    for (unsigned int t = 0; t < x.delay_ns; t += 1000) __nanosleep(1000);
  }
  fence_gpu();
  asm volatile("red.relaxed.gpu.global.add.u64 [%0], 1;" ::"l"(&x.slots->arrived) : "memory");
  bool ok = true;
  for (;;) {
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(&x.slots->arrived) : "memory");
    if (v >= x.target) break;
    if (++n > x.limit) {
      ok = false;
      break;
    }
  }
  fence_gpu();
  return ok;
}

// Grid barrier of a cooperative launch with a sum of A over all threads: every
// block publishes its partial sums, arrives at one counter and, once all have,
// reads all partial sums and adds them in the same order as every other block;
// fin(totals) then runs on thread 0 of every block, on identical bits, so no
// result has to be sent back. On B200, 148 blocks: 3500 cycles (1.85 us) for
// store, arrival, wait and reading back; polling the blocks' slots instead of
// a counter took 5800 (the pollers delay the stores), pushing the sums to
// every block 4900. A wait is bounded; false (in every thread) where this
// block's has run out. It has arrived all the same, so blocks that come later
// pass and only miss it at the next exchange: after the last one they end the
// solve without it, which is why the verdict waits for `publish`.
template <class A, class F>
__device__ __forceinline__ bool grid_exchange(Exchange& x, ExchangeShared& sh, A v, F&& fin) {
  using W = AccWords<A>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int G = gridDim.x;
  x.target += G;
  x.parity ^= 1;
  warp_total(v);
  if (lane == 0)
#pragma unroll
    for (int i = 0; i < W::n; i++) sh.warp[warp][i] = W::get(v, i);
  __syncthreads();
  if (warp == 0) {
    double(*slot)[kMaxBlocks] = x.slots->w[x.parity];
#pragma unroll
    for (int i = 0; i < W::n; i++) W::set(v, i, lane < nw ? sh.warp[lane][i] : 0.0);
    warp_total(v, nw > 16 ? 32 : (nw > 8 ? 16 : 8));
    bool ok = true;
    if (lane == 0) {
#pragma unroll
      for (int i = 0; i < W::n; i++) __stcg(&slot[i][blockIdx.x], W::get(v, i));
      ok = arrive_and_wait(x);
    }
    __syncwarp();
    A t;
    double w[5][W::n];
#pragma unroll
    for (int q = 0; q < 5; q++)
#pragma unroll
      for (int i = 0; i < W::n; i++) w[q][i] = q * 32 + lane < G ? __ldcg(&slot[i][q * 32 + lane]) : 0.0;
#pragma unroll
    for (int q = 0; q < 5; q++) {
      A o;
#pragma unroll
      for (int i = 0; i < W::n; i++) W::set(o, i, w[q][i]);
      if (q == 0) t = o;
      else W::add(t, o);
    }
    warp_total(t);
    if (lane == 0) {
      sh.ok = ok;
      fin([&](int k) { return W::total(t, k); });
    }
  }
  __syncthreads();
  return sh.ok != 0;
}

// The same without a sum.
__device__ __forceinline__ bool grid_barrier(Exchange& x, ExchangeShared& sh) {
  x.target += gridDim.x;
  x.parity ^= 1;
  __syncthreads();
  if (threadIdx.x == 0) sh.ok = arrive_and_wait(x);
  __syncthreads();
  return sh.ok != 0;
}

// ---------------------------------------------------------------------------
// The block's rows
// ---------------------------------------------------------------------------
// Vectors are written by the launch that reads them: no __restrict__ (the
// read-only path is not coherent), plain loads (each exchange makes the SM's
// L1 refetch).
template <class T>
struct PersistArgs {
  SellView<double> A64;
  SellView2 A32;
  const long long* slptr;  // slice offsets of the loop precision's layout
  int N, prec;
  int below, above;  // band: columns of row i lie in [i - below, i + above]
  const double* b;
  double* x;
  const T* alu;
  T* own[7];   // global room for the block's own vectors that do not fit in shared memory
  T *z, *zt;   // vectors read by other blocks: z (CG), pt and st (BiCGSTAB)
  T* y;        // FP32 correction where the refresh reads it (refined solves)
  SolverState* st;
  double* hist;
  ExchangeSlots* slots;
  unsigned long long limit, delay_at;
  unsigned int delay_ns;
  int per;       // slices of a block, at most
  int win_rows;  // rows of a window, at most
  int cb_cap;    // column bases kept in shared memory
  int win_at;    // byte offset of the window
  int smem;      // dynamic shared memory, bytes
};

template <class T>
__host__ __device__ constexpr int slice_rows() { return sizeof(T) == 8 ? 32 : 64; }
template <class T>
struct Loop;
template <>
struct Loop<double> {
  using Val = double;
  using Idx = int;
};
template <>
struct Loop<float> {
  using Val = float2;
  using Idx = int2;
};

// Shared memory of a block: slice offsets (with the flag bits of slc), widths,
// the slices' first column base, the column bases where they fit, and row
// (pair) lengths, so that the addresses of every matrix load are known without
// a dependent load; then the window; then the own vectors that still fit; then
// slices of the matrix. The arrays are addressed from the arguments, not
// through kept pointers: registers are what the products run out of.
extern __shared__ __align__(16) unsigned char g_smem[];
__host__ __device__ constexpr int up16(int b) { return (b + 15) & ~15; }
__host__ __device__ inline int meta_bytes(int per, int cb_cap) { return up16(per * 16 + cb_cap * 4 + per * 64); }
template <class T>
struct BlockRows {
  int s0, n;   // first slice, slices
  int r0, r1;  // rows
  int w0, w1;  // rows of the window
  const long long* off;
  const int* wid;
  const int* cb0;
  const int* cb;  // null: read from global memory
  const unsigned short* len;
  T* win;    // the window, indexed by the vector's own index
  int used;  // shared memory taken so far
  int ncache;  // slices kept in shared memory
  const unsigned char* cval;
};
// bytes of a slot of a slice kept in shared memory
template <int B, class T>
__host__ __device__ constexpr int cache_slot() { return 32 * (B * B * 8 + (sizeof(T) == 8 ? 4 : 8)); }

template <int B, bool kWin, class T>
__device__ __forceinline__ BlockRows<T> block_rows(const PersistArgs<T>& a) {
  constexpr int H = slice_rows<T>();
  const int nsl = (a.N + H - 1) / H;
  BlockRows<T> m;
  m.s0 = (int)((long long)nsl * blockIdx.x / gridDim.x);
  m.n = (int)((long long)nsl * (blockIdx.x + 1) / gridDim.x) - m.s0;
  m.r0 = m.s0 * H;
  m.r1 = min(a.N, (m.s0 + m.n) * H);
  m.w0 = kWin ? max(0, m.r0 - a.below) & ~3 : m.r0;  // whole 16-byte words
  m.w1 = kWin ? (int)min((long long)a.N, (long long)m.r1 + a.above) : m.r1;
  const long long* slc;
  const int* cbg;
  const int* rowptr;
  if constexpr (sizeof(T) == 8) {
    slc = a.A64.slc;
    cbg = a.A64.cbase;
    rowptr = a.A64.rowptr;
  } else {
    slc = a.A32.slc2;
    cbg = a.A32.cbase2;
    rowptr = a.A32.rowptr;
  }
  const long long p0 = a.slptr[m.s0], p1 = a.slptr[m.s0 + m.n];
  const bool fits = (p1 - p0) / H <= a.cb_cap;
  long long* off = reinterpret_cast<long long*>(g_smem);
  int* wid = reinterpret_cast<int*>(off + a.per);
  int* cb0 = wid + a.per;
  int* cb = cb0 + a.per;
  unsigned short* len = reinterpret_cast<unsigned short*>(cb + a.cb_cap);
  for (int s = threadIdx.x; s < m.n; s += blockDim.x) {
    off[s] = slc[m.s0 + s];
    wid[s] = (int)((a.slptr[m.s0 + s + 1] - a.slptr[m.s0 + s]) / H);
    cb0[s] = (int)((a.slptr[m.s0 + s] - p0) / H);
  }
  for (int i = threadIdx.x; i < m.n * 32; i += blockDim.x) {
    int l = 0;
    if constexpr (sizeof(T) == 8) {
      const int row = m.s0 * 32 + i;
      if (row < a.N) l = rowptr[row + 1] - rowptr[row];
    } else {
      const int row = 2 * (m.s0 * 32 + i);
      if (row < a.N) l = rowptr[row + 1] - rowptr[row];
      if (row + 1 < a.N) l = max(l, rowptr[row + 2] - rowptr[row + 1]);
    }
    len[i] = (unsigned short)l;
  }
  if (fits)
    for (int i = threadIdx.x; i < (int)((p1 - p0) / H); i += blockDim.x) cb[i] = cbg[p0 / H + i];
  m.off = off;
  m.wid = wid;
  m.cb0 = cb0;
  m.cb = fits ? cb : nullptr;
  m.len = len;
  m.win = reinterpret_cast<T*>(g_smem + a.win_at) - (long long)m.w0 * B;
  m.used = a.win_at + up16(a.win_rows * B * (int)sizeof(T));
  m.ncache = 0;
  m.cval = g_smem;
  return m;
}

// The block's part of one of its own vectors, indexed by the vector's own
// index: in shared memory if there is room left, else a.own[k].
template <int B, class T>
__device__ __forceinline__ T* own_vector(const PersistArgs<T>& a, BlockRows<T>& m, int k) {
  const int bytes = up16(a.per * slice_rows<T>() * B * (int)sizeof(T));
  if (m.used + bytes > a.smem) return a.own[k];
  T* p = reinterpret_cast<T*>(g_smem + m.used) - (long long)m.r0 * B;
  m.used += bytes;
  return p;
}

// U slots of a lane: column words as loaded (decoded where they are used, so
// that nothing waits for the loads) and values.
template <int B, int U, class T>
struct Chunk {
  typename Loop<T>::Idx j[U];
  typename Loop<T>::Val a[U][B * B];
};

// Where a warp stands in its slices: slice s (of the block), slots from k.
struct Cursor {
  int s, k, w, len;
  long long sc;
  const int* cb;  // column bases of the slice
};
template <class T>
__device__ __forceinline__ void open_slice(const PersistArgs<T>& a, const BlockRows<T>& m, Cursor& q) {
  q.k = 0;
  if (q.s >= m.n) return;
  q.w = m.wid[q.s];
  q.len = m.len[q.s * 32 + (threadIdx.x & 31)];
  q.sc = m.off[q.s];
  if constexpr (sizeof(T) == 8) q.cb = m.cb ? m.cb + m.cb0[q.s] : a.A64.cbase + (q.sc >> 5);
  else q.cb = m.cb ? m.cb + m.cb0[q.s] : a.A32.cbase2 + (q.sc >> 6);
}
// U slots on; a slice without slots counts as one (empty) chunk
template <int U, class T>
__device__ __forceinline__ void advance(const PersistArgs<T>& a, const BlockRows<T>& m, Cursor& q) {
  q.k += U;
  if (q.k < q.w) return;
  q.s += blockDim.x >> 5;
  open_slice(a, m, q);
}

// the chunk at q, as far as the row has slots
template <int B, int U, class T>
__device__ __forceinline__ void load_chunk(const PersistArgs<T>& a, const BlockRows<T>& m, const Cursor& q,
                                           Chunk<B, U, T>& c) {
  using V = typename Loop<T>::Val;
  using I = typename Loop<T>::Idx;
  constexpr int B2 = B * B;
  if (q.s >= m.n) return;
  const int lane = threadIdx.x & 31, n = q.len - q.k;
  if (q.s < m.ncache) {
    const V* v = reinterpret_cast<const V*>(m.cval + (long long)m.cb0[q.s] * cache_slot<B, T>());
    const I* g = reinterpret_cast<const I*>(v + q.w * B2 * 32) + q.k * 32 + lane;
    v += q.k * B2 * 32 + lane;
#pragma unroll
    for (int u = 0; u < U; u++)
      if (u < n) {
        c.j[u] = g[u * 32];
#pragma unroll
        for (int e = 0; e < B2; e++) c.a[u][e] = v[(u * B2 + e) * 32];
      }
    return;
  }
  const long long base = q.sc & ~3LL;
  const V* v;
  if constexpr (sizeof(T) == 8) v = a.A64.val + base * B2 + lane;
  else v = reinterpret_cast<const float2*>(a.A32.val + base * B2) + lane;
  v += q.k * B2 * 32;
#pragma unroll
  for (int u = 0; u < U; u++)
    if (u < n) {
#pragma unroll
      for (int e = 0; e < B2; e++) c.a[u][e] = ld_mat<kStreamKeep>(v + (u * B2 + e) * 32);
    }
  if (q.sc & 2) return;
  if constexpr (sizeof(T) == 8) {
    if (q.sc & 1) {
      const int* g = a.A64.col + base + q.k * 32 + lane;
#pragma unroll
      for (int u = 0; u < U; u++)
        if (u < n) c.j[u] = __ldg(g + u * 32);
    } else {
      const short* d = a.A64.col16 + base + q.k * 32 + lane;
#pragma unroll
      for (int u = 0; u < U; u++)
        if (u < n) c.j[u] = __ldg(d + u * 32);
    }
  } else {
    if (q.sc & 1) {
      const int2* g = reinterpret_cast<const int2*>(a.A32.col2 + base) + q.k * 32 + lane;
#pragma unroll
      for (int u = 0; u < U; u++)
        if (u < n) c.j[u] = __ldg(g + u * 32);
    } else {
      const int* d = reinterpret_cast<const int*>(a.A32.col16p + base) + q.k * 32 + lane;  // a pair of differences
#pragma unroll
      for (int u = 0; u < U; u++)
        if (u < n) c.j[u].x = __ldg(d + u * 32);
    }
  }
}

// column(s) of slot q.k + u from the loaded word
template <int B, class T>
__device__ __forceinline__ typename Loop<T>::Idx column(const BlockRows<T>& m, const Cursor& q, int u,
                                                        typename Loop<T>::Idx raw) {
  const int lane = threadIdx.x & 31;
  if (q.s < m.ncache || (q.sc & 1)) return raw;
  const int cb = q.cb[q.k + u];
  if constexpr (sizeof(T) == 8) {
    return cb + lane + (q.sc & 2 ? 0 : raw);
  } else {
    const int2 d = q.sc & 2 ? make_int2(0, 0) : make_int2((short)(raw.x & 0xffff), raw.x >> 16);
    return make_int2(cb + 2 * lane + d.x, cb + 2 * lane + 1 + d.y);
  }
}

// Keeps the values and decoded columns of as many of the block's first slices
// as fit in the rest of the shared memory (for the whole solve: the matrix is
// the same in every iteration).
template <int B, class T>
__device__ __forceinline__ void cache_slices(const PersistArgs<T>& a, BlockRows<T>& m) {
  using V = typename Loop<T>::Val;
  using I = typename Loop<T>::Idx;
  constexpr int B2 = B * B;
  const int room = a.smem - m.used;
  m.cval = g_smem + m.used;
  int n = 0;
  while (n < m.n && (long long)(m.cb0[n] + m.wid[n]) * cache_slot<B, T>() <= room) n++;
  const int lane = threadIdx.x & 31;
  Cursor q;
  q.s = threadIdx.x >> 5;
  for (open_slice(a, m, q); q.s < n; advance<1>(a, m, q)) {
    V* v = reinterpret_cast<V*>(const_cast<unsigned char*>(m.cval) + (long long)m.cb0[q.s] * cache_slot<B, T>());
    I* g = reinterpret_cast<I*>(v + q.w * B2 * 32);
    Chunk<B, 1, T> c;
    load_chunk<B, 1, T>(a, m, q, c);
    if (q.k < q.len) {
      g[q.k * 32 + lane] = column<B, T>(m, q, 0, c.j[0]);
#pragma unroll
      for (int e = 0; e < B2; e++) v[(q.k * B2 + e) * 32 + lane] = c.a[0][e];
    }
  }
  __syncthreads();
  m.ncache = n;
}

// A warp's product in D chunk buffers: D - 1 chunks are in flight while one is
// multiplied (the buffers are indexed statically: a copy from one to the next
// would wait for its loads).
template <int B, int U, int D, class T>
struct Pipe {
  Chunk<B, U, T> c[D];
  Cursor tail;
};
// the first D - 1 chunks (issued before the wait that precedes the product:
// the matrix does not depend on it)
template <int B, int U, int D, class T>
__device__ __forceinline__ void fill_pipe(const PersistArgs<T>& a, const BlockRows<T>& m, Pipe<B, U, D, T>& p) {
  p.tail.s = threadIdx.x >> 5;
  open_slice(a, m, p.tail);
#pragma unroll
  for (int d = 0; d < D - 1; d++) {
    load_chunk<B, U, T>(a, m, p.tail, p.c[d]);
    if (p.tail.s < m.n) advance<U>(a, m, p.tail);
  }
}

// body(row, y) for every row of this block, y = (A x)[row], x indexed by the
// vector's own index (the window, or the vector in global memory). p filled.
template <int B, int U, int D, class T, class F>
__device__ __forceinline__ void product(const PersistArgs<T>& a, const BlockRows<T>& m, Pipe<B, U, D, T>& p, const T* x,
                                        F&& body) {
  constexpr int P = sizeof(T) == 8 ? 1 : 2;
  const int lane = threadIdx.x & 31;
  Cursor q;
  q.s = threadIdx.x >> 5;
  open_slice(a, m, q);
  T y[P][B];
#pragma unroll
  for (int h = 0; h < P; h++)
#pragma unroll
    for (int r = 0; r < B; r++) y[h][r] = T(0);
  while (q.s < m.n) {
#pragma unroll
    for (int d = 0; d < D; d++) {
      load_chunk<B, U, T>(a, m, p.tail, p.c[(d + D - 1) % D]);
      if (p.tail.s < m.n) advance<U>(a, m, p.tail);
      if (q.s < m.n) {
        Chunk<B, U, T>& c = p.c[d];
        T x0[U][B], x1[U][B];
#pragma unroll
        for (int u = 0; u < U; u++)
          if (u < q.len - q.k) {
            const auto j = column<B, T>(m, q, u, c.j[u]);
#pragma unroll
            for (int l = 0; l < B; l++) {
              if constexpr (P == 1) {
                x0[u][l] = x[j * B + l];
              } else {
                x0[u][l] = x[j.x * B + l];
                x1[u][l] = x[j.y * B + l];
              }
            }
          }
#pragma unroll
        for (int u = 0; u < U; u++)
          if (u < q.len - q.k) {
#pragma unroll
            for (int r = 0; r < B; r++)
#pragma unroll
              for (int l = 0; l < B; l++) {
                if constexpr (P == 1) {
                  y[0][r] = add_rn(y[0][r], mul_rn(c.a[u][r * B + l], x0[u][l]));
                } else {
                  y[0][r] = fmaf(c.a[u][r * B + l].x, x0[u][l], y[0][r]);
                  y[1][r] = fmaf(c.a[u][r * B + l].y, x1[u][l], y[1][r]);
                }
              }
          }
        if (q.k + U >= q.w) {
          const int row = ((m.s0 + q.s) * 32 + lane) * P;
#pragma unroll
          for (int h = 0; h < P; h++) {
            if (row + h < a.N) body(row + h, y[h]);
#pragma unroll
            for (int r = 0; r < B; r++) y[h][r] = T(0);
          }
        }
        advance<U>(a, m, q);
      }
    }
  }
}

// f(R, first row) for the whole 16-byte groups of R rows of [r0, r1), then with
// one row for the rest.
template <int B, class T>
constexpr int group_rows() { return B <= 2 ? RowGroup<T, B>::R : 1; }  // larger blocks: registers
template <int B, class T, class F>
__device__ __forceinline__ void row_groups(int r0, int r1, F&& f) {
  constexpr int R = group_rows<B, T>();
  const int ng = (r1 - r0) / R;
  for (int g = threadIdx.x; g < ng; g += blockDim.x) f(std::integral_constant<int, R>{}, r0 + g * R);
  if constexpr (R > 1)
    for (int row = r0 + ng * R + (int)threadIdx.x; row < r1; row += blockDim.x) f(std::integral_constant<int, 1>{}, row);
}
template <class T, int E>
__device__ __forceinline__ void gload(bool vec, const T* p, T (&v)[E]) {
  if constexpr ((E * sizeof(T)) % 16 == 0) {
    if (vec) {
      vload<T, E>(p, v);
      return;
    }
  }
#pragma unroll
  for (int i = 0; i < E; i++) v[i] = p[i];
}
template <class T, int E>
__device__ __forceinline__ void gstore(bool vec, T* p, const T (&v)[E]) {
  if constexpr ((E * sizeof(T)) % 16 == 0) {
    if (vec) {
      vstore<T, E>(p, v);
      return;
    }
  }
#pragma unroll
  for (int i = 0; i < E; i++) p[i] = v[i];
}
// w = M^-1 w for R rows of B values with the factors L
template <int B, class T, int R>
__device__ __forceinline__ void apply_diag(const T (&L)[B * B][R], T (&w)[R * B]) {
#pragma unroll
  for (int k = 0; k < R; k++) {
    T t[B];
#pragma unroll
    for (int c = 0; c < B; c++) t[c] = w[k * B + c];
    diag_solve<B, T>([&](int j, int kk) { return L[j * B + kk][k]; }, t);
#pragma unroll
    for (int c = 0; c < B; c++) w[k * B + c] = t[c];
  }
}

// f(i, n) for the window's entries: n = the entries of a 16-byte word, then 1
template <int B, class T, class F>
__device__ __forceinline__ void window_entries(const BlockRows<T>& m, F&& f) {
  constexpr int W = Vec16T<T>::n;
  const long long i0 = (long long)m.w0 * B;
  const int n = (m.w1 - m.w0) * B, nv = n / W;
#pragma unroll 4
  for (int g = threadIdx.x; g < nv; g += blockDim.x) f(std::integral_constant<int, W>{}, i0 + g * W);
  for (int i = nv * W + (int)threadIdx.x; i < n; i += blockDim.x) f(std::integral_constant<int, 1>{}, i0 + i);
}

template <class T>
struct Plain {
  const T* p;
  __device__ __forceinline__ T operator()(long long i) const { return p[i]; }
};
struct SumXY {
  const double* x;
  const float* y;
  __device__ __forceinline__ double operator()(long long i) const { return x[i] + (double)y[i]; }
};

// r = b - A x (refined: b - A (x + y), stored FP32) on the block's rows, and
// CG: z = M^-1 r, sums <r,r>, <r,z>; BiCGSTAB: <r,r>, <r,rt> (init: rt = r).
// Sums in double-double in either precision, as in the kernels per phase: the
// residual that decides convergence does not depend on their grouping.
template <int B, class T, bool Bicg>
__device__ __forceinline__ void residual(const PersistArgs<T>& a, const BlockRows<T>& m, T* r, T* rt /* CG: z */,
                                         DDAcc<2>& v, bool init = false) {
  constexpr bool kMixed = sizeof(T) == 4;
  constexpr int UR = B == 1 ? 4 : (B <= 3 ? 2 : 1);
  for (int row = m.r0 + (int)threadIdx.x; row < m.r1; row += blockDim.x) {
    double ax[B];
    if constexpr (kMixed) sell_row_f<B, UR, double, double, true, kStreamKeep>(a.A64, SumXY{a.x, a.y}, row, ax);
    else sell_row_f<B, UR, double, double, true, kStreamKeep>(a.A64, Plain<double>{a.x}, row, ax);
    T t[B], w[B];
#pragma unroll
    for (int c = 0; c < B; c++) {
      const long long i = (long long)row * B + c;
      const double rv = sub_rn(a.b[i], ax[c]);
      t[c] = (T)rv;
      v.add(0, rv, rv);
      r[i] = t[c];
      w[c] = t[c];
    }
    if constexpr (!Bicg) {
      if (a.prec) diag_row<B, T>(a.alu, a.N, row, w);
#pragma unroll
      for (int c = 0; c < B; c++) rt[(long long)row * B + c] = w[c];
    } else {
#pragma unroll
      for (int c = 0; c < B; c++) {
        const long long i = (long long)row * B + c;
        if (init) rt[i] = t[c];
        else w[c] = rt[i];
      }
    }
#pragma unroll
    for (int c = 0; c < B; c++) v.add(1, t[c], w[c]);
  }
}

// The end of a block that has written its part of X: the last of the grid
// leaves the verdict (S has the same bits in every block). One that gave up a
// wait never comes here, and *a.st then stays without a verdict.
template <class T>
__device__ __forceinline__ void publish(const PersistArgs<T>& a, const SolverState& S) {
  __syncthreads();
  if (threadIdx.x == 0) {
    fence_gpu();
    if (atomicAdd(&a.slots->finished, 1u) == gridDim.x - 1) *a.st = S;
  }
}

// dst = src on the block's entries
template <int B, class T>
__device__ __forceinline__ void copy_own(const BlockRows<T>& m, T* dst, const T* src) {
  for (long long i = (long long)m.r0 * B + threadIdx.x; i < (long long)m.r1 * B; i += blockDim.x) dst[i] = src[i];
}

// ---------------------------------------------------------------------------
// CG
// ---------------------------------------------------------------------------
template <int B, int U, int D, int TH, bool kWin, class T>
__global__ void __launch_bounds__(TH, 1) persist_cg_kernel(const PersistArgs<T> a) {
  constexpr bool kMixed = sizeof(T) == 4;
  __shared__ SolverState S;
  __shared__ ExchangeShared sh;
  Exchange ex{a.slots, a.limit, a.delay_at, a.delay_ns};
  if (threadIdx.x == 0) S = *a.st;
  BlockRows<T> m = block_rows<B, kWin>(a);
  T* r = own_vector<B>(a, m, 0);
  T* q = own_vector<B>(a, m, 1);
  T* xo = own_vector<B>(a, m, 2);  // X, or the correction Y
  // P: the window, updated there by every block from the Z it reads; without
  // a window, in global memory, the owner's rows updated by the owner
  T* const pw = kWin ? m.win : a.zt;
  T* const z = kWin ? a.z : own_vector<B>(a, m, 3);
  __syncthreads();
  cache_slices<B>(a, m);
  double* hist = blockIdx.x == 0 ? a.hist : nullptr;
  T* xg;  // where other blocks read it
  if constexpr (kMixed) xg = a.y;
  else xg = a.x;
  for (long long i = (long long)m.r0 * B + threadIdx.x; i < (long long)m.r1 * B; i += blockDim.x) {
    if constexpr (kMixed) a.y[i] = xo[i] = T(0);
    else xo[i] = a.x[i];
  }
  for (int i = threadIdx.x; i < (m.w1 - m.w0) * B; i += blockDim.x) pw[(long long)m.w0 * B + i] = T(0);
  auto finish = [&](auto tot) {
    if constexpr (kMixed) fin_mixed_refresh<false>(&S, tot(0), tot(1), hist);
    else fin_cg(&S, tot(0), tot(1), hist);
  };
  // the first residual reads x (and y = 0, just written) of other blocks
  if (!grid_barrier(ex, sh)) return;
  Pipe<B, U, D, T> pipe;
  {
    DDAcc<2> v;
    residual<B, T, false>(a, m, r, z, v);
    fill_pipe(a, m, pipe);
    if (!grid_exchange(ex, sh, v, finish)) return;
  }
  const bool alu_vec = (a.N % group_rows<B, T>()) == 0;
  while (!S.done) {
    // P = beta P + Z over the window; Q = A P, <P,Q> (and the fold of Y into X
    // after a refresh)
    {
      const T beta = (T)S.beta;
      const bool fold = kMixed && S.fold;
      window_entries<B, T>(m, [&](auto Wc, long long i) {
        constexpr int W = decltype(Wc)::value;
        T zv[W], pv[W];
        gload(W > 1, z + i, zv);
        gload(W > 1, pw + i, pv);
#pragma unroll
        for (int k = 0; k < W; k++) pv[k] = axpy_rn(beta, pv[k], zv[k]);
        gstore(W > 1, pw + i, pv);
      });
      if constexpr (kMixed)
        if (fold)
          for (long long i = (long long)m.r0 * B + threadIdx.x; i < (long long)m.r1 * B; i += blockDim.x) {
            a.x[i] += (double)xo[i];
            xo[i] = T(0);
          }
      if constexpr (kWin) {
        __syncthreads();
      } else {
        if (!grid_barrier(ex, sh)) return;
      }
      DotAcc<1, T> v;
      product(a, m, pipe, pw, [&](int row, const T(&y)[B]) {
#pragma unroll
        for (int c = 0; c < B; c++) {
          const long long i = (long long)row * B + c;
          q[i] = y[c];
          v.add(0, pw[i], y[c]);
        }
      });
      if (!grid_exchange(ex, sh, v, [&](auto tot) {
            S.omega = tot(0);
            S.alpha = S.rho / tot(0);
            S.fold = 0;
          }))
        return;
    }
    // X (refined: Y) += alpha P; R -= alpha Q; Z = M^-1 R; <R,R>, <R,Z>
    const bool rr_iter = !kMixed && (S.iter % S.iter_rr) == 0;
    const T alpha = (T)S.alpha;
    DotAcc<2, T> v;
    row_groups<B, T>(m.r0, m.r1, [&](auto Rc, int row0) {
      constexpr int R = decltype(Rc)::value, E = R * B;
      constexpr bool kVec = R == group_rows<B, T>();
      const long long e0 = (long long)row0 * B;
      T pv[E], xv[E], rv[E], qv[E], zv[E], L[B * B][R];
      if (a.prec && !rr_iter) load_alu_rows<T, B, R>(a.alu, a.N, row0, kVec && alu_vec, L);
      gload(kVec, pw + e0, pv);
      gload(kVec, xo + e0, xv);
#pragma unroll
      for (int i = 0; i < E; i++) xv[i] = axpy_rn(alpha, pv[i], xv[i]);
      if (rr_iter) {
        gstore(kVec, xo + e0, xv);
        return;
      }
      gload(kVec, r + e0, rv);
      gload(kVec, q + e0, qv);
#pragma unroll
      for (int i = 0; i < E; i++) zv[i] = rv[i] = axpy_rn(-alpha, qv[i], rv[i]);
      if (a.prec) apply_diag<B, T, R>(L, zv);
      gstore(kVec, z + e0, zv);
      gstore(kVec, xo + e0, xv);
      gstore(kVec, r + e0, rv);
#pragma unroll
      for (int i = 0; i < E; i++) {
        v.add(0, rv[i], rv[i]);
        v.add(1, rv[i], zv[i]);
      }
    });
    fill_pipe(a, m, pipe);
    if (!rr_iter)
      if (!grid_exchange(ex, sh, v, [&](auto tot) {
            if constexpr (kMixed) fin_mixed_inner(&S, tot(0), tot(1), hist);
            else fin_cg(&S, tot(0), tot(1), hist);
          }))
        return;
    if (rr_iter || (kMixed && S.refresh)) {
      __syncthreads();
      copy_own<B, T>(m, xg, xo);
      if (!grid_barrier(ex, sh)) return;
      DDAcc<2> w;
      residual<B, T, false>(a, m, r, z, w);
      if (!grid_exchange(ex, sh, w, finish)) return;
    }
  }
  // the last exchange is behind: no block reads X any more
  if constexpr (kMixed) {
    if (S.fold)
      for (long long i = (long long)m.r0 * B + threadIdx.x; i < (long long)m.r1 * B; i += blockDim.x) a.x[i] += (double)xo[i];
  } else {
    copy_own<B, T>(m, xg, xo);
  }
  publish(a, S);
}

// ---------------------------------------------------------------------------
// BiCGSTAB (FP64)
// ---------------------------------------------------------------------------
template <int B, int U, int D, int TH>
__global__ void __launch_bounds__(TH, 1) persist_bicg_kernel(const PersistArgs<double> a) {
  using T = double;
  __shared__ SolverState S;
  __shared__ ExchangeShared sh;
  Exchange ex{a.slots, a.limit, a.delay_at, a.delay_ns};
  if (threadIdx.x == 0) S = *a.st;
  BlockRows<T> m = block_rows<B, false>(a);
  T* r = own_vector<B>(a, m, 0);
  T* vv = own_vector<B>(a, m, 1);
  T* sv = own_vector<B>(a, m, 2);
  T* p = own_vector<B>(a, m, 3);
  T* t = own_vector<B>(a, m, 4);
  T* rt = own_vector<B>(a, m, 5);
  T* xo = own_vector<B>(a, m, 6);  // X
  __syncthreads();
  cache_slices<B>(a, m);
  double* hist = blockIdx.x == 0 ? a.hist : nullptr;
  copy_own<B, T>(m, xo, a.x);
  auto finish = [&](auto tot) { fin_bicg(&S, tot(0), tot(1), hist); };
  Pipe<B, U, D, T> pipe;
  {
    DDAcc<2> v;
    residual<B, T, true>(a, m, r, rt, v, true);
    if (!grid_exchange(ex, sh, v, finish)) return;
  }
  const bool alu_vec = (a.N % group_rows<B, T>()) == 0;
  while (!S.done) {
    // P = R + beta (P - omega V) (P = R first), PT = M^-1 P
    {
      const bool first = S.iter == 1;
      const T beta = (T)S.beta, omega = (T)S.omega;
      row_groups<B, T>(m.r0, m.r1, [&](auto Rc, int row0) {
        constexpr int R = decltype(Rc)::value, E = R * B;
        constexpr bool kVec = R == group_rows<B, T>();
        const long long e0 = (long long)row0 * B;
        T pv[E], rv[E], w[E], L[B * B][R];
        if (a.prec) load_alu_rows<T, B, R>(a.alu, a.N, row0, kVec && alu_vec, L);
        gload(kVec, r + e0, rv);
        if (first) {
#pragma unroll
          for (int i = 0; i < E; i++) pv[i] = rv[i];
        } else {
          T vw[E];
          gload(kVec, p + e0, pv);
          gload(kVec, vv + e0, vw);
#pragma unroll
          for (int i = 0; i < E; i++) pv[i] = add_rn(rv[i], mul_rn(beta, sub_rn(pv[i], mul_rn(omega, vw[i]))));
        }
#pragma unroll
        for (int i = 0; i < E; i++) w[i] = pv[i];
        if (a.prec) apply_diag<B, T, R>(L, w);
        gstore(kVec, a.z + e0, w);
        gstore(kVec, p + e0, pv);
      });
      fill_pipe(a, m, pipe);
      if (!grid_barrier(ex, sh)) return;
    }
    // V = A PT, <RT,V>
    {
      DotAcc<1, T> v;
      product(a, m, pipe, (const T*)a.z, [&](int row, const T(&y)[B]) {
#pragma unroll
        for (int c = 0; c < B; c++) {
          const long long i = (long long)row * B + c;
          vv[i] = y[c];
          v.add(0, rt[i], y[c]);
        }
      });
      if (!grid_exchange(ex, sh, v, [&](auto tot) {
            S.c2 = tot(0);
            if (tot(0) == 0.0) {
              S.done = 1;
              S.status = kBreakdown;
            } else {
              S.alpha = S.rho / tot(0);
            }
          }))
        return;
      if (S.done) break;
    }
    const T alpha = (T)S.alpha;
    // S = R - alpha V, ST = M^-1 S
    row_groups<B, T>(m.r0, m.r1, [&](auto Rc, int row0) {
      constexpr int R = decltype(Rc)::value, E = R * B;
      constexpr bool kVec = R == group_rows<B, T>();
      const long long e0 = (long long)row0 * B;
      T rv[E], vw[E], w[E], L[B * B][R];
      if (a.prec) load_alu_rows<T, B, R>(a.alu, a.N, row0, kVec && alu_vec, L);
      gload(kVec, r + e0, rv);
      gload(kVec, vv + e0, vw);
#pragma unroll
      for (int i = 0; i < E; i++) w[i] = rv[i] = axpy_rn(-alpha, vw[i], rv[i]);
      if (a.prec) apply_diag<B, T, R>(L, w);
      gstore(kVec, a.zt + e0, w);
      gstore(kVec, sv + e0, rv);
    });
    fill_pipe(a, m, pipe);
    if (!grid_barrier(ex, sh)) return;
    // T = A ST, (T,S), (T,T)
    {
      DotAcc<2, T> v;
      product(a, m, pipe, (const T*)a.zt, [&](int row, const T(&y)[B]) {
#pragma unroll
        for (int c = 0; c < B; c++) {
          const long long i = (long long)row * B + c;
          t[i] = y[c];
          v.add(0, y[c], sv[i]);
          v.add(1, y[c], y[c]);
        }
      });
      if (!grid_exchange(ex, sh, v, [&](auto tot) {
            S.ts = tot(0);
            S.tt = tot(1);
            S.omega = tot(1) == 0.0 ? 0.0 : tot(0) / tot(1);
          }))
        return;
    }
    // X += alpha PT + omega ST; R = S - omega T; <R,R>, <R,RT>
    const bool rr_iter = (S.iter % S.iter_rr) == 0;
    const T omega = (T)S.omega;
    DotAcc<2, T> v;
    row_groups<B, T>(m.r0, m.r1, [&](auto Rc, int row0) {
      constexpr int R = decltype(Rc)::value, E = R * B;
      constexpr bool kVec = R == group_rows<B, T>();
      const long long e0 = (long long)row0 * B;
      T pv[E], wv[E], xv[E];
      gload(kVec, a.z + e0, pv);
      gload(kVec, a.zt + e0, wv);
      gload(kVec, xo + e0, xv);
#pragma unroll
      for (int i = 0; i < E; i++) xv[i] = add_rn(add_rn(xv[i], mul_rn(alpha, pv[i])), mul_rn(omega, wv[i]));
      gstore(kVec, xo + e0, xv);
      if (rr_iter) return;
      T tv[E], rv[E], rtv[E];
      gload(kVec, t + e0, tv);
      gload(kVec, sv + e0, rv);
      gload(kVec, rt + e0, rtv);
#pragma unroll
      for (int i = 0; i < E; i++) {
        rv[i] = axpy_rn(-omega, tv[i], rv[i]);
        v.add(0, rv[i], rv[i]);
        v.add(1, rv[i], rtv[i]);
      }
      gstore(kVec, r + e0, rv);
    });
    if (!rr_iter) {
      if (!grid_exchange(ex, sh, v, finish)) return;
    } else {
      __syncthreads();
      copy_own<B, T>(m, a.x, xo);
      if (!grid_barrier(ex, sh)) return;
      DDAcc<2> w;
      residual<B, T, true>(a, m, r, rt, w);
      if (!grid_exchange(ex, sh, w, finish)) return;
    }
  }
  // the last exchange is behind: no block reads X any more
  copy_own<B, T>(m, a.x, xo);
  publish(a, S);
}

// Threads of a block, slots of a chunk and chunk buffers, by block size.
// BiCGSTAB at 3x3 has no registers for three slots: 28^3 nodes 46 us an
// iteration (41 where the compiler happens to spill), two slots 40.
template <int B, class T, bool Bicg>
struct Shape {
  static constexpr int threads = B == 1 ? 512 : 256;
  static constexpr int u = B == 1 ? 4 : (B <= 3 ? (Bicg && B == 3 ? 2 : 3) : 1);
  static constexpr int d = B == 1 ? 3 : 2;
};
constexpr int kSmemBytes = 220 * 1024, kSmemCache = 180 * 1024;
// CG keeps P in windows up to this block size; BiCGSTAB and larger blocks
// gather from global memory. us an iteration, window / no window: CG ndof 3,
// 33^3 nodes FP64 19.4 / 24.7, 8^3 11.8 / 16.0; ndof 6, 36^3 45.9 / 41.1;
// BiCGSTAB ndof 1, 101x67x53 46.8 / 43.4 (two windows to load, no pass saved).
constexpr int kWindowMaxNdof = 3;

// Launch geometry and shared memory of a solve.
struct PersistPlan {
  int grid = 0, per = 0, win_rows = 0, cb_cap = 0, smem = 0;
  bool window = false, ok = false;
};
int sm_count() {
  static const int sms = [] {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n;
  }();
  return sms;
}
PersistPlan make_plan(const SellMatrix& m, const SolveParams& p) {
  PersistPlan q;
  const bool mixed = p.precision == 1;
  const int H = mixed ? 64 : 32, nsl = (m.N + H - 1) / H, tsize = mixed ? 4 : 8, B = m.ndof;
  q.grid = std::min(std::min(sm_count(), kMaxBlocks), nsl);
  q.per = (nsl + q.grid - 1) / q.grid;
  if (m.wmax > 65535 || q.per > 1024) return q;
  const long long slots = (mixed ? m.padded2 : m.padded) / H;  // slot positions of all slices
  q.cb_cap = (int)std::min<long long>(2 * (slots / q.grid) + 64, 8192);
  const long long own = (long long)q.per * H, band = (long long)m.below + m.above;
  const int own_bytes = up16((int)(own * B * tsize));
  const int nown = p.method == 1 ? 4 : 7;
  const int meta = meta_bytes(q.per, q.cb_cap);
  const long long win = (std::min<long long>(m.N, own + band + 4)) * B * tsize;
  q.window = p.method == 1 && B <= kWindowMaxNdof && meta + win + 64 <= kSmemBytes;
  q.win_rows = q.window ? (int)(win / (B * tsize)) : 0;
  const long long cache = (slots / q.grid + m.wmax + 8) * (32LL * (B * B * 8 + (mixed ? 8 : 4)));  // about a block's part of the matrix
  // slices of the matrix up to kSmemCache only: beyond it they cost the loads
  // in flight more L1 than they save (57x49x61 nodes refined, 180 KB 43.4 us
  // an iteration, 220 KB 46.1; 33^3 FP64 18.3 and 19.2)
  const long long need = meta + (q.window ? up16((int)win) : 0) + (long long)nown * own_bytes;
  q.smem = (int)std::min<long long>(kSmemBytes, std::max(need, std::min<long long>(need + cache, kSmemCache)));
  q.ok = meta <= kSmemBytes;
  return q;
}

}  // namespace

// exchange slots, then ten vectors (7 own, z, zt, y) in the loop precision
size_t persist_work_bytes(const SellMatrix& m, const SolveParams& p) {
  const size_t v = ((size_t)m.N * m.ndof * (p.precision == 1 ? 4 : 8) + 255) / 256 * 256;
  return (sizeof(ExchangeSlots) + 255) / 256 * 256 + 10 * v;
}

// The one-kernel solve is taken while the matrix stream of an iteration (bytes
// of the loop precision's layout) is small enough that the phases' launches
// and reductions cost more than streaming from one block an SM with few loads
// in flight does. us an iteration, kernel per phase / one kernel (B200, solves
// of 200 to 400 iterations; the stream in MB, 7- or 27-entry rows, grids in natural
// and in random numbering and plates too wide for the window):
//   CG, FP64      ndof 1  0.1 MB 30 / 8.8, 24 MB 28 / 16, no window: 47 MB 40 / 32, 50 MB 32 / 29
//                 ndof 2  49 MB 39 / 27, 66 MB 38 / 35, 76 MB 41 / 39, 87 MB 41 / 45
//                 ndof 3  0.8 MB 31 / 12, 134 MB 42 / 34, 218 MB 67 / 52, 245 MB 66 / 62; no window: 93 MB 46 / 33
//                 ndof 4  93 MB 39 / 34;   ndof 5  94 MB 40 / 30;   ndof 6  82 MB 40 / 35, 97 MB 42 / 40
//   CG, refined   ndof 1  7 MB 24 / 8.5, 50 MB 31 / 24; no window: 48 MB 46 / 37, 60 MB 35 / 34
//                 ndof 2  56 MB 35 / 30, 79 MB 40 / 37, 87 MB 42 / 41, 110 MB 48 / 49
//                 ndof 3  8 MB 28 / 11, 127 MB 42 / 36, 210 MB 60 / 51, 244 MB 66 / 67
//                 ndof 4  91 MB 39 / 36;   ndof 5  93 MB 40 / 29;   ndof 6  91 MB 42 / 37
//   BiCGSTAB      ndof 1  1.2 MB 47 / 20, 31 MB 49 / 40, 60 MB 69 / 82
//                 ndof 2  47 MB 55 / 50, 57 MB 56 / 57, 63 MB 61 / 64
//                 ndof 3  70 MB 63 / 46, 76 MB 64 / 62 (random numbering 73 / 82), 83 MB 67 / 70
//                 ndof 4  107 MB 72 / 69;   ndof 5  101 MB 71 / 63;   ndof 6  84 MB 67 / 63, 89 MB 69 / 71
// Refined BiCGSTAB stays with the kernels per phase: its dot products cancel,
// so its FP32 recurrences hang on the grouping of their plain sums (symmetric
// elasticity, 33^3 nodes: 1467 iterations with one, none within 20000 with
// another; ndof 1, 3 MB 42 / 20 us, 18 MB 41 / 35). The sums of refined CG are
// sums of squares in effect: 64-bit rounding of them is lost in the FP32
// scalars (same bits in every solve compared).
bool persist_applies(const SellMatrix& m, const SolveParams& p) {
  const bool mixed = p.precision == 1;
  // (a matrix with columns beyond its rows has no place in the windows)
  if (p.shard || p.np_rows != m.N || p.timers || (p.method != 1 && (p.method != 5 || mixed))) return false;
  const PersistPlan q = make_plan(m, p);
  // MB by ndof; ndof 3 without a window: 100
  static constexpr double kCg[6] = {50, 75, 250, 100, 100, 100}, kCgMixed[6] = {60, 88, 225, 100, 100, 100},
                          kBicg[6] = {32, 54, 74, 100, 100, 86};
  double limit = (p.method == 5 ? kBicg : mixed ? kCgMixed : kCg)[m.ndof - 1];
  if (p.method == 1 && !q.window) limit = std::min(limit, 100.0);
  return q.ok && (mixed ? m.bytes32 : m.bytes64) <= limit * 1e6;
}

int persist_solve(const SellMatrix& m, const SolveParams& p, const double* b, double* x, void* work, SolverState* st,
                  double* hist, cudaStream_t s) {
  const PersistPlan q = make_plan(m, p);
  if (!q.ok) return kBadInput;
  MB_CUDA_OK(cudaMemsetAsync(work, 0, sizeof(ExchangeSlots), s));
  auto run = [&](auto kernel, auto a, int threads) -> int {
    using T = std::remove_pointer_t<decltype(a.z)>;
    a.A64 = view_of<double>(m);
    a.A32 = view2_of(m);
    a.slptr = sizeof(T) == 8 ? m.d_slptr : m.d_slptr2;
    a.N = m.N;
    a.prec = p.precond == 1;
    a.below = m.below;
    a.above = m.above;
    a.b = b;
    a.x = x;
    a.alu = sizeof(T) == 8 ? (const T*)m.d_alu64 : (const T*)m.d_alu32;
    char* vec = (char*)work + (sizeof(ExchangeSlots) + 255) / 256 * 256;
    const size_t stride = ((size_t)m.N * m.ndof * sizeof(T) + 255) / 256 * 256;
    for (int k = 0; k < 7; k++) a.own[k] = (T*)(vec + k * stride);
    a.z = (T*)(vec + 7 * stride);
    a.zt = (T*)(vec + 8 * stride);
    a.y = (T*)(vec + 9 * stride);
    a.st = st;
    a.hist = hist;
    a.slots = (ExchangeSlots*)work;
    a.limit = p.wait_limit ? p.wait_limit : 1ull << 22;
    a.delay_at = p.delay_ns ? (p.delay_at + 1) * (unsigned long long)q.grid : 0;
    a.delay_ns = p.delay_ns;
    a.per = q.per;
    a.win_rows = q.win_rows;
    a.cb_cap = q.cb_cap;
    a.win_at = meta_bytes(q.per, q.cb_cap);
    a.smem = q.smem;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes) != cudaSuccess)
      return kRefused;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.gridDim = dim3(q.grid);
    // as many warps as a block has slices (a reduction over idle warps costs time)
    cfg.blockDim = dim3(std::min(threads, 32 * std::max(4, q.per)));
    cfg.dynamicSmemBytes = q.smem;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    // a fault of an earlier kernel comes back here too, and again from the next call
    const cudaError_t e = p.refuse == 1 ? cudaErrorCooperativeLaunchTooLarge : cudaLaunchKernelEx(&cfg, kernel, a);
    return e == cudaSuccess ? kOk : kRefused;
  };
  return dispatch_ndof(m.ndof, [&](auto Bc) -> int {
    constexpr int B = decltype(Bc)::value;
    auto pick = [&](auto Wc, auto a) -> int {
      using T = std::remove_pointer_t<decltype(a.z)>;
      using Sh = Shape<B, T, false>;
      using Sb = Shape<B, T, true>;
      constexpr bool W = decltype(Wc)::value && B <= kWindowMaxNdof;
      if (p.method == 1) return run(persist_cg_kernel<B, Sh::u, Sh::d, Sh::threads, W, T>, a, Sh::threads);
      if constexpr (sizeof(T) == 8) return run(persist_bicg_kernel<B, Sb::u, Sb::d, Sb::threads>, a, Sb::threads);
      else return kBadInput;
    };
    if (p.precision == 0)
      return q.window ? pick(std::true_type{}, PersistArgs<double>{}) : pick(std::false_type{}, PersistArgs<double>{});
    return q.window ? pick(std::true_type{}, PersistArgs<float>{}) : pick(std::false_type{}, PersistArgs<float>{});
  });
}

}  // namespace mb
