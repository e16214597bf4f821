// assemble.cu -- assembly of the block-CSR values on the device: element
// matrices (monolis_add_matrix_to_sparse_matrix_R for many elements) and
// Dirichlet conditions (monolis_set_Dirichlet_bc_R for a list of them),
// bit-identical to the host calls made in order.
//
// Elements: one warp per block row walks the elements incident to its row in
// ascending element order (a node -> element incidence list built on the
// device), each lane holding one block of the row, and within an element the
// (a, b) pairs in the order of src/matrix/spmat_handler_util.f90:398-497,
// adding scale * K_e(a,b) to the lane's block where b is its column. Every
// entry therefore receives its contributions in element order, as with the
// serial loop, and no two warps write the same block.
//
// Dirichlet (src/matrix/spmat_handler_util.f90:604-677) applied to a list of
// (node, dof, value) in order has a closed form that this file evaluates in
// parallel:
//   * a dof never fixed: b[n] -= v_c * A[n][c] for every fixed column c of its
//     row, in the order of each column's first occurrence in the list, with
//     the value of that first occurrence (a repeated column finds its entries
//     already zero);
//   * every entry in a fixed row or a fixed column becomes 0, the diagonal
//     entry of a fixed dof 1;
//   * b of a fixed dof is the value of its last occurrence.
// (Contributions to a dof's b made before its own condition is processed are
// overwritten by it; after its row is zeroed the column moves add v * 0.)
#include <algorithm>
#include <cstdio>
#include <vector>

#include "spmv.cuh"

namespace mb {
namespace {

// incidence counts: element e counted once per distinct node; bad bit 1 for
// a node out of range
__global__ void incidence_count_kernel(const int* __restrict__ elem, int n_elem, int n_base, int NP,
                                       int* __restrict__ cnt, int* __restrict__ bad) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n_elem;
       e += (long long)gridDim.x * blockDim.x) {
    const int* en = elem + e * n_base;
    for (int a = 0; a < n_base; a++) {
      const int v = en[a];
      if (v < 0 || v >= NP) {
        atomicOr(bad, 1);
        continue;
      }
      bool dup = false;
      for (int q = 0; q < a; q++) dup |= en[q] == v;
      if (!dup) atomicAdd(cnt + v, 1);
    }
  }
}

// Exclusive prefix sum of cnt[0, n) into ptr[0, n], kScanItems items a block:
// block sums, then every block adds up the sums before its own.
constexpr int kScanThreads = 512, kScanPer = 8, kScanItems = kScanThreads * kScanPer;
__device__ __forceinline__ int block_sum_int(int v, int* sm) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v = __reduce_add_sync(0xffffffffu, v);
  if (lane == 0) sm[warp] = v;
  __syncthreads();
  int t = lane < (int)(blockDim.x >> 5) ? sm[lane] : 0;
  t = __reduce_add_sync(0xffffffffu, t);
  __syncthreads();
  return t;
}
__global__ void __launch_bounds__(kScanThreads) scan_sums_kernel(const int* __restrict__ cnt, int n,
                                                                 int* __restrict__ sums) {
  __shared__ int sm[32];
  int v = 0;
  for (int k = 0; k < kScanPer; k++) {
    const long long i = (long long)blockIdx.x * kScanItems + k * kScanThreads + threadIdx.x;
    if (i < n) v += cnt[i];
  }
  v = block_sum_int(v, sm);
  if (threadIdx.x == 0) sums[blockIdx.x] = v;
}
__global__ void __launch_bounds__(kScanThreads) scan_write_kernel(const int* __restrict__ cnt, int n,
                                                                  const int* __restrict__ sums, int* __restrict__ ptr) {
  __shared__ int sm[32], wsum[32];
  int base = 0;
  for (int i = threadIdx.x; i < (int)blockIdx.x; i += blockDim.x) base += sums[i];
  base = block_sum_int(base, sm);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long i0 = (long long)blockIdx.x * kScanItems + (long long)threadIdx.x * kScanPer;
  int v[kScanPer], t = 0;
#pragma unroll
  for (int k = 0; k < kScanPer; k++) {
    v[k] = i0 + k < n ? cnt[i0 + k] : 0;
    t += v[k];
  }
  int inc = t;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += u;
  }
  if (lane == 31) wsum[warp] = inc;
  __syncthreads();
  int before = base + inc - t;
  for (int w = 0; w < warp; w++) before += wsum[w];
#pragma unroll
  for (int k = 0; k < kScanPer; k++) {
    if (i0 + k < n) ptr[i0 + k] = before;
    before += v[k];
    if (i0 + k == n - 1) ptr[n] = before;
  }
}

// the counts become the fill positions: cnt[i] counts down to 0
__global__ void incidence_fill_kernel(const int* __restrict__ elem, int n_elem, int n_base, int NP,
                                      const int* __restrict__ ptr, int* __restrict__ cnt, int* __restrict__ list) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n_elem;
       e += (long long)gridDim.x * blockDim.x) {
    const int* en = elem + e * n_base;
    for (int a = 0; a < n_base; a++) {
      const int v = en[a];
      if (v < 0 || v >= NP) continue;
      bool dup = false;
      for (int q = 0; q < a; q++) dup |= en[q] == v;
      if (!dup) list[ptr[v] + atomicSub(cnt + v, 1) - 1] = (int)e;
    }
  }
}

__device__ __forceinline__ int find_slot(const int* __restrict__ rowptr, const int* __restrict__ item, int i, int j) {
  int lo = rowptr[i], hi = rowptr[i + 1] - 1;
  const int key = j + 1;
  while (lo <= hi) {
    const int mid = (lo + hi) >> 1;
    const int v = item[mid];
    if (v == key) return mid;
    if (v < key) lo = mid + 1;
    else hi = mid - 1;
  }
  return -1;
}

// One warp per block row; lane l holds block l of each group of 32 blocks of
// the row and adds the contributions of the row's elements to it in element
// order. The lists come unsorted (the fill's atomics): a list of up to 32
// elements is ordered by rank within the warp, a longer one sorted in place
// by one lane. What bounds it is the element matrices and the values, each
// read or written once: 70,110 nodes of 3 dofs, a matrix per element (300 MB
// in, 130 MB in and out), took 1850 us with a thread per row that searched
// the row's columns for every (a, b), 650 us with a warp per row taking one
// element at a time (each waits for its loads), about 300 us with the loads of
// kGroup elements in flight (whole call 3240 -> 782 -> 425 us).
template <int B>
__global__ void __launch_bounds__(256) add_elements_kernel(const int* __restrict__ rowptr, const int* __restrict__ item,
                                                           int N, const int* __restrict__ iptr, int* __restrict__ ilist,
                                                           const int* __restrict__ elem, int n_base,
                                                           const double* __restrict__ val, long long val_stride,
                                                           const double* __restrict__ scale, double* __restrict__ A,
                                                           int* __restrict__ bad) {
  constexpr int B2 = B * B, kGroup = B <= 2 ? 4 : (B <= 4 ? 2 : 1);
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int i = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (i >= N || (*bad & 1)) return;  // whole warps; bad input leaves the values as they were
  const int q0 = iptr[i], nq = iptr[i + 1] - q0;
  if (nq == 0) return;
  const int k0 = rowptr[i], k1 = rowptr[i + 1];
  int mine = 0;  // lane q: element q of the row (nq <= 32)
  if (nq <= 32) {
    const int v = lane < nq ? ilist[q0 + lane] : 0x7fffffff;
    int rank = 0;
    for (int t = 0; t < nq; t++) rank += __shfl_sync(kAll, v, t) < v ? 1 : 0;
    for (int t = 0; t < nq; t++) {  // the lane whose element has rank t
      const unsigned m = __ballot_sync(kAll, lane < nq && rank == t);
      const int e = __shfl_sync(kAll, v, __ffs(m) - 1);
      if (lane == t) mine = e;
    }
  } else {
    if (lane == 0)
      for (int p = q0 + 1; p < q0 + nq; p++) {
        const int v = ilist[p];
        int q = p - 1;
        while (q >= q0 && ilist[q] > v) {
          ilist[q + 1] = ilist[q];
          q--;
        }
        ilist[q + 1] = v;
      }
    __syncwarp();
  }
  const int ncol = n_base * B;
  int want = 0, got = 0;  // (a, b) pairs of the row, pairs that found their block
  for (int kb = k0; kb < k1 || kb == k0; kb += 32) {
    const int k = kb + lane;
    const bool has = k < k1;
    int col = has ? item[k] - 1 : -1;
    // a column stored twice: only the block the serial search finds
    const bool dup = has && ((k > k0 && item[k - 1] == col + 1) || (k + 1 < k1 && item[k + 1] == col + 1));
    if (dup && find_slot(rowptr, item, i, col) != k) col = -1;
    double acc[B2];
    double* dst = A + (long long)k * B2;
    if (has) {
#pragma unroll
      for (int e = 0; e < B2; e++) acc[e] = dst[e];
    }
    // kGroup elements at a time: their connectivities, then the values each
    // lane takes from them, are in flight together; added in element order
    for (int q = 0; q < nq; q += kGroup) {
      long long e[kGroup];
      int va[kGroup];
      unsigned hit[kGroup], rows[kGroup];  // b with this lane's column, a with this row
      bool plain = n_base <= 32;
#pragma unroll
      for (int g = 0; g < kGroup; g++) {
        const int qg = min(q + g, nq - 1);
        e[g] = nq <= 32 ? __shfl_sync(kAll, mine, qg) : ilist[q0 + qg];
        va[g] = q + g < nq && lane < n_base ? elem[e[g] * n_base + lane] : -1;
      }
#pragma unroll
      for (int g = 0; g < kGroup; g++) {
        rows[g] = __ballot_sync(kAll, va[g] == i);
        hit[g] = 0;
        for (int t = 0; t < min(n_base, 32); t++)
          if (__shfl_sync(kAll, va[g], t) == col) hit[g] |= 1u << t;
        if (q + g >= nq || col < 0) hit[g] = 0;
        // a node once in the element (and one 32-lane load of its nodes)
        plain = plain && __popc(rows[g]) <= 1 && !__any_sync(kAll, __popc(hit[g]) > 1);
      }
      if (plain) {
        double v[kGroup][B2], sc[kGroup];
#pragma unroll
        for (int g = 0; g < kGroup; g++) {
          if (rows[g] && kb == k0) want += n_base;
          if (!rows[g]) hit[g] = 0;
          if (!hit[g]) continue;
          got++;
          const double* Ka =
              val + e[g] * val_stride + (long long)(__ffs(rows[g]) - 1) * B * ncol + (__ffs(hit[g]) - 1) * B;
          sc[g] = scale ? scale[e[g]] : 1.0;
#pragma unroll
          for (int r = 0; r < B; r++)
#pragma unroll
            for (int c = 0; c < B; c++) v[g][r * B + c] = Ka[(long long)r * ncol + c];
        }
#pragma unroll
        for (int g = 0; g < kGroup; g++)
          if (hit[g]) {
#pragma unroll
            for (int x = 0; x < B2; x++) acc[x] = __dadd_rn(acc[x], scale ? __dmul_rn(sc[g], v[g][x]) : v[g][x]);
          }
        continue;
      }
      for (int g = 0; g < kGroup && q + g < nq; g++) {
        const long long eg = nq <= 32 ? __shfl_sync(kAll, mine, q + g) : ilist[q0 + q + g];
        const int* en = elem + eg * n_base;
        const double s = scale ? scale[eg] : 1.0;
        for (int a = 0; a < n_base; a++) {
          if (en[a] != i) continue;
          if (kb == k0) want += n_base;
          const double* Ka = val + eg * val_stride + (long long)a * B * ncol;
          for (int t = 0; t < n_base; t++) {
            if (en[t] != col) continue;
            got++;
#pragma unroll
            for (int r = 0; r < B; r++)
#pragma unroll
              for (int c = 0; c < B; c++) {
                const double v = Ka[(long long)r * ncol + t * B + c];
                acc[r * B + c] = __dadd_rn(acc[r * B + c], scale ? __dmul_rn(s, v) : v);
              }
          }
        }
      }
    }
    if (has) {
#pragma unroll
      for (int e = 0; e < B2; e++) dst[e] = acc[e];
    }
  }
  got = __reduce_add_sync(kAll, got);
  if (lane == 0 && got != want) atomicOr(bad, 2);
}

// first and last condition of every dof (ord, last: their positions in the
// list); bad: a fixed dof's row has no diagonal block
__global__ void dirichlet_list_kernel(const long long* __restrict__ dof, int n_bc, const int* __restrict__ rowptr,
                                      const int* __restrict__ item, int ndof, int* __restrict__ ord,
                                      int* __restrict__ last, int* __restrict__ bad) {
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n_bc; q += gridDim.x * blockDim.x) {
    atomicMin(reinterpret_cast<unsigned int*>(ord) + dof[q], (unsigned int)q);
    atomicMax(last + dof[q], q);
    const int i = (int)(dof[q] / ndof);
    bool diag = find_slot(rowptr, item, i, i) >= 0;
    for (int k = rowptr[i]; !diag && k < rowptr[i + 1]; k++) diag = item[k] - 1 == i;  // a row not in order
    if (!diag) atomicOr(bad, 1);
  }
}

// The closed form above for one block row a warp: b[n] -= v_first(c) * A[n][c]
// over the fixed columns c of the row in the order of their first occurrence
// (never-fixed dofs n), then zero fixed rows and columns, unit diagonal of
// fixed dofs, b = last value, in the CSR values and in the sliced layout. A
// row that touches no fixed dof reads its columns and their marks only. Bad
// conditions leave everything as it was.
template <int B>
__global__ void __launch_bounds__(256) dirichlet_kernel(const int* __restrict__ rowptr, const int* __restrict__ item,
                                                        int N, double* __restrict__ A, const long long* __restrict__ slptr,
                                                        double* __restrict__ sell, const int* __restrict__ ord,
                                                        const int* __restrict__ last, const double* __restrict__ val,
                                                        double* __restrict__ b, const int* __restrict__ bad) {
  constexpr int B2 = B * B;
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int i = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (i >= N || *bad) return;  // whole warps
  const int lo = rowptr[i], hi = rowptr[i + 1];
  bool fr[B], own = false;
#pragma unroll
  for (int r = 0; r < B; r++) {
    fr[r] = ord[(long long)i * B + r] >= 0;
    own |= fr[r];
  }
  bool any = false;
  for (int k = lo + lane; k < hi; k += 32) {
    const long long j = item[k] - 1;
#pragma unroll
    for (int c = 0; c < B; c++) any |= ord[j * B + c] >= 0;
  }
  any = __any_sync(kAll, any);
  if (!any && !own) return;
  for (int prev = -1; any;) {
    // the fixed column of this row with the smallest first occurrence after prev
    unsigned best = 0x7fffffffu;
    int bk = 0x7fffffff, bc = 0;
    for (int k = lo + lane; k < hi; k += 32) {
      const long long j = item[k] - 1;
#pragma unroll
      for (int c = 0; c < B; c++) {
        const int o = ord[j * B + c];
        if (o > prev && (unsigned)o < best) {
          best = o;
          bk = k;
          bc = c;
        }
      }
    }
    const unsigned first = __reduce_min_sync(kAll, best);
    if (first == 0x7fffffffu) break;
    // its block (the first one, should the column be stored twice)
    const int k = __reduce_min_sync(kAll, best == first ? bk : 0x7fffffff);
    const unsigned who = __ballot_sync(kAll, best == first && bk == k);
    const int c = __shfl_sync(kAll, bc, __ffs(who) - 1);
    if (lane == 0) {
      const double v = val[first];
#pragma unroll
      for (int r = 0; r < B; r++)
        if (!fr[r]) {
          const long long n = (long long)i * B + r;
          b[n] = __dsub_rn(b[n], __dmul_rn(v, A[(long long)k * B2 + r * B + c]));
        }
    }
    prev = (int)first;
  }
  __syncwarp();
  const long long base = slptr[i >> 5];
  for (int k = lo + lane; k < hi; k += 32) {
    const long long j = item[k] - 1;
    double* dst = A + (long long)k * B2;
    double* sl = sell + (base + (long long)(k - lo) * kSlice) * B2 + (i & (kSlice - 1));
#pragma unroll
    for (int c = 0; c < B; c++) {
      const bool fc = ord[j * B + c] >= 0;
#pragma unroll
      for (int r = 0; r < B; r++)
        if (fr[r] || fc) {
          const double u = fr[r] && j == i && c == r ? 1.0 : 0.0;
          dst[r * B + c] = u;
          sl[(r * B + c) * kSlice] = u;
        }
    }
  }
  if (lane == 0) {
#pragma unroll
    for (int r = 0; r < B; r++)
      if (fr[r]) b[(long long)i * B + r] = val[last[(long long)i * B + r]];
  }
}

// device scratch of one call, given back to the library's pool at its end
struct Temps {
  cudaStream_t s;
  std::vector<void*> p;
  ~Temps() {
    for (void* q : p) cudaFreeAsync(q, s);
  }
  template <class P>
  cudaError_t get(P** out, size_t n) {
    void* q = nullptr;
    const cudaError_t e = pool_alloc(&q, n * sizeof(P) + 16, s);
    if (e == cudaSuccess) p.push_back(q);
    *out = static_cast<P*>(q);
    return e;
  }
};

unsigned warps_grid(int N) { return (unsigned)(((long long)N * 32 + 255) / 256); }

}  // namespace

int device_clear_values(SellMatrix& m, cudaStream_t s) {
  const size_t B2 = (size_t)m.ndof * m.ndof;
  MB_CUDA_OK(cudaMemsetAsync(m.d_csrval, 0, (size_t)m.nz * B2 * sizeof(double), s));
  MB_CUDA_OK(cudaMemsetAsync(m.d_val64, 0, (size_t)m.padded * B2 * sizeof(double), s));
  sell_values_changed(m);
  return kOk;
}

int device_add_elements(SellMatrix& m, int NP, int n_elem, int n_base, const int* d_elem, const double* d_val,
                        long long val_stride, const double* d_scale, cudaStream_t s) {
  if (n_elem < 0 || n_base <= 0 || val_stride < 0 || !m.d_csrval) return kBadInput;
  if (n_elem == 0) return kOk;
  const int N = m.N;
  if (NP != N) return kBadInput;
  const long long ne = (long long)n_elem * n_base;
  const int nscan = (N + kScanItems - 1) / kScanItems;
  Temps tmp{s, {}};
  int *d_bad = nullptr, *d_cnt = nullptr, *d_ptr = nullptr, *d_list = nullptr;
  MB_CUDA_OK(tmp.get(&d_cnt, (size_t)N + 1 + nscan));  // counts, flag, block sums of the scan
  MB_CUDA_OK(tmp.get(&d_ptr, (size_t)N + 1));
  MB_CUDA_OK(tmp.get(&d_list, (size_t)ne));
  d_bad = d_cnt + N;
  int* d_sums = d_bad + 1;
  MB_CUDA_OK(cudaMemsetAsync(d_cnt, 0, sizeof(int) * ((size_t)N + 1), s));
  const int grid = (int)std::min<long long>(((long long)n_elem + 255) / 256, 148LL * 8);
  incidence_count_kernel<<<grid, 256, 0, s>>>(d_elem, n_elem, n_base, NP, d_cnt, d_bad);
  scan_sums_kernel<<<nscan, kScanThreads, 0, s>>>(d_cnt, N, d_sums);
  scan_write_kernel<<<nscan, kScanThreads, 0, s>>>(d_cnt, N, d_sums, d_ptr);
  incidence_fill_kernel<<<grid, 256, 0, s>>>(d_elem, n_elem, n_base, NP, d_ptr, d_cnt, d_list);
  int rc = dispatch_ndof(m.ndof, [&](auto Bc) {
    constexpr int B = decltype(Bc)::value;
    add_elements_kernel<B><<<warps_grid(N), 256, 0, s>>>(m.d_rowptr, m.d_item, N, d_ptr, d_list, d_elem, n_base, d_val,
                                                         val_stride, d_scale, m.d_csrval, d_bad);
    return kOk;
  });
  if (rc) return rc;
  MB_CUDA_OK(cudaGetLastError());
  const bool had[3] = {m.have_val32, m.have_alu, m.have_alu32};
  rc = sell_refill(m, s, d_bad);
  if (rc) return rc;
  int bad = 0;
  MB_CUDA_OK(cudaMemcpyAsync(&bad, d_bad, sizeof(int), cudaMemcpyDeviceToHost, s));
  MB_CUDA_OK(cudaStreamSynchronize(s));
  if (!bad) return kOk;
  // refused: the layout has not been refilled, and what is derived from it stands
  m.have_val32 = had[0];
  m.have_alu = had[1];
  m.have_alu32 = had[2];
  if (bad & 2) {
    // the entries that are in the pattern have been added: back to the layout's values
    fprintf(stderr, "** monolis_b200: device assembly: an element entry is not in the nonzero pattern\n");
    rc = sell_restore_csr(m, s);
    if (rc) return rc;
    MB_CUDA_OK(cudaStreamSynchronize(s));
  }
  return kBadInput;
}

int device_dirichlet(SellMatrix& m, int NP, double* d_b, int n_bc, const int* node, const int* dof, const double* val,
                     cudaStream_t s) {
  const int N = m.N, nd = m.ndof;
  const long long n = (long long)std::max(N, NP) * nd;  // columns: ghosts, never fixed here, after the own rows
  std::vector<long long> flat((size_t)n_bc);
  for (int q = 0; q < n_bc; q++) {
    if (node[q] < 0 || node[q] >= N || dof[q] < 0 || dof[q] >= nd) return kBadInput;
    flat[q] = (long long)node[q] * nd + dof[q];
  }
  if (n_bc == 0) return kOk;
  Temps tmp{s, {}};
  int *d_ord = nullptr, *d_last = nullptr, *d_bad = nullptr;
  long long* d_dof = nullptr;
  double* d_val = nullptr;
  MB_CUDA_OK(tmp.get(&d_ord, (size_t)n));
  MB_CUDA_OK(tmp.get(&d_last, (size_t)n));
  MB_CUDA_OK(tmp.get(&d_dof, (size_t)n_bc));
  MB_CUDA_OK(tmp.get(&d_val, (size_t)n_bc));
  MB_CUDA_OK(tmp.get(&d_bad, 1));
  MB_CUDA_OK(cudaMemsetAsync(d_ord, 0xff, sizeof(int) * n, s));  // -1: never fixed
  MB_CUDA_OK(cudaMemsetAsync(d_last, 0xff, sizeof(int) * n, s));
  MB_CUDA_OK(cudaMemsetAsync(d_bad, 0, sizeof(int), s));
  MB_CUDA_OK(cudaMemcpyAsync(d_dof, flat.data(), sizeof(long long) * n_bc, cudaMemcpyHostToDevice, s));
  MB_CUDA_OK(cudaMemcpyAsync(d_val, val, sizeof(double) * n_bc, cudaMemcpyHostToDevice, s));
  dirichlet_list_kernel<<<std::min((n_bc + 255) / 256, 148 * 8), 256, 0, s>>>(d_dof, n_bc, m.d_rowptr, m.d_item, nd,
                                                                           d_ord, d_last, d_bad);
  int rc = dispatch_ndof(nd, [&](auto Bc) {
    constexpr int B = decltype(Bc)::value;
    dirichlet_kernel<B><<<warps_grid(N), 256, 0, s>>>(m.d_rowptr, m.d_item, N, m.d_csrval, m.d_slptr, m.d_val64, d_ord,
                                                      d_last, d_val, d_b, d_bad);
    return kOk;
  });
  if (rc) return rc;
  MB_CUDA_OK(cudaGetLastError());
  int bad = 0;
  MB_CUDA_OK(cudaMemcpyAsync(&bad, d_bad, sizeof(int), cudaMemcpyDeviceToHost, s));
  MB_CUDA_OK(cudaStreamSynchronize(s));
  if (bad) {
    fprintf(stderr, "** monolis_b200: set Dirichlet: diagonal block not found\n");
    return kBadInput;
  }
  sell_values_changed(m);
  return kOk;
}

}  // namespace mb
