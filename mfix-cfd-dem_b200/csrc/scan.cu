// scan.cu -- exclusive prefix sum over int32 (cell counts, row counts).
//
// Two launches: each block of 512 threads adds up a tile of 2048 items (4 per
// thread), then each block scans its tile (warp shuffles and one
// shared-memory pass) behind the sum of the tiles before it, which it adds up
// itself from the first launch's sums: a few hundred for a million items, read
// from L2.  Past SCAN_DIRECT tiles the sums are scanned first.  Deterministic
// (integer arithmetic).  The scans of a rebuild are short, so what they cost
// is launches: the pair of them replaced four (tile scan, scan of the sums,
// their addition, total).
#include "dem_internal.cuh"

namespace demb {

constexpr int SCAN_THREADS = 512;
constexpr int SCAN_ITEMS = 4;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;
constexpr int SCAN_DIRECT = 4096;  // tiles whose sums each block adds up itself

// Sum of v over the block, in every thread.
__device__ __forceinline__ int block_sum(int v, int* warp_tot) {
  v = __reduce_add_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0) warp_tot[threadIdx.x >> 5] = v;
  __syncthreads();
  int t = 0;
#pragma unroll
  for (int w = 0; w < SCAN_THREADS / 32; ++w) t += warp_tot[w];
  __syncthreads();
  return t;
}

// `go` (when given): nothing is done unless it is set.
__global__ void __launch_bounds__(SCAN_THREADS)
k_scan_sums(const int* __restrict__ in, int n, int* __restrict__ sums, const int* __restrict__ go) {
  __shared__ int warp_tot[SCAN_THREADS / 32];
  const int z = pdl_wait();
  pdl_next();
  if (go && !go[z]) return;
  const int base = blockIdx.x * SCAN_TILE + z;
  int s = 0;
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    const int idx = base + k * SCAN_THREADS + threadIdx.x;
    if (idx < n) s += in[idx];
  }
  s = block_sum(s, warp_tot);
  if (threadIdx.x == 0) sums[blockIdx.x] = s;
}

// The tile's exclusive scan; `scanned`: sums holds the tiles' offsets, not
// their sums.  The last block writes the total.  CLEAR zeroes the input.
template <bool CLEAR>
__global__ void __launch_bounds__(SCAN_THREADS)
k_scan_tile(int* in, int* out, int n, const int* __restrict__ sums, int scanned, int* __restrict__ total,
            const int* __restrict__ go) {
  __shared__ int warp_tot[SCAN_THREADS / 32];
  const int z = pdl_wait();
  pdl_next();
  if (go && !go[z]) return;
  int off = 0;
  if (scanned) {
    off = sums[blockIdx.x + z];
  } else if (blockIdx.x) {
    int s = 0;
    for (int b = threadIdx.x; b < (int)blockIdx.x; b += SCAN_THREADS) s += sums[b + z];
    off = block_sum(s, warp_tot);
  }
  const int base = blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_ITEMS + z;
  int v[SCAN_ITEMS];
  int s = 0;
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    const int idx = base + k;
    v[k] = idx < n ? in[idx] : 0;
    s += v[k];
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int incl = s;  // inclusive warp scan of per-thread sums
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_tot[wid] = incl;
  __syncthreads();
  int before = 0;
#pragma unroll
  for (int w = 0; w < SCAN_THREADS / 32; ++w) before += w < wid ? warp_tot[w] : 0;
  int run = off + before + incl - s;
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    const int idx = base + k;
    if (idx < n) {
      if (CLEAR) in[idx] = 0;
      out[idx] = run;
    }
    run += v[k];
  }
  if (total && blockIdx.x == gridDim.x - 1 && threadIdx.x == SCAN_THREADS - 1) *total = run;
}

static size_t scratch_need(int n) {
  size_t need = 0;
  long long m = n;
  while (m > SCAN_TILE) {
    m = (m + SCAN_TILE - 1) / SCAN_TILE;
    need += (size_t)m + 1;
  }
  return need + 1;
}

static void scan_rec(dem_handle* h, int* in, int* out, int n, int* tmp, int* total, bool clear, const int* go) {
  const int nb = (n + SCAN_TILE - 1) / SCAN_TILE;
  if (nb > 1) launch_pdl(h, k_scan_sums, nb, SCAN_THREADS, in, n, tmp, go);
  const bool deep = nb > SCAN_DIRECT;
  if (deep) scan_rec(h, tmp, tmp, nb, tmp + nb + 1, nullptr, false, go);
  launch_pdl(h, clear ? k_scan_tile<true> : k_scan_tile<false>, nb, SCAN_THREADS, in, out, n, tmp, deep ? 1 : 0, total,
             go);
}

int reserve_scan(dem_handle* h, int n) {
  const size_t need = n > 0 ? scratch_need(n) : 0;
  if (need <= h->scan_tmp_elems) return 0;
  if (h->capturing) return set_err(h, DEM_ERR_STATE, "scan scratch too small inside a captured step");
  invalidate_graphs(h);  // captured builds scan in the old scratch
  cudaStreamSynchronize(h->stream);
  if (h->scan_tmp) cudaFree(h->scan_tmp);
  h->scan_tmp = nullptr;
  h->scan_tmp_elems = 0;
  if (int rc = check_cuda(h, dev_alloc(h, &h->scan_tmp, need * sizeof(int)), "cudaMalloc scan")) return rc;
  h->scan_tmp_elems = need;
  return 0;
}

int exclusive_scan(dem_handle* h, int* in, int* out, int n, int* d_total, bool clear, const int* go) {
  if (n <= 0) {
    if (d_total) check_cuda(h, cudaMemsetAsync(d_total, 0, sizeof(int), h->stream), "memset");
    h->joined = true;
    return 0;
  }
  if (int rc = reserve_scan(h, n)) return rc;
  scan_rec(h, in, out, n, h->scan_tmp, d_total, clear, go);
  return check_cuda(h, cudaGetLastError(), "scan");
}

}  // namespace demb
