// Set-up on the device of the mixed policy's own cell and face order: cells along a Hilbert curve
// through their centres, internal faces by their first cell in that order.  All of it runs on the
// solver's stream (keys, a stable radix sort, scans): on the host the same took 37 ns a cell, more than
// the rest of the field upload (30k cells: 1.1 of 1.6 ms).
#pragma once

#include "afar_policy.cuh"

namespace afar {

// The device's order of cells and internal faces (null: the caller's).  perm and fperm give the caller's
// cell or face of a device one, inv and finv the other way.  Ghosts and boundary faces keep their order.
struct DeviceOrder {
  const int *perm = nullptr, *inv = nullptr, *fperm = nullptr, *finv = nullptr;
  __device__ int cell(int c) const { return perm ? perm[c] : c; }
  __device__ int face(int f) const { return fperm ? fperm[f] : f; }
};

__global__ void k_box_init(long long* box) {
  if (threadIdx.x < 4) box[threadIdx.x] = threadIdx.x < 2 ? 0x7FFFFFFFFFFFFFFFll : -0x7FFFFFFFFFFFFFFFll;
}
// The smallest and largest finite coordinates of centres i, i + stride, .., as ordered integers (dkey) into box:
// (min x, min y, max x, max y).  All lanes of a warp take part.
__device__ __forceinline__ void box_of(int i, const int stride, const int n, const V2<double>* c, long long* box) {
  long long lo[2] = {0x7FFFFFFFFFFFFFFFll, 0x7FFFFFFFFFFFFFFFll}, hi[2] = {-0x7FFFFFFFFFFFFFFFll, -0x7FFFFFFFFFFFFFFFll};
  for (; i < n; i += stride) {
    const V2<double> v = c[i];
    const double x[2] = {v.x, v.y};
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      if ((dbits(x[q]) & 0x7FFFFFFFFFFFFFFFull) >= kInfBits) continue;
      const long long k = dkey(x[q]);
      lo[q] = min(lo[q], k);
      hi[q] = max(hi[q], k);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      lo[q] = min(lo[q], __shfl_xor_sync(0xffffffffu, lo[q], o));
      hi[q] = max(hi[q], __shfl_xor_sync(0xffffffffu, hi[q], o));
    }
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      atomicMin(box + q, lo[q]);
      atomicMax(box + 2 + q, hi[q]);
    }
  }
}
__global__ void __launch_bounds__(256) k_box(int n, const V2<double>* c, long long* box) {
  box_of(blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x, n, c, box);
}
__device__ __forceinline__ double undkey(const long long k) {
  return __longlong_as_double(k ^ ((k >> 63) & 0x7FFFFFFFFFFFFFFFll));
}
// Position along the Hilbert curve of order `bits` over the square at (x0, y0) of side `ext` (a coordinate that
// is not finite counts as the smallest).
__device__ __forceinline__ unsigned hilbert_key(const int bits, const V2<double> c, const double x0, const double y0,
                                                const double ext) {
  const unsigned top = (1u << bits) - 1u;
  const double scale = ext > 0.0 ? (double)top / ext : 0.0;
  const double gx = (c.x - x0) * scale, gy = (c.y - y0) * scale;
  unsigned x = gx >= 0.0 && gx <= (double)top ? (unsigned)gx : 0u, y = gy >= 0.0 && gy <= (double)top ? (unsigned)gy : 0u, d = 0;
  for (unsigned s = (top + 1) >> 1; s > 0; s >>= 1) {
    const unsigned rx = (x & s) != 0, ry = (y & s) != 0;
    d += s * s * ((3 * rx) ^ ry);
    if (!ry) {
      if (rx) {
        x = top - x;
        y = top - y;
      }
      const unsigned t = x;
      x = y;
      y = t;
    }
  }
  return d;
}
// The keys over the centres' bounding square (cells of one key keep the caller's order).
__global__ void k_hilbert_keys(int n, int bits, const V2<double>* c, const long long* box, unsigned* key, int* id) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double x0 = undkey(box[0]), y0 = undkey(box[1]);
  key[i] = hilbert_key(bits, c[i], x0, y0, fmax(undkey(box[2]) - x0, undkey(box[3]) - y0));
  id[i] = i;
}

// The whole order of up to 4096 cells in one block: a curve of order 9 at most, so that key and cell fit 32
// bits, sorted in shared memory.  Set-up of a mixed solver with this / as the launches of larger meshes: 1024
// cells 465 / 505 us, 4096 707 / 735.
constexpr int kOrderSmall = 4096;
__global__ void __launch_bounds__(1024) k_hilbert_small(int n, int bits, const V2<double>* c, int* perm) {
  __shared__ unsigned v[kOrderSmall];
  __shared__ long long box[4];
  const int t = threadIdx.x;
  if (t < 4) box[t] = t < 2 ? 0x7FFFFFFFFFFFFFFFll : -0x7FFFFFFFFFFFFFFFll;
  __syncthreads();
  box_of(t, 1024, n, c, box);
  __syncthreads();
  const double x0 = undkey(box[0]), y0 = undkey(box[1]), ext = fmax(undkey(box[2]) - x0, undkey(box[3]) - y0);
  const int N = n <= kOrderSmall / 2 ? kOrderSmall / 2 : kOrderSmall;
  for (int i = t; i < N; i += 1024)
    v[i] = i < n ? hilbert_key(bits, c[i], x0, y0, ext) << 12 | (unsigned)i : 0xFFFFFFFFu;
  for (int k = 2; k <= N; k <<= 1)  // bitonic sort
    for (int j = k >> 1; j > 0; j >>= 1) {
      __syncthreads();
      for (int p = t; p < N / 2; p += 1024) {
        const int lo = (p & ~(j - 1)) * 2 + (p & (j - 1)), hi = lo + j;
        const unsigned a = v[lo], b = v[hi];
        if ((a > b) == ((lo & k) == 0)) {
          v[lo] = b;
          v[hi] = a;
        }
      }
    }
  __syncthreads();
  for (int i = t; i < n; i += 1024) perm[i] = (int)(v[i] & (kOrderSmall - 1));
}

// ---- exclusive scan of n ints in place: block sums (2048 a block), their scan by one block, the rest
constexpr int kScan = 2048;
__device__ __forceinline__ int block_scan256(int v, int* total) {  // exclusive over 256 threads
  __shared__ int ws[8];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += u;
  }
  __syncthreads();
  if (lane == 31) ws[w] = x;
  __syncthreads();
  int base = 0, sum = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    if (k < w) base += ws[k];
    sum += ws[k];
  }
  *total = sum;
  return base + x - v;
}
__global__ void __launch_bounds__(256) k_scan_sums(int n, const int* a, int* sums) {
  int v = 0;
  for (int k = 0; k < kScan / 256; ++k) {
    const int i = blockIdx.x * kScan + k * 256 + threadIdx.x;
    if (i < n) v += a[i];
  }
  int total;
  block_scan256(v, &total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}
__global__ void __launch_bounds__(256) k_scan_top(int n, int* sums) {
  int run = 0;
  for (int b = 0; b < n; b += 256) {
    const int i = b + threadIdx.x;
    int total;
    const int e = block_scan256(i < n ? sums[i] : 0, &total);
    if (i < n) sums[i] = run + e;
    run += total;
  }
}
__global__ void __launch_bounds__(256) k_scan_apply(int n, int* a, const int* sums) {
  int run = sums[blockIdx.x];
  for (int k = 0; k < kScan / 256; ++k) {
    const int i = blockIdx.x * kScan + k * 256 + threadIdx.x;
    int total;
    const int e = block_scan256(i < n ? a[i] : 0, &total);
    if (i < n) a[i] = run + e;
    run += total;
  }
}
// all of a short array in one block, 256 at a time
__global__ void __launch_bounds__(256) k_scan_short(int n, int* a) {
  int run = 0;
  for (int k = 0; k < n; k += 256) {
    const int i = k + threadIdx.x;
    int total;
    const int e = block_scan256(i < n ? a[i] : 0, &total);
    if (i < n) a[i] = run + e;
    run += total;
  }
}
inline int scan_blocks(int n) { return (n + kScan - 1) / kScan; }
inline void device_scan(int n, int* a, int* sums, cudaStream_t st) {  // sums: scan_blocks(n) ints
  const int b = scan_blocks(n);
  if (b == 0) return;
  if (b == 1) {
    k_scan_short<<<1, 256, 0, st>>>(n, a);
    return;
  }
  k_scan_sums<<<b, 256, 0, st>>>(n, a, sums);
  k_scan_top<<<1, 256, 0, st>>>(b, sums);
  k_scan_apply<<<b, 256, 0, st>>>(n, a, sums);
}

// ---- stable sort of (key, id) pairs by 8-bit digits, 2048 pairs a block
constexpr int kSort = 2048;
__global__ void __launch_bounds__(256) k_sort_count(int n, const unsigned* key, int shift, int* cnt) {
  __shared__ int h[256];
  h[threadIdx.x] = 0;
  __syncthreads();
  for (int k = 0; k < kSort / 256; ++k) {
    const int i = blockIdx.x * kSort + k * 256 + threadIdx.x;
    if (i < n) atomicAdd(&h[(key[i] >> shift) & 255], 1);
  }
  __syncthreads();
  cnt[threadIdx.x * gridDim.x + blockIdx.x] = h[threadIdx.x];
}
__global__ void __launch_bounds__(256) k_sort_scatter(int n, const unsigned* key, const int* id, int shift,
                                                      const int* cnt, unsigned* key2, int* id2) {
  __shared__ int base[256], off[8][256];
  base[threadIdx.x] = cnt[threadIdx.x * gridDim.x + blockIdx.x];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int k = 0; k < kSort / 256; ++k) {  // 256 pairs at a time, in order
    const int i = blockIdx.x * kSort + k * 256 + threadIdx.x;
    const unsigned kv = i < n ? key[i] : 0;
    const int d = i < n ? (int)((kv >> shift) & 255) : 256;  // 256: no pair
#pragma unroll
    for (int q = 0; q < 8; ++q) off[q][threadIdx.x] = 0;
    __syncthreads();
    const unsigned same = __match_any_sync(0xffffffffu, d);
    const int rank = __popc(same & ((1u << lane) - 1));
    if (d < 256 && rank == 0) off[w][d] = __popc(same);
    __syncthreads();
    int run = base[threadIdx.x];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int c = off[q][threadIdx.x];
      off[q][threadIdx.x] = run;
      run += c;
    }
    base[threadIdx.x] = run;
    __syncthreads();
    if (d < 256) {
      const int to = off[w][d] + rank;
      key2[to] = kv;
      id2[to] = id[i];
    }
    __syncthreads();
  }
}

// The Hilbert order of n cells into perm (position -> caller's cell).  scratch: order_scratch(n) bytes.
inline size_t order_scratch(int n) {
  const size_t nb = (n + kSort - 1) / kSort;
  return 64 + 16 * (size_t)n + 4 * 256 * nb + 4 * (size_t)scan_blocks((int)(256 * nb)) + 64;
}
inline void hilbert_order(int n, const V2<double>* centre, int* perm, void* scratch, cudaStream_t st) {
  // A curve of 64 places or more a cell: a small mesh's set-up is a chain of launches, and every 8 bits of
  // the key are three of them or five (23 with the 26 bits of a large mesh).
  int bits = 4;
  while (bits < 13 && (1ll << (2 * bits)) < 64ll * n) ++bits;
  if (n <= kOrderSmall) {
    k_hilbert_small<<<1, 1024, 0, st>>>(n, bits, centre, perm);
    return;
  }
  long long* box = static_cast<long long*>(scratch);
  unsigned* key[2] = {reinterpret_cast<unsigned*>(box + 8), nullptr};
  key[1] = key[0] + n;
  int* id[2] = {reinterpret_cast<int*>(key[1] + n), nullptr};
  id[1] = id[0] + n;
  int* cnt = id[1] + n;
  const int nb = (n + kSort - 1) / kSort;
  int* sums = cnt + 256 * (size_t)nb;
  k_box_init<<<1, 32, 0, st>>>(box);
  k_box<<<nb < 512 ? nb : 512, 256, 0, st>>>(n, centre, box);
  const int passes = (2 * bits + 7) / 8;
  k_hilbert_keys<<<(n + 255) / 256, 256, 0, st>>>(n, bits, centre, box, key[0], id[0]);
  for (int pass = 0; pass < passes; ++pass) {
    const int a = pass & 1, b = a ^ 1;
    k_sort_count<<<nb, 256, 0, st>>>(n, key[a], 8 * pass, cnt);
    device_scan(256 * nb, cnt, sums, st);
    k_sort_scatter<<<nb, 256, 0, st>>>(n, key[a], id[a], 8 * pass, cnt, key[b], pass == passes - 1 ? perm : id[b]);
  }
}

// Cells, and what follows them (ghosts) in place, from the caller's order into the device's.
template <class T>
__global__ void k_gather(int Nc, int n, const T* in, T* out, DeviceOrder o) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = in[i < Nc ? o.cell(i) : i];
}

// The internal faces by their first cell in the device's order, then by the other (upper-triangular, as
// the caller's are in theirs).  pass 0 counts each cell's faces to later cells into start, pass 1 (start
// scanned) numbers them.  Every internal face is in the lists of both its cells, once (checked by the
// caller of this).
__global__ void k_face_order(int Nc, int Nf, int maxM, const uint8_t* nM, const int* cellFaces, const int* neighbour,
                             DeviceOrder o, int* start, int* fperm, int* finv, int pass) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= Nc) return;
  const int h = o.perm[c];
  int other[4], face[4], n = 0;
  for (int i = 0; i < nM[c] && i < 4; ++i) {
    const int fid = cellFaces[(size_t)maxM * h + i], f = abs(fid) - 1;
    if (f >= Nf) continue;
    const int x = o.inv[neighbour[2 * (size_t)f + (fid > 0)]];
    if (x < c || (x == c && fid < 0)) continue;  // a face of a cell with itself counts once
    int k = n++;
    while (k > 0 && (other[k - 1] > x || (other[k - 1] == x && face[k - 1] > f))) {
      other[k] = other[k - 1];
      face[k] = face[k - 1];
      --k;
    }
    other[k] = x;
    face[k] = f;
  }
  if (pass == 0) {
    start[c] = n;
  } else {
    for (int k = 0; k < n; ++k) {
      fperm[start[c] + k] = face[k];
      finv[face[k]] = start[c] + k;
    }
  }
}
// Owners and neighbours in the device's order (a face keeps its owner).
__global__ void k_setup_owners(int Nf, const int2* raw, int2* on, DeviceOrder o) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= Nf) return;
  const int2 h = raw[o.face(f)];
  on[f] = o.inv ? int2{o.inv[h.x], o.inv[h.y]} : h;
}
// The cells' list lengths in the device's order, the way back to it (inv, where there is one), and the largest
// stencil of each 128-cell tile (at least 1: the tile kernel loads the boxes of that size).
__global__ void __launch_bounds__(128) k_setup_counts(int Nc, const uint8_t* nS0, const uint8_t* nM0, uint8_t* nS,
                                                      uint8_t* nM, uint8_t* tileS, int* inv, DeviceOrder o) {
  __shared__ int m;
  if (threadIdx.x == 0) m = 1;
  __syncthreads();
  const int c = blockIdx.x * 128 + threadIdx.x;
  if (c < Nc) {
    const int h = o.cell(c);
    nS[c] = nS0[h];
    nM[c] = nM0[h];
    if (inv) inv[h] = c;
    atomicMax(&m, (int)nS0[h]);
  }
  __syncthreads();
  if (threadIdx.x == 0) tileS[blockIdx.x] = (uint8_t)m;
}

}  // namespace afar
