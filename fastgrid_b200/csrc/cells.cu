// Helper kernels of the affinity pass and the small per-point maps:
//  * the device cell list (counting sort of atoms into cells, file order
//    kept inside each cell) that replaces FastGrid's cutoff grid
//    (SpatialGrid.h:50-315),
//  * the nearest H donor of every grid point (the role of FastGrid's ANN
//    kd-tree query, CalculateGridmaps.cpp:246-250, 417-431),
//  * the covalent map (main.cpp:32-52) and the floating grid (main.cpp:54-79).
#include <cuda_runtime.h>

#include <cstdint>

#include "ag_device.cuh"
#include "ag_kernels.h"

namespace agk {

// Exact FP64 squared distance as the reference forms it (Vec3d::MagnitudeSqr
// of atom - gridPos, left to right, separately rounded).
__device__ __forceinline__ double rsq_exact_c(double ax, double ay, double az, double gx, double gy, double gz) {
  const double dx = __dsub_rn(ax, gx), dy = __dsub_rn(ay, gy), dz = __dsub_rn(az, gz);
  return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
}

// ---------------------------------------------------------------------------
// Cell list: counting sort into cells (or into type-major (type, cell) keys);
// file order inside each key.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int cell_key(const CellBuild& C, int i) {
  if (C.donorsOnly && ((C.info[i] >> 5) & 7) != 1 && ((C.info[i] >> 5) & 7) != 2) return -1;  // DS, D1
  const double4 a = C.xyz[i];
  const int cx = (int)floor((a.x - C.lo[0]) / C.edge), cy = (int)floor((a.y - C.lo[1]) / C.edge),
            cz = (int)floor((a.z - C.lo[2]) / C.edge);
  if (cx < 0 || cy < 0 || cz < 0 || cx >= C.ncell[0] || cy >= C.ncell[1] || cz >= C.ncell[2]) return -1;
  const int type = C.ntypes > 0 ? C.info[i] & 31 : 0;
  return ((type * C.ncell[2] + cz) * C.ncell[1] + cy) * C.ncell[0] + cx;
}

// Atom v's record at place `at` of the sorted order.
__device__ __forceinline__ void place_record(const CellBuild& C, int at, int v) {
  C.sXyz[at] = C.xyz[v];
  C.sAux[at] = make_float4(C.vol[v], C.solq[v], __int_as_float(C.info[v]), __int_as_float(v));
}

__global__ void cell_count_kernel(CellBuild C) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < C.n_atoms; i += gridDim.x * blockDim.x) {
    const int key = cell_key(C, i);
    C.cellOf[i] = key;
    if (key >= 0) atomicAdd(&C.count[key], 1);
  }
}

// Exclusive scan over the CTA's threads of v; `sum` receives the total.
__device__ __forceinline__ int block_scan(int v, int* warpSums, int& sum) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += u;
  }
  __syncthreads();  // the previous scan's sums are read
  if (lane == 31) warpSums[warp] = incl;
  __syncthreads();
  int off = 0;
  sum = 0;
  for (int w = 0; w < nw; w++) {
    if (w == warp) off = sum;
    sum += warpSums[w];
  }
  return off + incl - v;
}

// Exclusive scan of the counts by one CTA, 8,192 keys per round.
__global__ void __launch_bounds__(1024) cell_scan_kernel(const int* count, int n, int* start) {
  __shared__ int warpSums[32];
  int carry = 0;
  for (int b = 0; b < n; b += 8192) {
    const int i0 = b + 8 * threadIdx.x;
    int c[8], s = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) {
      c[k] = i0 + k < n ? count[i0 + k] : 0;
      s += c[k];
    }
    int total;
    int run = carry + block_scan(s, warpSums, total);
#pragma unroll
    for (int k = 0; k < 8; k++) {
      if (i0 + k < n) start[i0 + k] = run;
      run += c[k];
    }
    carry += total;
  }
  if (threadIdx.x == 0) start[n] = carry;
}

__global__ void cell_scatter_kernel(CellBuild C, int* fill) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < C.n_atoms; i += gridDim.x * blockDim.x) {
    const int cell = C.cellOf[i];
    if (cell >= 0) C.cellAtoms[C.cellStart[cell] + atomicAdd(&fill[cell], 1)] = i;
  }
}

// Restore file order inside each key (one warp per key, rank sort); the
// type-major list gets the sorted records instead of the indexes.
__global__ void cell_sort_kernel(CellBuild C, int nkeys) {
  const int warpsPerBlock = blockDim.x / 32;
  const int lane = threadIdx.x & 31;
  int* tmp = C.cellOf;  // n_atoms entries, free after the scatter
  for (int c = blockIdx.x * warpsPerBlock + threadIdx.x / 32; c < nkeys; c += gridDim.x * warpsPerBlock) {
    const int b = C.cellStart[c], e = C.cellStart[c + 1];
    for (int i = b + lane; i < e; i += 32) {
      const int v = C.cellAtoms[i];
      int rank = 0;
      for (int j = b; j < e; j++) rank += C.cellAtoms[j] < v;
      if (C.ntypes > 0) place_record(C, b + rank, v);
      else tmp[b + rank] = v;
    }
    if (C.ntypes > 0) continue;
    __syncwarp();
    for (int i = b + lane; i < e; i += 32) C.cellAtoms[i] = tmp[i];
  }
}

// The whole type-major list by one CTA, its counts in shared memory: small
// receptors are bound by the launches of the four kernels, not by their work
// (2,000 atoms: one launch of 9 us instead of six of 3 us each).
__global__ void __launch_bounds__(1024) cell_list_kernel(CellBuild C, int nkeys) {
  extern __shared__ int cnt[];  // nkeys + 1
  __shared__ int warpSums[32];
  for (int k = threadIdx.x; k <= nkeys; k += blockDim.x) cnt[k] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < C.n_atoms; i += blockDim.x) {
    const int key = cell_key(C, i);
    C.cellOf[i] = key;
    if (key >= 0) atomicAdd(&cnt[key], 1);
  }
  __syncthreads();
  const int per = (nkeys + blockDim.x - 1) / blockDim.x;
  const int b = min(nkeys, (int)threadIdx.x * per), e = min(nkeys, b + per);
  int s = 0;
  for (int k = b; k < e; k++) s += cnt[k];
  int total;
  int run = block_scan(s, warpSums, total);
  for (int k = b; k < e; k++) {
    const int c = cnt[k];
    cnt[k] = run;
    C.cellStart[k] = run;
    run += c;
  }
  if (threadIdx.x == 0) C.cellStart[nkeys] = total;
  __syncthreads();
  for (int i = threadIdx.x; i < C.n_atoms; i += blockDim.x) {
    const int key = C.cellOf[i];
    if (key >= 0) C.cellAtoms[atomicAdd(&cnt[key], 1)] = i;
  }
  __syncthreads();  // cnt[key] is now the end of the key's atoms
  for (int i = threadIdx.x; i < C.n_atoms; i += blockDim.x) {
    const int key = C.cellOf[i];
    if (key < 0) continue;
    const int kb = key > 0 ? cnt[key - 1] : 0, ke = cnt[key];
    int rank = 0;
    for (int j = kb; j < ke; j++) rank += C.cellAtoms[j] < i;
    place_record(C, kb + rank, i);
  }
}

cudaError_t cells_launch(const CellBuild& C, cudaStream_t st, int* launched) {
  const int nkeys = C.ncell[0] * C.ncell[1] * C.ncell[2] * (C.ntypes > 0 ? C.ntypes : 1);
  // One CTA where its serial work is short (a round of 1,024 atoms takes about
  // 1 us and 1,024 keys 0.5 us) and the counts fit shared memory.
  if (C.ntypes > 0 && C.n_atoms <= 8192 && nkeys <= 32768) {
    const size_t smem = sizeof(int) * (size_t)(nkeys + 1);
    cudaError_t e = cudaFuncSetAttribute(cell_list_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    cell_list_kernel<<<1, 1024, smem, st>>>(C, nkeys);
    *launched += 1;
    return cudaGetLastError();
  }
  cudaError_t e = cudaMemsetAsync(C.count, 0, sizeof(int) * 2 * ((size_t)nkeys + 1), st);
  if (e != cudaSuccess) return e;
  const int blocks = max(1, min(1184, (C.n_atoms + 255) / 256));
  cell_count_kernel<<<blocks, 256, 0, st>>>(C);
  cell_scan_kernel<<<1, 1024, 0, st>>>(C.count, nkeys, C.cellStart);
  cell_scatter_kernel<<<blocks, 256, 0, st>>>(C, C.count + nkeys + 1);
  cell_sort_kernel<<<max(1, min(2048, (nkeys + 7) / 8)), 256, 0, st>>>(C, nkeys);
  *launched += 4;
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Nearest H donor per grid point (argmin over DS/D1 atoms within the 27 cells
// around the point's cell, ties to the lower file index), FP64 like the
// reference's kd-tree query (CalculateGridmaps.cpp:246-250).
// ---------------------------------------------------------------------------
__global__ void closest_h_kernel(ClosestHParams P) {
  for (int64_t pt = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; pt < P.npoints;
       pt += (int64_t)gridDim.x * blockDim.x) {
    const int ix = (int)(pt % P.nx), iy = (int)((pt / P.nx) % P.ny), iz = (int)(pt / ((int64_t)P.nx * P.ny));
    const double gx = __dmul_rn((double)(ix - P.n2x), P.h), gy = __dmul_rn((double)(iy - P.n2y), P.h),
                 gz = __dmul_rn((double)(iz - P.n2z), P.h);
    const int cx = (int)floor((gx - P.cellLo[0]) / 8.0), cy = (int)floor((gy - P.cellLo[1]) / 8.0),
              cz = (int)floor((gz - P.cellLo[2]) / 8.0);
    int best = -1;
    double bestR = 1e300;
    for (int dz = -1; dz <= 1; dz++)
      for (int dy = -1; dy <= 1; dy++)
        for (int dx = -1; dx <= 1; dx++) {
          const int x = cx + dx, y = cy + dy, z = cz + dz;
          if (x < 0 || y < 0 || z < 0 || x >= P.ncell[0] || y >= P.ncell[1] || z >= P.ncell[2]) continue;
          const int c = (z * P.ncell[1] + y) * P.ncell[0] + x;
          for (int j = P.cellStart[c]; j < P.cellStart[c + 1]; j++) {
            const int ia = P.cellAtoms[j];
            const double4 a = P.xyz[ia];
            const double r = rsq_exact_c(a.x, a.y, a.z, gx, gy, gz);
            if (r < bestR || (r == bestR && ia < best)) { bestR = r; best = ia; }
          }
        }
    P.closestH[pt] = (bestR <= 64.0) ? best : -1;
  }
}

cudaError_t closest_h_launch(const ClosestHParams& P, cudaStream_t st) {
  const int64_t blocks = (P.npoints + 255) / 256;
  closest_h_kernel<<<(int)(blocks < 65535 * 16 ? blocks : 65535 * 16), 256, 0, st>>>(P);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Covalent map and floating grid
// ---------------------------------------------------------------------------
__global__ void covalent_kernel(float* out, int nx, int ny, int nz, double h, double cx, double cy, double cz,
                                double hwInv, double barrier) {
  const int64_t n = (int64_t)nx * ny * nz;
  for (int64_t pt = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; pt < n; pt += (int64_t)gridDim.x * blockDim.x) {
    const int ix = (int)(pt % nx), iy = (int)((pt / nx) % ny), iz = (int)(pt / ((int64_t)nx * ny));
    const double dx = cx - __dmul_rn((double)(ix - nx / 2), h), dy = cy - __dmul_rn((double)(iy - ny / 2), h),
                 dz = cz - __dmul_rn((double)(iz - nz / 2), h);
    double r = __dmul_rn(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz)), hwInv);
    if (r < 1.0e-12) r = 1.0e-12;
    out[pt] = (float)(barrier * (1 - exp(-0.69314718055994529 * r)));
  }
}

cudaError_t covalent_launch(float* out, int nx, int ny, int nz, double h, const double cov[3], double hwInv,
                            double barrier, cudaStream_t st) {
  covalent_kernel<<<1184, 256, 0, st>>>(out, nx, ny, nz, h, cov[0], cov[1], cov[2], hwInv, barrier);
  return cudaGetLastError();
}

__global__ void floating_kernel(const double4* xyz, int n, int nx, int ny, int nz, double h, float* out) {
  __shared__ double4 tile[256];
  const int64_t np = (int64_t)nx * ny * nz;
  const int64_t pt = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const bool valid = pt < np;
  const int ix = (int)(pt % nx), iy = (int)((pt / nx) % ny), iz = (int)(pt / ((int64_t)nx * ny));
  const double gx = (double)(ix - nx / 2) * h, gy = (double)(iy - ny / 2) * h, gz = (double)(iz - nz / 2) * h;
  double best = 1e24;
  for (int t0 = 0; t0 < n; t0 += 256) {
    if (t0 + (int)threadIdx.x < n) tile[threadIdx.x] = xyz[t0 + threadIdx.x];
    __syncthreads();
    const int m = min(256, n - t0);
    for (int j = 0; j < m; j++) {
      const double dx = tile[j].x - gx, dy = tile[j].y - gy, dz = tile[j].z - gz;
      const double r = dx * dx + dy * dy + dz * dz;
      best = r < best ? r : best;
    }
    __syncthreads();
  }
  if (valid) out[pt] = (float)sqrt(best);
}

cudaError_t floating_launch(const double4* xyz, int n, int nx, int ny, int nz, double h, float* out,
                            cudaStream_t st) {
  const int64_t np = (int64_t)nx * ny * nz;
  floating_kernel<<<(int)((np + 255) / 256), 256, 0, st>>>(xyz, n, nx, ny, nz, h, out);
  return cudaGetLastError();
}

}  // namespace agk
