// Launch interfaces of the grid-map kernels (host side of the CUDA code).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace agk {

constexpr int kNX = 8;            // e-map: consecutive x points per thread
constexpr int kEmapKahan = 0;
constexpr int kEmapPlain = 1;
constexpr int kItemInterleaved = 1 << 30;  // e-map item flag: x points shared alternately with the partner column
constexpr int kEmapCtasPerSm = 3;  // e-map CTAs resident per SM (register bound 85)
constexpr int kEmapPackedBytes = 16384;  // e-map: shared-memory region of the packed table tail

// A CTA's work in the e-map: items [item0, item0+nitems) of the item list and
// the CTA's box: local origin (grid-centred frame, A) and half extents
// (scaled by 100) that contain every point of those items.
// A CTA that is one tile names it (tileMode != 0) and forms its items itself.
struct EmapBlock {
  int item0, nitems;
  short x0, x1, y0, y1, z0, z1;   // tile: items x in [x0, x1) (8 points each), rows y, planes z
  int tileMode;                   // 0: items from the list; 1 rows, 2 warp-compact, 3 warp-compact and interleaved order
  double ox, oy, oz;
  float hx, hy, hz;
  float rfar2;                    // (100 * rFar)^2, rFar >= 50 A
  int clampMid;                   // 1 if rFar + box diagonal can reach 81.9 A: clamp mid-list bins at 8191
  float rnode;                    // the largest half extent (0.01 A)
};

struct EmapParams {
  const double4* atoms;           // n_atoms (x, y, z, w), grid-centred
  int n_atoms, chunk, nsplit, nblocks;
  const int* items;               // packed (xc | y << 8 | z << 19)
  const EmapBlock* blocks;
  int nx, ny, nz, n2x, n2y, n2z;
  int64_t npoints;
  double h;
  const float* table;             // 8192 entries of 332/eps(r), FP32
  const double* thr;              // thr[k]: least r^2 whose reference bin is >= k
  float rnear2;                   // (100 * rNear)^2
  float delta;                    // guard half-width around bin edges (units of 0.01 A)
  // Packed copies of the table's saturating tail (null: not used).  Entry b
  // of the table, for b >= b16 (b8), is bits(table[8191]) + k with k stored
  // in 16 (8) bits; the 16-bit entries for bins [b16, 8192) come first, then
  // the 8-bit entries for bins [b8, 8192), each part padded to 16 bytes.
  const uint4* packed;
  int packedVecs;                 // 16-byte vectors in `packed`
  int vec8;                       // vector at which the 8-bit part starts
  int b16, b8;
  float r16sq, r8sq;              // (b16 + 2)^2, (b8 + 2)^2: mid atoms at least that far (0.01 A units) from the box
  float kScale;                   // 2^(e + 126) / g, g = table[8191] = 2^e * m: turns 100 w g 2^-16 into 100 w ulp(g) 2^133
  // Atoms at least max(rnodeMin, rnodeHalfWidths * EmapBlock::rnode) from the box (0.01 A) are summed at its nodes;
  // with the distance-dependent dielectric, from the radius on that emap_launch finds for each box, of which that
  // is the least.
  float rnodeMin;                 // +inf: none
  float rnodeHalfWidths;
  float2* radius;                 // nblocks: node and far-node radii, filled by the launch (null: constant dielectric, or no node sums)
  int testIdleWait;               // test hook: > 0 adds a wait of that many polls on a barrier nothing arrives on
  float* out;
  double* partial;                // nsplit * npoints, when nsplit > 1
  unsigned* status;
  double* checksum;               // per split: FP64 sum of the weights the split's first CTA consumed (or null)
  // Near-field mode of the far-field surrogate: only atoms within rcut of a
  // point count, each as w * (exact term - psi(r)), psi(r) = (psi[0] +
  // psi[1] r2 + psi[2] r2^2) / 100 with r2 in (0.01 A)^2 units.
  float rcut2;                    // (100 * rcut)^2
  float psi[3];
  const float4* tileLo;           // near field: per 256-atom tile, bounding box of its atoms (A)
  const float4* tileHi;
};

cudaError_t emap_launch(const EmapParams& P, bool ddd, int mode, int grid, cudaStream_t st);
// Near field of the surrogate e-map (distance-dependent dielectric, Kahan).
cudaError_t emap_near_launch(const EmapParams& P, int grid, cudaStream_t st);
// Direct e-map of the CTA boxes list[0 .. *count) (no atom split), by `grid`
// persistent CTAs; the surrogate's fallback for boxes whose probe failed.
cudaError_t emap_list_launch(const EmapParams& P, const int* list, const int* count, int* counter, int grid,
                             cudaStream_t st);
size_t emap_smem_bytes();
// Persistent e-map over the units (job, CTA box) of many jobs (no atom split, distance-dependent dielectric).
cudaError_t emap_batch_launch(const EmapParams* jobs, const int2* units, int nunits, int* counter, int grid,
                              cudaStream_t st);

// ---------------------------------------------------------------------------
// Affinity + desolvation
// ---------------------------------------------------------------------------
constexpr int kAffTX = 8, kAffTY = 8, kAffTZ = 4;   // points per CTA (one per thread)
constexpr int kAffRows = 801;                       // table rows kept: r <= 8 A
constexpr int kMaxTypes = 32;                       // receptor types
constexpr int kMaxMapsPass = 16;                    // ligand maps per pass
constexpr int kMaxMinMax = 4;                       // maps per pass with H-bond min/max bookkeeping

// Per (receptor type, map) H-bond handling, 2 bits per map in typeModes[t]
// (CalculateGridmaps.cpp:206-228): 0 add E; 1 acceptor probe vs donor atom
// (Hramp, racc weighting); 2 A1 probe vs donor atom (min/max, racc);
// 3 donor probe vs acceptor atom (min/max, rdon).
struct AffParams {
  // receptor (device)
  int n_atoms;
  const double4* xyz;             // FP64 grid-centred x, y, z (w unused)
  const int* info;                // type | hbond << 5 | disorder << 8 | rexp << 9
  const float* vol;
  const float* solq;              // solpar + solparQ * |q|
  const float4* rv8;              // per atom: rvector, 0, rvector2, 0 (FP32)
  const double* rv64;             // rvector, 3 per atom (FP64, for exact sign decisions)
  // cell list (two-point kernel: type-major keys over 4 A cells; one-point: 8 A cells)
  const int* cellStart;           // ncell + 1
  const int* cellAtoms;
  double cellLo[3];
  int ncell[3];
  const int* closestH;            // per point: index of the nearest H donor within 8 A, or -1
  // grid
  int nx, ny, nz, n2x, n2y, n2z;
  int64_t npoints;
  double h;
  // maps of this pass
  int nmaps, nmPad, ntypes, hydrogen;
  const float* table;             // [ntypes][kAffRows][nmPad] FP32
  const float* tableH;            // [kAffRows][nmPad] rows of the "HD" type (disordered donors), or null
  const float* sol;               // kAffRows
  const double* thr;              // thr[k]: least r^2 whose reference bin int(100/(1/sqrt(r^2))) is >= k
  float delta;                    // guard half-width around bin edges (units of 0.01 A)
  int typeHbond[kMaxTypes];
  unsigned typeModes[kMaxTypes];
  int typeNeedsAngular[kMaxTypes];
  int mapMinMaxSlot[kMaxMapsPass];
  int mapCov[kMaxMapsPass];
  float solparProbe[kMaxMapsPass], volProbe[kMaxMapsPass];
  float solparQ;
  float* out;                     // this pass's first map: [nmaps][npoints]
  float* dmap;
  unsigned* status;
};

size_t aff_smem_bytes(int nmPad);
cudaError_t aff_launch(const AffParams& P, cudaStream_t st);
// Persistent affinity pass over the units (job, CTA block) of many jobs.
cudaError_t aff_batch_launch(const AffParams* jobs, const int2* units, int nunits, int* counter, int nmPadMax,
                             int nmapsMax, int grid, cudaStream_t st);

// Cell list build (counting sort of atoms into cells, file order kept inside each cell).
struct CellBuild {
  const double4* xyz;
  int n_atoms;
  double lo[3];
  double edge;                    // A
  int ncell[3];
  int* cellOf;                    // n_atoms scratch
  int* count;                     // 2 * (keys + 1) scratch
  int* cellStart;                 // keys + 1
  int* cellAtoms;                 // n_atoms
  int donorsOnly;                 // only H donors (by their info bits)
  // Type-major list of the two-point affinity kernel (ntypes > 0): key = type *
  // cells + cell, and the atoms' records copied into sorted order.
  int ntypes;
  const int* info;                // type | hbond << 5 | ...
  const float *vol, *solq;
  double4* sXyz;
  float4* sAux;                   // vol, solq, info bits, atom index bits
};
// Returns the number of kernels it launched in *launched.
cudaError_t cells_launch(const CellBuild& C, cudaStream_t st, int* launched);

// ---------------------------------------------------------------------------
// Affinity + desolvation, two grid points per thread (affinity2.cu)
// ---------------------------------------------------------------------------
constexpr int kA2Slots = 4;         // H-bond maps per pass handled by the two-point kernel
constexpr int kA2PlaneRows = 804;   // rows of a slot's table plane (kAffRows, padded to 16 bytes)
enum { A2_SPH = 0, A2_D1 = 1, A2_A1 = 2, A2_A2 = 3 };          // angular class of a receptor type
enum { A2_SLOT_ACC = 0, A2_SLOT_A1 = 1, A2_SLOT_DON = 2 };     // H-bond map kind (probe class)

struct Aff2Params {
  // receptor (device)
  const double4* xyz;             // FP64 grid-centred x, y, z
  const float4* rv8;              // per atom: rvector, 0, rvector2, 0 (FP32)
  const double* rv64;             // rvector (FP64) for exact sign decisions
  // type-major cell list: the atoms of type t in cell c, in file order, are the
  // sorted entries ctStart[t * ncells + c] .. ctStart[t * ncells + c + 1]
  const int* ctStart;
  const double4* ctXyz;           // sorted: FP64 record
  const float4* ctAux;            // sorted: vol, solq, info bits, atom index bits
  double cellEdge;                // A
  double cellLo[3];
  int ncell[3];
  // grid
  int nx, ny, nz, n2x, n2y, n2z;
  int64_t npoints;
  double h;
  // maps of this pass
  int nmaps, nmPad, ntypes, hydrogen;
  // Rows [ntypes][kAffRows][aff2_row_stride(nmPad)] FP32: the maps' pair energies (0 where the
  // map is an H-bond slot for the type), the desolvation value in the last
  // column.  The first nClassTypes types of plainOrder take class rows
  // (ncPad columns, strided likewise) instead: maps whose columns are equal for all of
  // those types share a column (map g has column 4 bits of classOf from 4 g).
  const float* table;
  const float* classTable;
  int nClassTypes, ncPad;
  unsigned long long classOf;
  unsigned char plainOrder[kMaxTypes];
  int nSlotTypes;                 // types with H-bond slots, and their list
  unsigned char slotOrder[kMaxTypes];
  const double* thr;              // affinity bin thresholds (kAffRows + 1)
  float delta;                    // guard half-width around bin edges (bins)
  int needClosestH;               // some D1 type meets an acceptor-probe slot: find the nearest donor
  int typeAng[kMaxTypes];         // A2_SPH / A2_D1 / A2_A1 / A2_A2
  int nDonorTypes;                // DS and D1 types (candidates of the nearest-donor search), and their list
  unsigned char donorOrder[kMaxTypes];
  unsigned typeSlots[kMaxTypes];  // bit k: H-bond slot k applies to this type
  int nslots;
  int slotMap[kA2Slots];          // map index of each H-bond slot
  int slotKind[kA2Slots];         // A2_SLOT_*
  unsigned slotMaps;              // bit g: map g has an H-bond slot that applies to some type
  const float* slotTable;         // [ntypes][kA2Slots][kA2PlaneRows] the slots' columns, a plane each
  const float* planeH;            // the "HD" type's planes, or null
  int mapCov[kMaxMapsPass];
  float solparProbe[kMaxMapsPass], volProbe[kMaxMapsPass];
  float solparQ;
  float* out;                     // this pass's first map: [nmaps][npoints]
  float* dmap;
  unsigned* status;
  int ctaBase;                    // first CTA block of a launch (0, or a z-slab chunk's first block)
};
cudaError_t aff2_launch(const Aff2Params& P, cudaStream_t st);
// Blocks [b0, b1) of the pass (the grid's CTA blocks run z-slab by z-slab).
cudaError_t aff2_launch_range(const Aff2Params& P, int b0, int b1, cudaStream_t st);
// Floats from one table row of `columns` (a multiple of 4) to the next.
int aff2_row_stride(int columns);
// CTA blocks (work units) of the two-point kernel on an nx x ny x nz grid.
int aff2_ctas(int nx, int ny, int nz);
// Persistent two-point pass over the units (job, CTA block) of many jobs.
cudaError_t aff2_batch_launch(const Aff2Params* jobs, int njobs, const int2* units, int nunits, int* counter,
                              int nmPadMax, bool anySlots, int sms, cudaStream_t st);

// Build a pass's tables on the device from the staged pair energies.
struct AffTableJob {
  const float* energy;            // [ntypes][kAffRows][nmAll]
  const float* sol;               // kAffRows
  int ntypes, nmAll, m0, nm;      // the pass: maps m0 .. m0 + nm
  int pad1, nmPad, ncPad, nc, nslots;
  unsigned long long classMap;    // 4 bits per class: a map of it
  int slotMap[kA2Slots];
  unsigned typePlain[kMaxTypes];  // bit g: map g takes the plain table sum for this type
  float *rows1, *rows, *classRows, *planes;
};
cudaError_t aff_tables_launch(const AffTableJob& J, cudaStream_t st);

struct ClosestHParams {
  const double4* xyz;
  const int* cellStart;
  const int* cellAtoms;           // donor-only cell list
  double cellLo[3];
  int ncell[3];
  int nx, ny, nz, n2x, n2y, n2z;
  int64_t npoints;
  double h;
  int* closestH;
};
cudaError_t closest_h_launch(const ClosestHParams& P, cudaStream_t st);

// Covalent map (main.cpp:32-52) and floating grid (main.cpp:54-79).
cudaError_t covalent_launch(float* out, int nx, int ny, int nz, double h, const double cov[3], double hwInv,
                            double barrier, cudaStream_t st);
cudaError_t floating_launch(const double4* xyz, int n_atoms, int nx, int ny, int nz, double h, float* out,
                            cudaStream_t st);

}  // namespace agk
