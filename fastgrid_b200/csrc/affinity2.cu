// Affinity maps for every ligand type plus the desolvation map, two grid
// points per thread (FastGrid CalculateGridmaps.cpp:84-316).
//
// The arithmetic and the exact edge decisions are those of affinity_kernel
// (affinity.cu): FP32 geometry in a CTA-local frame; the 8 A cutoff, the
// 0.01 A table bin and the sign of cos(theta) for D1 and ordered A2 atoms
// decided in FP64 exactly as the reference computes them whenever the FP32
// value lies in a guard band around the edge.  What changes is the
// organisation, for fewer instructions per point-atom pair:
//
//  * each thread holds two z-neighbouring points, whose geometry is packed
//    FP32x2: one shared-memory record and one guard test per candidate serve both;
//  * a block covers 8 x 8 x 8 points and each warp a 4 x 4 x 4 sub-box; a warp
//    walks only the candidates within 8 A of its own sub-box;
//  * a block is two CTAs that add into zeroed slot maps: PLAIN sums whole table
//    rows, SLOTS the maps whose H-bond term applies to a type (at most four per
//    pass).  Apart they need 80 registers instead of 128 and share an SM;
//  * candidates are gathered from a type-major cell list (a type's cells of one
//    row along x are one run, file order inside each cell), so a batch arrives
//    sorted by receptor type without a sort, and each type's table is loaded
//    once per batch (one TMA bulk copy);
//  * the plain sums add whole table rows with packed FP32x2 adds; a slot map's
//    column is zero there, maps whose columns agree for every type share one, and
//    the last column carries the desolvation value;
//  * a point beyond 8 A of the atom reads an all-zero extra table row, so the
//    plain sums need no branch;
//  * the nearest H donor of each point (the reference's kd-tree query,
//    CalculateGridmaps.cpp:246-250) is found in the kernel from the donors
//    within 8 A of the box, exactly in FP64 with ties to the lower file index,
//    before the map sums need it.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <cstdint>

#include "ag_device.cuh"
#include "ag_kernels.h"

// Lambdas that must be inlined: their captured sums stay in registers.
#define AG_INLINE __attribute__((always_inline))

namespace agk {

using namespace agd;

namespace {

constexpr int kT = 256;              // threads per CTA, two points each
constexpr int kW = kT / 32;
constexpr int kSegs = kT;            // cell-list segments per gather round (one per thread)
constexpr float kBias = 8388608.f;   // 2^23

constexpr int kPlaneRows = kA2PlaneRows;
static_assert(kPlaneRows >= kAffRows && kPlaneRows * sizeof(float) % 16 == 0, "plane rows");

// The two CTAs of a block: PLAIN forms the whole-row map sums of every type,
// SLOTS the H-bond slots, from the types they apply to.
enum { PART_PLAIN = 0, PART_SLOTS = 1 };

// Candidate data only one of the parts needs.
template <int PART>
struct PartSmem;
template <>
struct PartSmem<PART_PLAIN> {
  static constexpr int kCap = 640;   // candidate atoms per batch
  float2 vs[kCap];                   // vol, solq
};
template <>
struct PartSmem<PART_SLOTS> {
  static constexpr int kCap = 512;
  float4 rvA[kCap];                  // rvector x, y, z, rvector2 x
  float2 rvB[kCap];                  // rvector2 y, z
  float4 rch[kT][2];                 // per thread and point: rvector of the nearest H donor
};

// The CTA's box in the grid-centred frame and the cells around it.
struct Box {
  double ox, oy, oz;                 // CTA frame origin (its first lattice point)
  double lo[3], hi[3];               // CTA box
  int c0[3], ncx, ncy, nrows;        // cells around the box: nrows rows of ncx cells along x
};

template <int PART>
struct A2Smem : PartSmem<PART> {
  using PartSmem<PART>::kCap;
  float4 pos[kCap];                  // CTA-local x, y, z; w = info bits
  int idx[kCap];                     // atom index
  unsigned short wlist[kW][kCap];    // per warp: candidates within 8 A of its sub-box
  int wStart[kW][kMaxTypes + 1];     // per warp: first wlist entry of each type (in the part's type order)
  int typeCount[kMaxTypes];
  int typeStart[kMaxTypes + 1];
  int segPre[kSegs + 1];             // atoms before each segment of the round
  int segBeg[kSegs];                 // each segment's first entry in the sorted atoms
  int cnt[kW];
  Box box;
  float sblo[kW][3], sbhi[kW][3];    // each warp's sub-box in the CTA frame (lo > hi: past the grid edge)
};

// The barrier of a CTA's table copies.  It has shared memory of its own and is
// set up once per CTA: the parts lay out the dynamic memory differently, and
// an mbarrier's memory must not hold anything else while it is valid.
struct TableBar {
  uint64_t* bar;
  unsigned phase;                    // copies waited for so far
  __device__ __forceinline__ void init(uint64_t* b) {
    bar = b;
    phase = 0;
    if (threadIdx.x == 0) {
      mbar_init(b, 1);
      fence_barrier_init();
    }
    __syncthreads();
  }
};

// Dynamic shared memory: A2Smem, then the current type's table.  PLAIN: rows of
// ncPad or nmPad columns, an extra all-zero row last (points beyond the
// cutoff).  SLOTS: one plane per H-bond slot; the nearest-donor search keeps
// each candidate's FP64 record there (the two phases do not overlap).
template <int PART>
__host__ __device__ constexpr size_t tabOffset() {
  return ((sizeof(A2Smem<PART>) + 127) / 128) * 128;
}
constexpr size_t kSlotsRegion = kA2Slots * kPlaneRows * sizeof(float) > PartSmem<PART_SLOTS>::kCap * sizeof(double4)
                                    ? kA2Slots * kPlaneRows * sizeof(float)
                                    : PartSmem<PART_SLOTS>::kCap * sizeof(double4);

__device__ __forceinline__ double rsq64(double ax, double ay, double az, double gx, double gy, double gz) {
  const double dx = __dsub_rn(ax, gx), dy = __dsub_rn(ay, gy), dz = __dsub_rn(az, gz);
  return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
}

// Exact FP64 cos(theta) = -dot(unit(atom - gridPos), rvector) (CalculateGridmaps.cpp:89).
__device__ double costheta64(double ax, double ay, double az, double gx, double gy, double gz, const double* rv) {
  const double dx = __dsub_rn(ax, gx), dy = __dsub_rn(ay, gy), dz = __dsub_rn(az, gz);
  double rSq = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
  if (rSq < 1.0e-24) rSq = 1.0e-24;
  const double invR = __drcp_rn(__dsqrt_rn(rSq));
  const double ux = __dmul_rn(dx, invR), uy = __dmul_rn(dy, invR), uz = __dmul_rn(dz, invR);
  return -__dadd_rn(__dadd_rn(__dmul_rn(ux, rv[0]), __dmul_rn(uy, rv[1])), __dmul_rn(uz, rv[2]));
}

__device__ __forceinline__ float acos_clamped(float f) { return (f > 1.f) ? 0.f : (f < -1.f) ? 3.14159265f : acosf(f); }

// A thread's two points (p = 0, 1 at z and z + 1).
struct Pts {
  float px, py;
  float2 npz;                        // minus their z; 1e4 for a point past the grid edge: candidates have z >= -8 A,
                                     // so it is beyond every cutoff
  int ix, iy, iz0;
};

// Their plain sums.
template <int NMAX>
struct PlainSums {
  float2 em[2][NMAX / 2];            // maps (2i, 2i+1)
  float s1[2], s2[2];                // desolvation sums (sol * vol, sol * solq)
};

// Their H-bond slots.
struct SlotSums {
  int ch[2];                         // nearest H donor, or -1 (its rvector is in shared memory)
  float mn[2][kA2Slots], mx[2][kA2Slots];  // additive sum (acceptor probes) or min / max
  unsigned fl[2];                    // per slot: a min / max value was recorded
};

// FP64 grid-point coordinate as the reference forms it.
__device__ __forceinline__ double gcoord(int i, int n2, double h) { return __dmul_rn((double)(i - n2), h); }

constexpr uint32_t kBiasBits = 0x4B000000u;  // bits of 2^23

// One candidate against the two points: offsets, 1 / r, table row and whether
// the point is within the 8 A cutoff.  Packed FP32 over the two points.
// Returns false if the candidate is for no lane.
struct Pair {
  float dx, dy;
  float2 dz, rs;
  uint32_t row[2];                   // kBiasBits + table row; row kAffRows (all zero) beyond the cutoff
  bool in[2];
  __device__ __forceinline__ bool set(const Aff2Params& P, const int* idx, const int c, const float4 a, const Pts& q) {
    dx = a.x - q.px;
    dy = a.y - q.py;
    // The 1e-30 keeps r^2 > 0 (an atom on a grid point).
    const float dxy = fmaf(dy, dy, dx * dx) + 1.0e-30f;
    dz = __fadd2_rn(make_float2(a.z, a.z), q.npz);
    const float2 r2 = __ffma2_rn(dz, dz, make_float2(dxy, dxy));
    in[0] = r2.x <= 64.0002f;
    in[1] = r2.y <= 64.0002f;
    if (!__any_sync(0xffffffffu, in[0] || in[1])) return false;
    rs = make_float2(rsqrt_approx(r2.x), rsqrt_approx(r2.y));
    const float2 rs100 = __fmul2_rn(rs, make_float2(100.f, 100.f)), bias = make_float2(kBias, kBias);
    const float2 kf = __ffma2_rd(r2, rs100, bias);   // 2^23 + floor(100 r)
    const float2 kn = __ffma2_rn(r2, rs100, bias);   // 2^23 + the integer nearest 100 r
    const float2 d = __ffma2_rn(r2, rs100, __ffma2_rn(kn, make_float2(-1.f, -1.f), bias));  // 100 r minus it
    const float2 t = __fadd2_rn(r2, make_float2(-64.f, -64.f));
    uint32_t b[2] = {__float_as_uint(kf.x), __float_as_uint(kf.y)};
    // Within the guard band of a bin edge or of the cutoff: the reference's
    // FP64 decisions (its bin int(100 / (1 / sqrt(r^2))) through the table of
    // r^2 thresholds).
    if (min(fabsf(d.x), fabsf(d.y)) < P.delta || min(fabsf(t.x), fabsf(t.y)) < 2.0e-4f) {
      const double4 a64 = P.xyz[idx[c]];
#pragma unroll
      for (int p = 0; p < 2; p++) {
        const float dp = p ? d.y : d.x, tp = p ? t.y : t.x;
        if (!in[p] || !(fabsf(dp) < P.delta || fabsf(tp) < 2.0e-4f)) continue;
        const double r64 = rsq64(a64.x, a64.y, a64.z, gcoord(q.ix, P.n2x, P.h), gcoord(q.iy, P.n2y, P.h),
                                 gcoord(q.iz0 + p, P.n2z, P.h));
        if (r64 > 64.0) in[p] = false;
        const int k = min((int)(__float_as_uint(p ? kn.y : kn.x) - kBiasBits), kAffRows);
        if (fabsf(dp) < P.delta) b[p] = kBiasBits + (uint32_t)(k == 0 ? 0 : r64 >= P.thr[k] ? k : k - 1);
      }
    }
#pragma unroll
    for (int p = 0; p < 2; p++) row[p] = in[p] ? b[p] : kBiasBits + kAffRows;
    return true;
  }
};

// Whether a candidate is left out: the reference skips disordered hydrogens
// (CalculateGridmaps.cpp:280).  ISH: the candidate's type is "HD".
template <bool ISH>
__device__ __forceinline__ bool skipped(const float4 a) {
  return ISH && ((__float_as_int(a.w) >> 8) & 1);
}

// Distance between table rows of rowQ float4s, in float4s: odd, so that the
// rows a quarter-warp reads at once start in any of the eight 16-byte bank
// groups (rows 8 columns apart would meet in four of them).
__host__ __device__ constexpr int row_stride(int rowQ) { return rowQ | 1; }

// Plain sums of one receptor type's candidates in this warp's list: whole table
// rows of rowQ float4s, whose last entry is the desolvation value.
template <int NMAX, bool ISH>
__device__ __forceinline__ void plain_sums(const Aff2Params& P, const A2Smem<PART_PLAIN>& S, const float* tab,
                                           const int rowQ, const int j0, const int j1, const unsigned short* wl,
                                           const Pts& q, PlainSums<NMAX>& s) {
  const int strideQ = row_stride(rowQ);
  // Shared-window address of the row with bits kBiasBits + row: the bias is in
  // the base (mod 2^32).
  const uint32_t stride = 16u * (uint32_t)strideQ, base = smem_u32(tab) - kBiasBits * stride;
  // The next candidate's record is read one iteration ahead (its shared-memory
  // latency overlaps the current candidate's arithmetic).
  int cNext = j0 < j1 ? wl[j0] : 0;
  float4 aNext = j0 < j1 ? S.pos[cNext] : make_float4(0.f, 0.f, 0.f, 0.f);
  for (int jj = j0; jj < j1; jj++) {
    const int c = cNext;
    const float4 a = aNext;
    if (jj + 1 < j1) {
      cNext = wl[jj + 1];
      aNext = S.pos[cNext];
    }
    Pair w;
    if (skipped<ISH>(a) || !w.set(P, S.idx, c, a, q)) continue;  // uniform: one candidate
    float solv[2] = {0.f, 0.f};
    const uint32_t at[2] = {base + w.row[0] * stride, base + w.row[1] * stride};
#pragma unroll
    for (int g4 = 0; g4 < NMAX / 4; g4++) {
      if (g4 >= rowQ) break;         // uniform
#pragma unroll
      for (int p = 0; p < 2; p++) {
        float4 e4;
        asm("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
            : "=f"(e4.x), "=f"(e4.y), "=f"(e4.z), "=f"(e4.w)
            : "r"(at[p] + 16u * g4));
        s.em[p][2 * g4] = __fadd2_rn(s.em[p][2 * g4], make_float2(e4.x, e4.y));
        s.em[p][2 * g4 + 1] = __fadd2_rn(s.em[p][2 * g4 + 1], make_float2(e4.z, e4.w));
        solv[p] = e4.w;
      }
    }
    const float2 v = S.vs[c];
#pragma unroll
    for (int p = 0; p < 2; p++) {
      s.s1[p] = fmaf(solv[p], v.x, s.s1[p]);
      s.s2[p] = fmaf(solv[p], v.y, s.s2[p]);
    }
  }
}

// From column-class sums to map sums: each map takes its class's sum.
template <int NMAX>
__device__ __forceinline__ void expand_classes(const Aff2Params& P, PlainSums<NMAX>& s) {
#pragma unroll
  for (int p = 0; p < 2; p++) {
    float old[NMAX], v[NMAX];
#pragma unroll
    for (int g = 0; g < NMAX; g++) old[g] = (g & 1) ? s.em[p][g >> 1].y : s.em[p][g >> 1].x;
#pragma unroll
    for (int g = 0; g < NMAX; g++) {
      const int c = (int)(P.classOf >> (4 * g)) & 15;
      v[g] = 0.f;
#pragma unroll
      for (int k = 0; k < NMAX; k++) v[g] = k == c ? old[k] : v[g];
    }
#pragma unroll
    for (int g = 0; g < NMAX / 2; g++) s.em[p][g] = make_float2(v[2 * g], v[2 * g + 1]);
  }
}

// H-bond slots of one receptor type's candidates (CalculateGridmaps.cpp:199-232)
// with the directional factors of its angular class ANG (:84-197).
template <int ANG, bool ISH>
__device__ __forceinline__ void slot_terms(const Aff2Params& P, const A2Smem<PART_SLOTS>& S, const float* tab,
                                           const int j0, const int j1, const unsigned short* wl, const unsigned slots,
                                           const Pts& q, SlotSums& s) {
  int cNext = j0 < j1 ? wl[j0] : 0;
  float4 aNext = j0 < j1 ? S.pos[cNext] : make_float4(0.f, 0.f, 0.f, 0.f);
  for (int jj = j0; jj < j1; jj++) {
    const int c = cNext;
    const float4 a = aNext;
    if (jj + 1 < j1) {
      cNext = wl[jj + 1];
      aNext = S.pos[cNext];
    }
    Pair w;
    if (skipped<ISH>(a) || !w.set(P, S.idx, c, a, q)) continue;  // uniform: one candidate
    const int info = __float_as_int(a.w);
    const bool dis = (info >> 8) & 1;
    float racc[2] = {1.f, 1.f}, rdon[2] = {1.f, 1.f}, hramp[2] = {1.f, 1.f};
    if (ANG != A2_SPH) {
      const int idx = S.idx[c];
      const float4 ra = S.rvA[c];
      const float2 rb = S.rvB[c];
#pragma unroll
      for (int p = 0; p < 2; p++) {
        if (!w.in[p]) continue;
        const float rsp = p ? w.rs.y : w.rs.x;
        const float ux = w.dx * rsp, uy = w.dy * rsp, uz = (p ? w.dz.y : w.dz.x) * rsp;
        float cosT = -(ux * ra.x + uy * ra.y + uz * ra.z);
        bool gt0 = cosT > 0.f, ge0 = cosT >= 0.f;
        if ((ANG == A2_D1 || (ANG == A2_A2 && !dis)) && fabsf(cosT) < 1.0e-5f) {
          // The D1 and ordered-A2 factors jump where cos(theta) changes sign.
          const double4 a64 = P.xyz[idx];
          const double c64 = costheta64(a64.x, a64.y, a64.z, gcoord(q.ix, P.n2x, P.h), gcoord(q.iy, P.n2y, P.h),
                                        gcoord(q.iz0 + p, P.n2z, P.h), P.rv64 + 3 * (size_t)idx);
          cosT = (float)c64;
          gt0 = c64 > 0.0;
          ge0 = c64 >= 0.0;
        }
        if (ANG == A2_D1) {
          racc[p] = 0.f;
          if (gt0) {
            float ra2 = cosT;
            const int rexp = (info >> 9) & 7;
            if (rexp == 4) ra2 = ra2 * ra2;
            if (rexp == 4 || rexp == 2) ra2 = ra2 * ra2;
            racc[p] = ra2;
            if (idx != s.ch[p] && s.ch[p] >= 0) {
              const float4 rc = S.rch[threadIdx.x][p];
              const float cc = rc.x * ra.x + rc.y * ra.y + rc.z * ra.z;
              // cos on the SFU over [0, pi]; cos(x) = cos(2 pi - x) folds 4 theta / 3.
              const float xr = acos_clamped(cc) * (120.f / 90.f);
              hramp[p] = 0.5f - 0.5f * __cosf(fminf(xr, 6.28318531f - xr));
            }
          }
        } else if (ANG == A2_A1) {
          rdon[p] = gt0 ? cosT * cosT : 0.f;
        } else {  // A2
          if (dis) {
            // theta <= 1.24791 + pi/2  <=>  cos(theta) >= -sin(1.24791)
            racc[p] = 0.f;
            rdon[p] = 0.f;
            if (cosT >= -0.94832352f) {
              const float sn = sqrtf(fmaxf(0.f, 1.f - cosT * cosT));
              const float cs = cosT * 0.31730505f + sn * 0.94832352f;  // cos(theta - 1.24791)
              rdon[p] = (cs * cs) * (cs * cs);
              racc[p] = rdon[p];
            }
          } else {
            float rd = 0.f;
            if (ge0) {
              // sin(2 ti), ti = |acos(x) - pi/2| = |asin(x)|:  2 |x| sqrt(1 - x^2)
              const float cxp = uy * rb.y - uz * rb.x;
              const float cyp = uz * ra.w - ux * rb.y;
              const float czp = ux * rb.x - uy * ra.w;
              const float rd2 = fmaxf(cxp * cxp + cyp * cyp + czp * czp, 1.0e-6f);
              float x = rsqrt_approx(rd2) * (cxp * ra.x + cyp * ra.y + czp * ra.z);
              x = fminf(fabsf(x), 1.f);
              rd = 0.9f + 0.2f * x * sqrtf(fmaxf(0.f, 1.f - x * x));
            } else if (cosT >= -0.34202f) {
              const float qq = 0.116978f - cosT * cosT;
              rd = 562.25f * (qq * qq * qq);
            }
            // cos(pi/2 - acos(y)) = sqrt(1 - y^2), y = dot(u, rvector2)
            const float y = ux * ra.w + uy * rb.x + uz * rb.y;
            rdon[p] = rd * sqrtf(fmaxf(0.f, 1.f - y * y));
          }
        }
      }
    }
#pragma unroll
    for (int k = 0; k < kA2Slots; k++) {
      if (!((slots >> k) & 1u)) continue;   // uniform
      const int kind = P.slotKind[k];
#pragma unroll
      for (int p = 0; p < 2; p++) {
        if (!w.in[p]) continue;
        const int iR = (int)(w.row[p] - kBiasBits);
        const float E = tab[k * kPlaneRows + iR];
        const float rsph = fminf(fmaxf(E * 0.01f, 0.f), 1.f);
        if (kind == A2_SLOT_ACC) {
          // Disordered donors take the "HD" type's row 1.1 A in.
          const float e = dis ? (P.planeH ? __ldg(P.planeH + k * kPlaneRows + max(0, iR - 110)) : 0.f) : E;
          s.mn[p][k] += e * hramp[p] * (racc[p] + (1.f - racc[p]) * rsph);
        } else {
          const float f = (kind == A2_SLOT_A1) ? racc[p] : rdon[p];
          const float val = E * (f + (1.f - f) * rsph);
          s.mn[p][k] = fminf(s.mn[p][k], val);
          s.mx[p][k] = fmaxf(s.mx[p][k], val);
          s.fl[p] |= 1u << k;
        }
      }
    }
  }
}

}  // namespace

static size_t aff2_smem(int nmPad, bool slots) {
  const size_t plain = tabOffset<PART_PLAIN>() + sizeof(float4) * (size_t)(kAffRows + 1) * row_stride(nmPad >> 2);
  return slots ? std::max(plain, tabOffset<PART_SLOTS>() + kSlotsRegion) : plain;
}

// The segments g0 .. g0 + kSegs of the cells around the box (each type of the
// part's order in turn, row by row: a row's cells are one run of the type-major
// list): S.segBeg / S.segPre.  Returns the round's atom count.
template <int PART>
__device__ __forceinline__ int segment_round(const Aff2Params& P, A2Smem<PART>& S, const unsigned char* order,
                                             const int nsegs, const int g0) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const Box& B = S.box;
  int cnt = 0;
  const int i = g0 + tid;
  if (i < nsegs) {
    const int pos = i / B.nrows, row = i - pos * B.nrows;
    const int ry = row % B.ncy, rz = row / B.ncy;
    const int key = (((int)order[pos] * P.ncell[2] + B.c0[2] + rz) * P.ncell[1] + B.c0[1] + ry) * P.ncell[0] + B.c0[0];
    const int beg = P.ctStart[key];
    cnt = P.ctStart[key + B.ncx] - beg;
    S.segBeg[tid] = beg;
  }
  int incl = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) S.cnt[warp] = incl;
  __syncthreads();
  int off = 0, total = 0;
#pragma unroll
  for (int w = 0; w < kW; w++) {
    if (w == warp) off = total;
    total += S.cnt[w];
  }
  S.segPre[tid + 1] = off + incl;
  if (tid == 0) S.segPre[0] = 0;
  __syncthreads();
  return total;
}

// Up to kT atoms v0 .. v0 + kT of the current round that lie within 8 A of the
// CTA box, appended to the candidate arrays at slot nb (d64: with their FP64
// records there, else with the fields of the part's sums).  Returns the new
// count.
template <int PART>
__device__ __forceinline__ int gather_chunk(const Aff2Params& P, A2Smem<PART>& S, const int g0, const int total,
                                            const int v0, const int nb, double4* d64) {
  const Box& B = S.box;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int v = v0 + tid;
  bool keep = false;
  int seg = 0;
  double4 a = make_double4(0, 0, 0, 0);
  float4 aux = make_float4(0.f, 0.f, 0.f, 0.f);
  if (v < total) {
    int hi_i = kSegs - 1;            // last segment with segPre <= v
    while (seg < hi_i) {
      const int mid = (seg + hi_i + 1) >> 1;
      if (S.segPre[mid] <= v) seg = mid; else hi_i = mid - 1;
    }
    const int j = S.segBeg[seg] + (v - S.segPre[seg]);
    a = P.ctXyz[j];
    aux = P.ctAux[j];                // vol, solq, info bits, atom index
    const double ddx = fmax(fmax(B.lo[0] - a.x, a.x - B.hi[0]), 0.0);
    const double ddy = fmax(fmax(B.lo[1] - a.y, a.y - B.hi[1]), 0.0);
    const double ddz = fmax(fmax(B.lo[2] - a.z, a.z - B.hi[2]), 0.0);
    keep = ddx * ddx + ddy * ddy + ddz * ddz <= 64.001;
  }
  const unsigned kbal = __ballot_sync(0xffffffffu, keep);
  if (lane == 0) S.cnt[warp] = __popc(kbal);
  __syncthreads();
  int tot = 0, off = 0;
#pragma unroll
  for (int w = 0; w < kW; w++) {
    if (w == warp) off = tot;
    tot += S.cnt[w];
  }
  if (keep) {
    const int j = nb + off + __popc(kbal & ((1u << lane) - 1u));
    const int atom = __float_as_int(aux.w);
    S.pos[j] = make_float4((float)(a.x - B.ox), (float)(a.y - B.oy), (float)(a.z - B.oz), aux.z);
    S.idx[j] = atom;
    if constexpr (PART == PART_PLAIN) {
      S.vs[j] = make_float2(aux.x, aux.y);
      atomicAdd(&S.typeCount[(g0 + seg) / B.nrows], 1);
    } else if (d64) {
      d64[j] = a;
    } else {
      const float4 va = __ldg(P.rv8 + 2 * (size_t)atom), vb = __ldg(P.rv8 + 2 * (size_t)atom + 1);
      S.rvA[j] = make_float4(va.x, va.y, va.z, vb.x);
      S.rvB[j] = make_float2(vb.y, vb.z);
      atomicAdd(&S.typeCount[(g0 + seg) / B.nrows], 1);
    }
  }
  __syncthreads();
  return nb + tot;
}

// The candidates of the part's `ntypes` types, in type-major order, in batches
// of at most kCap: batch(nb) takes each.  Returns false if batch does.
template <int PART, class Batch>
__device__ __forceinline__ bool gather_batches(const Aff2Params& P, A2Smem<PART>& S, const unsigned char* order,
                                               const int ntypes, double4* d64, const Batch& batch) {
  const int nsegs = ntypes * S.box.nrows;
  int g = -kSegs, v0 = 0, total = 0, nb = 0;
  for (;;) {
    bool last = false;
    for (;;) {
      if (v0 >= total) {
        g += kSegs;
        if (g >= nsegs) {
          last = true;
          break;
        }
        total = segment_round<PART>(P, S, order, nsegs, g);
        v0 = 0;
        continue;
      }
      if (nb + min(kT, total - v0) > A2Smem<PART>::kCap) break;  // a chunk keeps at most that many atoms
      nb = gather_chunk<PART>(P, S, g, total, v0, nb, d64);
      v0 += kT;
    }
    if (nb > 0 && !batch(nb)) return false;
    if (last) return true;
    nb = 0;
  }
}

// Nearest H donor of both points over candidates 0 .. nb (FP64 exact, ties to
// the lower file index), folded into best / bi.  A first FP32 pass finds each
// point's smallest r^2 in the batch; the FP64 distance (from the records in
// shared memory) is formed only for the candidates within 1e-3 A^2 of it,
// which the FP32 error (< 1e-4 A^2) cannot hide.
__device__ __forceinline__ void scan_donors(const Aff2Params& P, const A2Smem<PART_SLOTS>& S, const double4* d64,
                                            const int nb, double (&best)[2], int (&bi)[2], const Pts& q) {
  __syncthreads();
  float lim[2] = {3.0e38f, 3.0e38f};
  for (int j = 0; j < nb; j++) {
    const float4 a = S.pos[j];
    const float dx = a.x - q.px, dy = a.y - q.py;
    const float dxy = fmaf(dy, dy, dx * dx);
#pragma unroll
    for (int p = 0; p < 2; p++) {
      const float dz = a.z + (p ? q.npz.y : q.npz.x);
      lim[p] = fminf(lim[p], fmaf(dz, dz, dxy));
    }
  }
#pragma unroll
  for (int p = 0; p < 2; p++) lim[p] = fminf(lim[p], (float)best[p]) + 1.0e-3f;
  for (int j = 0; j < nb; j++) {
    const float4 a = S.pos[j];
    const float dx = a.x - q.px, dy = a.y - q.py;
    const float dxy = fmaf(dy, dy, dx * dx);
#pragma unroll
    for (int p = 0; p < 2; p++) {
      const float dz = a.z + (p ? q.npz.y : q.npz.x);
      if (fmaf(dz, dz, dxy) <= lim[p]) {
        const int id = S.idx[j];
        const double4 a64 = d64[j];
        const double r64 = rsq64(a64.x, a64.y, a64.z, gcoord(q.ix, P.n2x, P.h), gcoord(q.iy, P.n2y, P.h),
                                 gcoord(q.iz0 + p, P.n2z, P.h));
        if (r64 < best[p] || (r64 == best[p] && id < bi[p])) {
          best[p] = r64;
          bi[p] = id;
        }
      }
    }
  }
  __syncthreads();
}

// One batch of nb candidates: per-warp lists, then the part's ntypes types one
// by one.  load(pos) starts the copy of the table of the type at place `pos`
// of the part's order (one thread), and sums(pos, ...) takes the type's
// candidates [j0, j1) of the warp's list.  Returns false if a table copy's
// bounded wait expired (status set).
template <int PART, class Load, class Sums>
__device__ __forceinline__ bool process_batch(const Aff2Params& P, A2Smem<PART>& S, const int ntypes, const int nb,
                                              TableBar& tb, const Load& load, const Sums& sums) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  __syncthreads();  // candidate records and counts are complete
  if (tid == 0) {
    int s = 0;
    for (int t = 0; t < ntypes; t++) {
      S.typeStart[t] = s;
      s += S.typeCount[t];
      S.typeCount[t] = 0;
    }
    S.typeStart[ntypes] = s;
  }
  __syncthreads();
  // This warp's list: the candidates within 8 A of its sub-box (FP32 with margin).
  int nw = 0;
  const float* sblo = S.sblo[warp];
  const float* sbhi = S.sbhi[warp];
  if (sblo[0] <= sbhi[0])
    for (int base = 0; base < nb; base += 32) {
      const int j = base + lane;
      bool keep = false;
      if (j < nb) {
        const float4 a = S.pos[j];
        const float ddx = fmaxf(fmaxf(sblo[0] - a.x, a.x - sbhi[0]), 0.f);
        const float ddy = fmaxf(fmaxf(sblo[1] - a.y, a.y - sbhi[1]), 0.f);
        const float ddz = fmaxf(fmaxf(sblo[2] - a.z, a.z - sbhi[2]), 0.f);
        keep = fmaf(ddz, ddz, fmaf(ddy, ddy, ddx * ddx)) <= 64.01f;
      }
      const unsigned b = __ballot_sync(0xffffffffu, keep);
      if (keep) S.wlist[warp][nw + __popc(b & ((1u << lane) - 1u))] = (unsigned short)j;
      nw += __popc(b);
    }
  __syncwarp();
  for (int t = lane; t <= ntypes; t += 32) {  // first entry of each type (the list is sorted)
    const int target = S.typeStart[t];
    int a = 0, b = nw;
    while (a < b) {
      const int mid = (a + b) >> 1;
      if ((int)S.wlist[warp][mid] < target) a = mid + 1; else b = mid;
    }
    S.wStart[warp][t] = a;
  }
  __syncwarp();
  for (int t = 0; t < ntypes; t++) {
    if (S.typeStart[t + 1] == S.typeStart[t]) continue;  // uniform
    if (tid == 0) {
      fence_proxy_async();
      load(t);
    }
    const bool ok = mbar_wait_bounded(tb.bar, tb.phase & 1u, P.status);
    if (__syncthreads_or(!ok)) {
      if (tid == 0) mbar_wait_bounded(tb.bar, tb.phase & 1u, P.status);  // let the copy land before leaving
      return false;
    }
    tb.phase++;
    sums(t, S.wStart[warp][t], S.wStart[warp][t + 1], S.wlist[warp]);
    __syncthreads();  // the table buffer is free for the next type
  }
  return true;
}

// One work unit: a part of the CTA block `cta` of job P.  The two parts of a
// block run in either order or together: maps with an H-bond slot start at
// zero and both parts add to them (a sum of two terms, the same in any order).
// Returns false if a wait expired (status set; the barrier is not used again).
template <int NMAX, int PART>
__device__ __forceinline__ bool aff2_unit(const Aff2Params& P, const int cta, unsigned char* smem_raw, TableBar& tb) {
  A2Smem<PART>& S = *reinterpret_cast<A2Smem<PART>*>(smem_raw);
  float* tab = reinterpret_cast<float*>(smem_raw + tabOffset<PART>());
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int kCap = A2Smem<PART>::kCap;

  // This CTA's 8 x 8 x 8 points; this warp's 4 x 4 x 4 sub-box; this thread's two points.
  const int tbx = (P.nx + 7) / 8, tby = (P.ny + 7) / 8;
  const int x0 = (cta % tbx) * 8, y0 = ((cta / tbx) % tby) * 8, z0 = (cta / (tbx * tby)) * 8;
  const int wx = x0 + (warp & 1) * 4, wy = y0 + ((warp >> 1) & 1) * 4, wz = z0 + (warp >> 2) * 4;
  Pts q;
  q.ix = wx + (lane & 3);
  q.iy = wy + ((lane >> 2) & 3);
  q.iz0 = wz + (lane >> 4) * 2;
  const bool valid[2] = {q.ix < P.nx && q.iy < P.ny && q.iz0 < P.nz, q.ix < P.nx && q.iy < P.ny && q.iz0 + 1 < P.nz};
  {
    const double h = P.h;
    const double ox = gcoord(x0, P.n2x, h), oy = gcoord(y0, P.n2y, h), oz = gcoord(z0, P.n2z, h);
    q.px = (float)(gcoord(q.ix, P.n2x, h) - ox);
    q.py = (float)(gcoord(q.iy, P.n2y, h) - oy);
    q.npz.x = valid[0] ? -(float)(gcoord(q.iz0, P.n2z, h) - oz) : 1.0e4f;
    q.npz.y = valid[1] ? -(float)(gcoord(q.iz0 + 1, P.n2z, h) - oz) : 1.0e4f;
    // CTA box (FP64, grid-centred) and the cells within 8 A of it.
    if (tid == 0) {
      Box& B = S.box;
      B.ox = ox;
      B.oy = oy;
      B.oz = oz;
      B.lo[0] = ox; B.hi[0] = gcoord(min(x0 + 8, P.nx) - 1, P.n2x, h);
      B.lo[1] = oy; B.hi[1] = gcoord(min(y0 + 8, P.ny) - 1, P.n2y, h);
      B.lo[2] = oz; B.hi[2] = gcoord(min(z0 + 8, P.nz) - 1, P.n2z, h);
      int nc[3];
#pragma unroll
      for (int d = 0; d < 3; d++) {
        B.c0[d] = max(0, (int)floor((B.lo[d] - 8.0 - P.cellLo[d]) / P.cellEdge));
        nc[d] = min(P.ncell[d] - 1, (int)floor((B.hi[d] + 8.0 - P.cellLo[d]) / P.cellEdge)) - B.c0[d] + 1;
      }
      B.ncx = nc[0];
      B.ncy = nc[1];
      B.nrows = (nc[0] > 0 && nc[1] > 0 && nc[2] > 0) ? nc[1] * nc[2] : 0;
    }
    // This warp's sub-box in the CTA frame (empty when it lies past the grid edge).
    if (lane == 0) {
      const bool empty = wx >= P.nx || wy >= P.ny || wz >= P.nz;
      S.sblo[warp][0] = empty ? 1.f : (float)(gcoord(wx, P.n2x, h) - ox);
      S.sbhi[warp][0] = empty ? 0.f : (float)(gcoord(min(wx + 3, P.nx - 1), P.n2x, h) - ox);
      S.sblo[warp][1] = (float)(gcoord(wy, P.n2y, h) - oy);
      S.sbhi[warp][1] = (float)(gcoord(min(wy + 3, P.ny - 1), P.n2y, h) - oy);
      S.sblo[warp][2] = (float)(gcoord(wz, P.n2z, h) - oz);
      S.sbhi[warp][2] = (float)(gcoord(min(wz + 3, P.nz - 1), P.n2z, h) - oz);
    }
  }
  for (int t = tid; t < kMaxTypes; t += kT) S.typeCount[t] = 0;

  // Batches of candidates in type-major order, walked type by type.
  auto walk = [&](const unsigned char* order, const int ntypes, auto load, auto sums) AG_INLINE -> bool {
    return gather_batches<PART>(P, S, order, ntypes, nullptr, [&](int nb) AG_INLINE -> bool {
      return process_batch<PART>(P, S, ntypes, nb, tb, load, sums);
    });
  };

  if constexpr (PART == PART_PLAIN) {
    PlainSums<NMAX> s;
#pragma unroll
    for (int p = 0; p < 2; p++) {
      s.s1[p] = 0.f;
      s.s2[p] = 0.f;
#pragma unroll
      for (int g = 0; g < NMAX / 2; g++) s.em[p][g] = make_float2(0.f, 0.f);
    }
    __syncthreads();
    // The types come in two groups: first those whose equal columns are summed
    // once per class, then those that need every map's own column.
    bool classes = P.nClassTypes > 0;  // the sums are still per class
    const bool ok = walk(
        P.plainOrder, P.ntypes,
        [&](int pos) AG_INLINE {
          const int t = P.plainOrder[pos], pad = 4 * row_stride((pos < P.nClassTypes ? P.ncPad : P.nmPad) >> 2);
          const float* src = (pos < P.nClassTypes ? P.classTable : P.table) + (size_t)t * kAffRows * pad;
          const unsigned bytes = (unsigned)(kAffRows * pad * sizeof(float));
          mbar_arrive_expect_tx(tb.bar, bytes);
          tma_load_1d(tab, src, bytes, tb.bar);
          for (int i = 0; i < pad; i += 4)  // the zero row, read after the barrier that follows
            reinterpret_cast<float4*>(tab + kAffRows * pad + i)[0] = make_float4(0.f, 0.f, 0.f, 0.f);
        },
        [&](int pos, int j0, int j1, const unsigned short* wl) AG_INLINE {
          if (classes && pos >= P.nClassTypes) {
            expand_classes(P, s);
            classes = false;
          }
          const int rowQ = (classes ? P.ncPad : P.nmPad) >> 2;
          if (P.plainOrder[pos] == P.hydrogen) plain_sums<NMAX, true>(P, S, tab, rowQ, j0, j1, wl, q, s);
          else plain_sums<NMAX, false>(P, S, tab, rowQ, j0, j1, wl, q, s);
        });
    if (!ok) return false;
    if (classes) expand_classes(P, s);
#pragma unroll
    for (int p = 0; p < 2; p++) {
      if (!valid[p]) continue;
      const int64_t pt = ((int64_t)(q.iz0 + p) * P.ny + q.iy) * P.nx + q.ix;
#pragma unroll
      for (int g = 0; g < NMAX; g++) {
        if (g >= P.nmaps) break;
        if (P.mapCov[g]) continue;
        float* o = P.out + (int64_t)g * P.npoints + pt;
        const float e = ((g & 1) ? s.em[p][g >> 1].y : s.em[p][g >> 1].x) +
                        (P.solparProbe[g] * s.s1[p] + P.volProbe[g] * s.s2[p]);
        if ((P.slotMaps >> g) & 1u) atomicAdd(o, e);
        else *o = e;
      }
      P.dmap[pt] = P.solparQ * s.s1[p];
    }
  } else {
    SlotSums s;
#pragma unroll
    for (int p = 0; p < 2; p++) {
      s.fl[p] = 0u;
      s.ch[p] = -1;
#pragma unroll
      for (int k = 0; k < kA2Slots; k++) {
        s.mn[p][k] = (P.slotKind[k] == A2_SLOT_ACC) ? 0.f : 999999.f;
        s.mx[p][k] = -999999.f;
      }
    }
    __syncthreads();
    // The nearest H donor of both points, from the donors within 8 A of the box.
    if (P.needClosestH) {
      double4* d64 = reinterpret_cast<double4*>(tab);
      double best[2] = {1e300, 1e300};
      int bi[2] = {-1, -1};
      gather_batches<PART>(P, S, P.donorOrder, P.nDonorTypes, d64, [&](int nb) AG_INLINE -> bool {
        scan_donors(P, S, d64, nb, best, bi, q);
        return true;
      });
#pragma unroll
      for (int p = 0; p < 2; p++) {
        s.ch[p] = (best[p] <= 64.0) ? bi[p] : -1;
        S.rch[tid][p] = s.ch[p] >= 0 ? __ldg(P.rv8 + 2 * (size_t)s.ch[p]) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
      __syncthreads();
    }
    const bool ok = walk(
        P.slotOrder, P.nSlotTypes,
        [&](int pos) AG_INLINE {
          const unsigned bytes = (unsigned)(P.nslots * kPlaneRows * sizeof(float));
          mbar_arrive_expect_tx(tb.bar, bytes);
          tma_load_1d(tab, P.slotTable + (size_t)P.slotOrder[pos] * kA2Slots * kPlaneRows, bytes, tb.bar);
        },
        [&](int pos, int j0, int j1, const unsigned short* wl) AG_INLINE {
          const int t = P.slotOrder[pos];
          const unsigned slots = P.typeSlots[t];
          const bool ish = t == P.hydrogen;
          switch (P.typeAng[t]) {  // uniform
            case A2_D1:
              if (ish) slot_terms<A2_D1, true>(P, S, tab, j0, j1, wl, slots, q, s);
              else slot_terms<A2_D1, false>(P, S, tab, j0, j1, wl, slots, q, s);
              break;
            case A2_A1: slot_terms<A2_A1, false>(P, S, tab, j0, j1, wl, slots, q, s); break;
            case A2_A2: slot_terms<A2_A2, false>(P, S, tab, j0, j1, wl, slots, q, s); break;
            default:
              if (ish) slot_terms<A2_SPH, true>(P, S, tab, j0, j1, wl, slots, q, s);
              else slot_terms<A2_SPH, false>(P, S, tab, j0, j1, wl, slots, q, s);
              break;
          }
        });
    if (!ok) return false;
#pragma unroll
    for (int p = 0; p < 2; p++) {
      if (!valid[p]) continue;
      const int64_t pt = ((int64_t)(q.iz0 + p) * P.ny + q.iy) * P.nx + q.ix;
#pragma unroll
      for (int k = 0; k < kA2Slots; k++) {
        if (k >= P.nslots || !((P.slotMaps >> P.slotMap[k]) & 1u)) continue;
        float v = 0.f;
        if (P.slotKind[k] == A2_SLOT_ACC) v = s.mn[p][k];
        else if ((s.fl[p] >> k) & 1u) v = s.mn[p][k] + s.mx[p][k];
        atomicAdd(P.out + (int64_t)P.slotMap[k] * P.npoints + pt, v);
      }
    }
  }
  return true;
}

// CTAs per SM: three (80 registers, 76 KB of shared memory), so that the plain
// parts' table reads, which fill the shared-memory pipe, overlap the slot
// parts' arithmetic; rows of 16 columns (64 KB tables) leave room for two.
template <int NMAX>
constexpr int aff2_ctas_per_sm() {
  return NMAX <= 12 ? 3 : 2;
}

// A block's parts are neighbouring CTAs, so that both kinds share every SM.
template <int NMAX>
__global__ void __launch_bounds__(kT, aff2_ctas_per_sm<NMAX>()) affinity2_kernel(const __grid_constant__ Aff2Params P) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ uint64_t s_bar;
  TableBar tb;
  tb.init(&s_bar);
  if (P.slotMaps == 0u)
    aff2_unit<NMAX, PART_PLAIN>(P, P.ctaBase + blockIdx.x, smem_raw, tb);
  else if (blockIdx.x & 1)
    aff2_unit<NMAX, PART_PLAIN>(P, P.ctaBase + (blockIdx.x >> 1), smem_raw, tb);
  else
    aff2_unit<NMAX, PART_SLOTS>(P, P.ctaBase + (blockIdx.x >> 1), smem_raw, tb);
}

// Persistent kernel over the work units (job, CTA block) of a batch of
// receptors, taken part by part from an atomic counter in the host's
// (decreasing cost) order.
template <int NMAX>
__global__ void __launch_bounds__(kT, aff2_ctas_per_sm<NMAX>())
    affinity2_batch_kernel(const Aff2Params* __restrict__ jobs, const int2* __restrict__ units, int nunits,
                           int* counter) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ int s_unit;
  __shared__ uint64_t s_bar;
  TableBar tb;
  tb.init(&s_bar);
  for (;;) {
    __syncthreads();  // the previous unit is finished by every thread
    if (threadIdx.x == 0) s_unit = atomicAdd(counter, 1);
    __syncthreads();
    const int u = s_unit;
    if (u >= 2 * nunits) return;
    const int2 w = units[u >> 1];
    bool ok = true;
    if (u & 1) {
      ok = aff2_unit<NMAX, PART_PLAIN>(jobs[w.x], w.y, smem_raw, tb);
    } else if (jobs[w.x].slotMaps != 0u) {
      ok = aff2_unit<NMAX, PART_SLOTS>(jobs[w.x], w.y, smem_raw, tb);
    }
    if (!ok) return;  // uniform
  }
}

// Zero the values [off, off + cnt) of a pass's slot maps (blockIdx.y: slot).
__device__ __forceinline__ void zero_slot(const Aff2Params& P, int64_t off, int64_t cnt) {
  const int k = blockIdx.y;
  if (k >= P.nslots || !((P.slotMaps >> P.slotMap[k]) & 1u)) return;
  float* o = P.out + (int64_t)P.slotMap[k] * P.npoints + off;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < cnt; i += (int64_t)gridDim.x * blockDim.x)
    o[i] = 0.f;
}
__global__ void aff2_zero_kernel(const __grid_constant__ Aff2Params P, int64_t off, int64_t cnt) {
  zero_slot(P, off, cnt);
}
__global__ void aff2_zero_batch_kernel(const Aff2Params* __restrict__ jobs) {
  const Aff2Params& P = jobs[blockIdx.z];
  zero_slot(P, 0, P.npoints);
}

// The tables of one pass from the pair energies (one thread per type and row):
// the one-point kernel's rows, the two-point kernel's rows (slot maps' columns
// zero, the desolvation value last), its class rows and its slot planes.
__global__ void aff_tables_kernel(const __grid_constant__ AffTableJob J) {
  const int u = blockIdx.x * blockDim.x + threadIdx.x;
  if (u >= J.ntypes * kAffRows) return;
  const int t = u / kAffRows, i = u - t * kAffRows;
  const float* e = J.energy + (size_t)u * J.nmAll + J.m0;
  const float sol = J.sol[i];
  for (int g = 0; g < J.pad1; g++) J.rows1[(size_t)u * J.pad1 + g] = g < J.nm ? e[g] : 0.f;
  const int rowStride = 4 * row_stride(J.nmPad >> 2), classStride = 4 * row_stride(J.ncPad >> 2);
  for (int g = 0; g < J.nmPad; g++)
    J.rows[(size_t)u * rowStride + g] =
        g == J.nmPad - 1 ? sol : (g < J.nm && ((J.typePlain[t] >> g) & 1u)) ? e[g] : 0.f;
  for (int c = 0; c < J.ncPad; c++) {
    const int g = (int)(J.classMap >> (4 * c)) & 15;
    J.classRows[(size_t)u * classStride + c] =
        c == J.ncPad - 1 ? sol : (c < J.nc && ((J.typePlain[t] >> g) & 1u)) ? e[g] : 0.f;
  }
  for (int k = 0; k < J.nslots; k++) J.planes[((size_t)t * kA2Slots + k) * kA2PlaneRows + i] = e[J.slotMap[k]];
}

cudaError_t aff_tables_launch(const AffTableJob& J, cudaStream_t st) {
  aff_tables_kernel<<<(J.ntypes * kAffRows + 127) / 128, 128, 0, st>>>(J);
  return cudaGetLastError();
}

int aff2_row_stride(int columns) { return 4 * row_stride(columns >> 2); }

int aff2_ctas(int nx, int ny, int nz) { return ((nx + 7) / 8) * ((ny + 7) / 8) * ((nz + 7) / 8); }

cudaError_t aff2_batch_launch(const Aff2Params* jobs, int njobs, const int2* units, int nunits, int* counter,
                              int nmPadMax, bool anySlots, int sms, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(counter, 0, sizeof(int), st);
  if (e != cudaSuccess) return e;
  if (anySlots) aff2_zero_batch_kernel<<<dim3(16, kA2Slots, njobs), 256, 0, st>>>(jobs);
  const size_t smem = aff2_smem(nmPadMax, anySlots);
#define AG_AFF2B(N)                                                                                               \
  do {                                                                                                            \
    e = cudaFuncSetAttribute(affinity2_batch_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
    if (e != cudaSuccess) return e;                                                                               \
    affinity2_batch_kernel<N><<<sms * aff2_ctas_per_sm<N>(), kT, smem, st>>>(jobs, units, nunits, counter);       \
  } while (0)
  if (nmPadMax <= 4) AG_AFF2B(4);
  else if (nmPadMax <= 8) AG_AFF2B(8);
  else if (nmPadMax <= 12) AG_AFF2B(12);
  else AG_AFF2B(16);
#undef AG_AFF2B
  return cudaGetLastError();
}

cudaError_t aff2_launch_range(const Aff2Params& P0, int b0, int b1, cudaStream_t st) {
  const int tbxy = ((P0.nx + 7) / 8) * ((P0.ny + 7) / 8), nb = aff2_ctas(P0.nx, P0.ny, P0.nz);
  b0 = max(0, b0);
  b1 = min(nb, b1);
  if (b1 <= b0) return cudaSuccess;
  Aff2Params P = P0;
  P.ctaBase = b0;
  const bool slots = P.slotMaps != 0u;
  if (slots) {  // the z slabs that hold the range (a range is whole slabs)
    const int64_t plane = (int64_t)P.nx * P.ny;
    const int64_t z0 = 8LL * (b0 / tbxy), z1 = std::min<int64_t>(P.nz, 8LL * ((b1 + tbxy - 1) / tbxy));
    aff2_zero_kernel<<<dim3(74, kA2Slots), 256, 0, st>>>(P, z0 * plane, (z1 - z0) * plane);
  }
  const int grid = (b1 - b0) * (slots ? 2 : 1);
  const size_t smem = aff2_smem(P.nmPad, slots);
  cudaError_t e;
#define AG_AFF2(N)                                                                                           \
  do {                                                                                                       \
    e = cudaFuncSetAttribute(affinity2_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);  \
    if (e != cudaSuccess) return e;                                                                          \
    affinity2_kernel<N><<<grid, kT, smem, st>>>(P);                                                          \
  } while (0)
  if (P.nmPad <= 4) AG_AFF2(4);
  else if (P.nmPad <= 8) AG_AFF2(8);
  else if (P.nmPad <= 12) AG_AFF2(12);
  else AG_AFF2(16);
#undef AG_AFF2
  return cudaGetLastError();
}

cudaError_t aff2_launch(const Aff2Params& P, cudaStream_t st) { return aff2_launch_range(P, 0, 1 << 30, st); }

}  // namespace agk
