// Electrostatic map (e-map) by direct summation over all receptor atoms.
//
//   e(p) = sum_a w_a * min(1/r, 2) * invEps[min(int(100 r), 8191)]
//
// (FastGrid electrostatics/Cpu.cpp:27-88; the table is InputDataLoader.cpp:
// 715-742).  There is no cutoff, so the work is N_atoms x N_points pairs and
// the kernel is bound by the SM's instruction issue (one SFU rsqrt, one
// shared-memory table read and ~6 FP32/INT ops per pair), not by HBM.
//
// Layout and schedule
//  * Work item = NX consecutive x points of one (y, z) row; one thread per item,
//    256 items per CTA, items grouped by the host into compact boxes.
//  * Atoms stream through shared memory in tiles of kTile FP64 (x, y, z, w)
//    records, fetched with 1-D TMA bulk copies into a two-slot ring and
//    tracked by mbarriers (no multicast).
//  * Each tile is converted once per CTA to CTA-local coordinates scaled by
//    100 (so 100 r comes straight out of r^2 * rsqrt(r^2)) and split by the
//    atom's distance d to the CTA's box into three lists:
//      near (d < rNear): 1/r capped at 2, Kahan-compensated per pair, and the
//        bin decided exactly in FP64 (squared-distance threshold table) when
//        100 r lies within `delta` of a bin edge.  Decided again per warp:
//        a warp whose own points are all at least rNear away evaluates the
//        atom with the mid arithmetic (each term still compensated), and the
//        cap and the table clamp are dropped where they cannot apply;
//      mid (rNear <= d < rFar): bin by a round-down FMA, table read;
//      far (d >= rFar, at least 50 A): the table has saturated there (its
//        entries differ from entry 8191 by < 2e-6 relative), so the term is
//        w * invEps[8191] / r with no table read.
//    Mid atoms whose every bin lies in the table's saturating tail read a
//    packed copy of it instead: entry b is bits(g) + k_b, g = invEps[8191],
//    with k_b < 2^16 from about 22 A and < 2^8 from about 40 A.  Half- and
//    quarter-width entries put two or four neighbouring bins in one 32-bit
//    shared-memory word, so a warp's reads (its lanes' distances span ~1 A,
//    ~100 bins) touch fewer distinct words per bank: 2.0 and 1.5 wavefronts
//    per read instead of 2.6 (simulated), and those wavefronts are the
//    kernel's binding resource.  Decoding costs no instruction: k_b read as
//    float bits is the subnormal k_b 2^-149, and one packed FMA forms
//    100 w 2^-16 (g + k_b ulp(g)) = 100 w 2^-16 invEps[b] from it.
//    Mid and far terms are summed in plain FP32 over chunks of kChunk atoms
//    and the chunk sums are Kahan-compensated.
//  * Atoms at least R from the box (24 A; more for boxes wider than 5.6 A, and
//    up to 36 A for boxes beside the receptor: box_radii) do not enter point by
//    point: their sum is a smooth function over the box, so it is formed at
//    5 x 5 x 5 nodes of the box and interpolated to the box's 2,048 points in
//    FP64 at the end (node_atoms, node_row).
//  * When the grid is too small to fill the GPU, atoms are split across CTAs
//    and the per-CTA results are reduced in FP64, in a fixed order, by a
//    second kernel.
#include <cuda_runtime.h>

#include <cstdint>

#include "ag_device.cuh"
#include "ag_kernels.h"

namespace agk {

using namespace agd;

constexpr int kThreads = 256;
constexpr int kTile = 256;        // atoms per shared-memory tile
constexpr int kTabLen = 8192;     // invEps entries
constexpr int kChunk = 32;        // atoms per plain-FP32 chunk sum

// Atom classes of a tile, in their order in EmapSmem::list.
enum { kClsNode = 0, kClsNear = 1, kClsMid = 2, kClsMid16 = 3, kClsMid8 = 4, kClsFar = 5, kNumCls = 6 };

constexpr int kNodes1 = 5;                             // interpolation nodes per axis
constexpr int kNodes = kNodes1 * kNodes1 * kNodes1;    // per CTA box
constexpr int kNodeGroups = 4;                         // thread groups that share a tile's node atoms
constexpr int kNodeChunk = 16;                         // atom pairs per plain-FP32 node sum (32: up to 25 % more error)
// Atoms at least this far from the box (0.01 A, and half extents) need only
// 4 x 4 x 4 nodes and the saturated dielectric: 8.63 exp(-0.3154 r), the
// largest part of a term left out, is 1.4e-7 at 57 A, and interpolation from 4
// nodes errs by at most 1.2e-6 of a term (rms 4e-7) at 20 half extents, as from
// 5 nodes at about 8.5 (1.5e-6, rms 4e-7).  A quarter of the SFU operations per
// atom: 60,000 atoms on 255^3 points 59.3 -> 49.3 ms, 40,000 on 201^3 26.0 -> 23.5,
// 20,000 on 161^3 10.6 -> 10.4, and 2.15 ms either way for 8,000 on 125 x 97 x 83.
constexpr float kFarNodeRadius = 5700.f, kFarNodeHalfWidths = 20.f;
constexpr int kFarNodes1 = 4;
constexpr int kFarNodes = kFarNodes1 * kFarNodes1 * kFarNodes1;
static_assert(kFarNodes == 2 * 32, "a warp holds two far nodes per lane");
// Node radii of a box (box_radii): from the least one to three steps outwards.
constexpr int kRadiusSteps = 3;
constexpr float kRadiusStep = 1.f / 6.f;               // of the least radius: 24 to 28, 32 and 36 A
constexpr float kRadiusMargin = 3.f, kRadiusLean = 0.35f;
// Boxes per CTA of that kernel, which the atoms' reads from L2 bound: 22 us for 5,000
// atoms and 360 boxes, 130 for 20,000 and 2,541 (4 boxes: 6 us more for the first).
constexpr int kRadiusBoxes = 2;

struct EmapSmem {
  float tab[kTabLen];             // 32 KB
  double4 ring[2][kTile];         // 16 KB, TMA destination
  // Packed table tail; the last 4 KB hold the far nodes' sums (farAcc) where the
  // box's mid atoms do not read that far.
  __align__(16) unsigned char packed[kEmapPackedBytes];
  // This tile's atoms grouped by class: local scaled x, y, z and 100*w
  // (near, mid), 100*w*g*2^-16 (packed mid) or 100*w*g (far).  The node atoms
  // come first, two atoms in two entries: (x0, x1, y0, y1), (z0, z1, w0, w1);
  // far-node atoms, where the box has such, are the last class in the same form.
  float4 list[kTile + 4];
  float4 nodeAcc[kThreads];       // per thread: Kahan sum and compensation of its two nodes
  short nearIdx[kTile + 2];       // tile slot of each near atom (for FP64 lookups)
  // Near atom: bit w set if it lies within rNear of warp w's points, bit 8 + w
  // if within 0.51 A of them (the 1/r cap can apply).
  unsigned short nearMask[kTile + 2];
  float4 wlo[kThreads / 32], whi[kThreads / 32];  // each warp's box (local, scaled), widened by 0.01 A
  int cnt[kNumCls][kThreads / 32];
  double wpart[kThreads / 32];
  float rnode2, rfn2;             // squared radii of the box's node and far-node atoms
  int unit;                       // persistent batch kernel: the unit being processed
  uint64_t bar[2];
  uint64_t barIdle;               // never arrived on (target of the expiry test hook)

  // Per thread: Kahan sum and compensation of its two far nodes.
  __device__ __forceinline__ float4* farAcc() {
    return reinterpret_cast<float4*>(packed + kEmapPackedBytes) - kThreads;
  }
};
constexpr int kFarAccVecs = (kEmapPackedBytes - kThreads * (int)sizeof(float4)) / 16;  // tail vectors that leave room

__device__ __forceinline__ void unpack_item(int v, int& xc, int& y, int& z) {
  xc = v & 0xFF;
  y = (v >> 8) & 0x7FF;
  z = (v >> 19) & 0x7FF;
}

// Item k of a CTA's tile.  Warp-compact order: blocks of 4 rows x 4 planes over
// the tile's width, x fastest; otherwise rows, then planes.  Interleaved: the
// two items of a pair of x columns share its points alternately (a column
// whose partner is past the tile's end keeps its own).
__device__ __forceinline__ int tile_item(const EmapBlock& B, int k) {
  const int w = B.x1 - B.x0, H = B.y1 - B.y0, D = B.z1 - B.z0;
  const int by = B.tileMode >= 2 ? 4 : H, bz = B.tileMode >= 2 ? 4 : D;
  const int zb = k / (bz * w * H);
  k -= zb * bz * w * H;
  const int zn = min(bz, D - zb * bz), yb = k / (by * zn * w);
  k -= yb * by * zn * w;
  const int yn = min(by, H - yb * by), z = k / (yn * w);
  k -= z * yn * w;
  const int y = k / w, x = B.x0 + k - y * w;
  const bool il = B.tileMode == 3 && (B.x0 & 1) == 0 && (x ^ 1) < B.x1;
  return x | ((B.y0 + yb * by + y) << 8) | ((B.z0 + zb * bz + z) << 19) | (il ? kItemInterleaved : 0);
}

// Packed FP32 pairs: Blackwell issues one instruction for two lanes of FP32
// arithmetic (add/mul/fma .f32x2), each half rounded exactly as the scalar
// operation, so the pair loops below halve their FP32 instruction count
// without changing a bit of the result.  A thread's kNX points are held as
// the pairs (x0, x1), (x2, x3), ...
__device__ __forceinline__ float2 dup2(float v) { return make_float2(v, v); }

__device__ __forceinline__ float2 rsqrt2(float2 v) { return make_float2(rsqrt_approx(v.x), rsqrt_approx(v.y)); }

__device__ __forceinline__ float lo_hi(const float2& v, int k) { return (k & 1) ? v.y : v.x; }

// One Kahan step on a pair, (x - c), (s + y), ((s1 - s) - y) each rounded once
// as in the scalar form (a * -1 + b is exact before its single rounding).  The
// compensation is kept negated, n = -c, so that a product's step takes it as
// the addend of the product's own FMA.
__device__ __forceinline__ void kahan2_y(float2& s, float2& n, const float2 y) {
  const float2 m1 = dup2(-1.f);
  const float2 s1 = __fadd2_rn(s, y);
  n = __ffma2_rn(__ffma2_rn(s, m1, s1), m1, y);
  s = s1;
}
__device__ __forceinline__ void kahan2(float2& s, float2& n, const float2 x) { kahan2_y(s, n, __fadd2_rn(x, n)); }
__device__ __forceinline__ void kahan2_product(float2& s, float2& n, const float2 a, const float2 b) {
  kahan2_y(s, n, __ffma2_rn(a, b, n));
}

// Fold a chunk's plain FP32 sums into the running sums (Kahan), or, in plain
// mode, take them over (the chunk sums started from the running sums).
template <int MODE>
__device__ __forceinline__ void add_chunk(float2 (&sum)[kNX / 2], float2 (&cmp)[kNX / 2],
                                          const float2 (&cs)[kNX / 2]) {
#pragma unroll
  for (int k = 0; k < kNX / 2; k++) {
    if (MODE == kEmapKahan)
      kahan2(sum[k], cmp[k], cs[k]);
    else
      sum[k] = cs[k];
  }
}

// Table read at the bin encoded in the low bits of f = 2^23 + bin: the shared
// address is tabBiased + 4 * bits(f) in 32-bit shared-window arithmetic,
// where tabBiased = address(tab) - 4 * bits(2^23) (mod 2^32).
__device__ __forceinline__ float lds_bin(uint32_t tabBiased, float f) {
  const uint32_t a = tabBiased + ((uint32_t)__float_as_int(f) << 2);
  float v;
  asm("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
  return v;
}

// Mid-list atoms: bin by a round-down FMA, table read, plain FP32 chunk sums.
// CLAMP: the CTA's box is large enough that a bin can pass the table's end.
// gxn holds minus the thread's x coordinates, in pairs (x0, x1), (x2, x3), ...
template <int MODE, bool CLAMP>
__device__ __forceinline__ void mid_atoms(const float4* __restrict__ list, uint32_t tabBiased, int n,
                                          const float2 (&gxn)[kNX / 2], float gy, float gz, float2 (&sum)[kNX / 2],
                                          float2 (&cmp)[kNX / 2]) {
  const float kBias = 8388608.f;
  const float2 bias2 = dup2(kBias);
#pragma unroll 1
  for (int j0 = 0; j0 < n; j0 += kChunk) {
    float2 cs[kNX / 2];
#pragma unroll
    for (int k = 0; k < kNX / 2; k++)
      cs[k] = (MODE == kEmapKahan) ? make_float2(0.f, 0.f) : sum[k];
    const int j1 = min(n, j0 + kChunk);
    // Unrolled over atoms: the scheduler interleaves several atoms' rsqrt and
    // table-read latencies (3 CTAs x 8 warps per SM alone do not hide them).
#pragma unroll 8
    for (int j = j0; j < j1; j++) {
      const float4 a = list[j];
      const float dy = a.y - gy, dz = a.z - gz;
      const float2 dyz2 = dup2(fmaf(dz, dz, dy * dy));
      const float2 ax = dup2(a.x), aw = dup2(a.w);
#pragma unroll
      for (int k = 0; k < kNX / 2; k++) {
        const float2 dx = __fadd2_rn(ax, gxn[k]);
        const float2 r2 = __ffma2_rn(dx, dx, dyz2);
        const float2 rs = rsqrt2(r2);
        float2 f = __ffma2_rd(r2, rs, bias2);
        if (CLAMP) {
          f.x = fminf(f.x, kBias + (float)(kTabLen - 1));
          f.y = fminf(f.y, kBias + (float)(kTabLen - 1));
        }
        const float2 g = make_float2(lds_bin(tabBiased, f.x), lds_bin(tabBiased, f.y));
        cs[k] = __ffma2_rn(__fmul2_rn(aw, rs), g, cs[k]);
      }
    }
    add_chunk<MODE>(sum, cmp, cs);
  }
}

// Entry k_b of a packed tail table (W = 2: 16-bit, W = 1: 8-bit) at the bin
// encoded in f = 2^23 + bin, returned as float bits (the subnormal k_b 2^-149).
// tabBiased = address(entry 0) - W * (bits(2^23) + first bin), mod 2^32.
template <int W>
__device__ __forceinline__ float lds_packed(uint32_t tabBiased, float f) {
  uint32_t v;
  if (W == 2)
    asm("ld.shared.u16 %0, [%1];" : "=r"(v) : "r"(tabBiased + ((uint32_t)__float_as_int(f) << 1)));
  else
    asm("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(tabBiased + (uint32_t)__float_as_int(f)));
  return __uint_as_float(v);
}

// Mid atoms whose bins all lie in a packed tail table.  With a.w = 100 w g
// 2^-16 and kScale = 2^(e+126) / g (g = 2^e m), aws = a.w kScale = 100 w
// ulp(g) 2^133, so aws * k_b 2^-149 + a.w = 100 w 2^-16 (g + k_b ulp(g)):
// the term's weight times the table entry, scaled by 2^-16 (exact), in one
// FMA whose product is exact for 8-bit k_b and rounded once for 16-bit.  The
// chunk sums run in the same scale and are scaled back by 2^16 (exact).
template <int MODE, int W>
__device__ __forceinline__ void mid_packed_atoms(const float4* __restrict__ list, uint32_t tabBiased, int n,
                                                 const float2 (&gxn)[kNX / 2], float gy, float gz,
                                                 float2 (&sum)[kNX / 2], float2 (&cmp)[kNX / 2], float kScale) {
  const float2 bias2 = dup2(8388608.f);
  const float2 down = dup2(1.0f / 65536.f), up = dup2(65536.f);
#pragma unroll 1
  for (int j0 = 0; j0 < n; j0 += kChunk) {
    float2 cs[kNX / 2];
#pragma unroll
    for (int k = 0; k < kNX / 2; k++)
      cs[k] = (MODE == kEmapKahan) ? make_float2(0.f, 0.f) : __fmul2_rn(sum[k], down);
    const int j1 = min(n, j0 + kChunk);
#pragma unroll 8
    for (int j = j0; j < j1; j++) {
      const float4 a = list[j];
      const float dy = a.y - gy, dz = a.z - gz;
      const float2 dyz2 = dup2(fmaf(dz, dz, dy * dy));
      const float2 ax = dup2(a.x), awg = dup2(a.w), aws = dup2(a.w * kScale);
#pragma unroll
      for (int k = 0; k < kNX / 2; k++) {
        const float2 dx = __fadd2_rn(ax, gxn[k]);
        const float2 r2 = __ffma2_rn(dx, dx, dyz2);
        const float2 rs = rsqrt2(r2);
        const float2 f = __ffma2_rd(r2, rs, bias2);
        const float2 kb = make_float2(lds_packed<W>(tabBiased, f.x), lds_packed<W>(tabBiased, f.y));
        cs[k] = __ffma2_rn(rs, __ffma2_rn(aws, kb, awg), cs[k]);
      }
    }
#pragma unroll
    for (int k = 0; k < kNX / 2; k++) cs[k] = __fmul2_rn(cs[k], up);
    add_chunk<MODE>(sum, cmp, cs);
  }
}

// Node k of an axis with half extent h (0.01 A): the Chebyshev node
// cos((2 k + 1) pi / 10) h, moved to a multiple of 0.5.  An atom's offset from
// it is then exact in FP32, as it is from a grid point; at the Chebyshev nodes
// themselves its rounding added up to 13 % to a map's error.
__device__ __forceinline__ float node_pos(int k, float h) {
  const float v = (k == 0 || k == 4) ? 0.95105652f : (k == 2 ? 0.f : 0.58778525f);
  const float x = 0.5f * rintf(2.f * v * h);
  return k > 2 ? -x : x;
}

// An axis' five nodes p, q, 0, -q, -p and what their Lagrange weights share.
// In FP64, as everything from the node sums on: a box's field is the small
// difference of large terms, and FP32 weights and products left 3e-7 of it.
struct NodeAxis {
  double p, q, a, b, c;
  __device__ __forceinline__ void set(float h) {
    p = (double)node_pos(0, h);
    q = (double)node_pos(1, h);
    const double p2 = p * p, q2 = q * q;
    a = 0.5 / (p2 * (p2 - q2));
    b = 0.5 / (q2 * (q2 - p2));
    c = 1.0 / (p2 * q2);
  }
  __device__ __forceinline__ void weights(double t, double (&w)[kNodes1]) const {
    const double tp = t * t - p * p, tq = t * t - q * q, u = t * tq * a, v = t * tp * b;
    w[0] = u * (t + p);
    w[1] = v * (t + q);
    w[2] = tp * tq * c;
    w[3] = v * (t - q);
    w[4] = u * (t - p);
  }
};

// Add a thread's sums over a tile (a pair's two atoms apart) at its two nodes to
// the running ones, each part compensated.
__device__ __forceinline__ void kahan(float& s, float& c, float x) {
  const float y = x - c, t = s + y;
  c = (t - s) - y;
  s = t;
}
__device__ __forceinline__ void add_nodes(float4& acc, const float2 s0, const float2 s1) {
  float4 a = acc;
  kahan(a.x, a.y, s0.x);
  kahan(a.x, a.y, s0.y);
  kahan(a.z, a.w, s1.x);
  kahan(a.z, a.w, s1.y);
  acc = a;
}

// Sum of a tile's node atoms at this thread's two nodes of the box (half
// extents hx, hy, hz).  64 threads cover the nodes, and the kNodeGroups groups
// of 64 take the atom pairs in turn; packed FP32 over the two atoms of a pair,
// whose record keeps equal components side by side (no register moves).  The
// kernel is the dielectric's smooth form, 332 / eps = g (1 + E (c1 + c2 E)),
// E = exp(-lambda (r - 0.005)) (half a bin in: the left-edge bins are met on
// average); the next term of the series is below 1e-9 from 24 A on.  (A
// polynomial in 1 / r in place of ex2, seven more FMAs for half the SFU work,
// was slower: 67.7 against 63.6 ms for 60,000 atoms on 255^3 points.)
template <bool DDD>
__device__ __forceinline__ void node_atoms(EmapSmem& S, const int npairs, const float hx, const float hy,
                                           const float hz) {
  const int q = threadIdx.x & 63, grp = threadIdx.x >> 6;
  float2 nx[2], ny[2], nz[2], s[2];
#pragma unroll
  for (int u = 0; u < 2; u++) {
    const int n = min(2 * q + u, kNodes - 1);
    nx[u] = dup2(-node_pos(n % kNodes1, hx));
    ny[u] = dup2(-node_pos((n / kNodes1) % kNodes1, hy));
    nz[u] = dup2(-node_pos(n / (kNodes1 * kNodes1), hz));
  }
  const float2 nl = dup2(-4.5499247e-3f);    // -lambda / (100 ln 2), lambda = 0.3153767175 per A
  const float2 sh = dup2(2.2749621e-3f);     // 0.005 lambda / ln 2
  const float2 c1 = dup2(8.6330307f);        // a + c, a = 7.7839, c = 66.57180475 / 78.4
  const float2 c2 = dup2(7.3305663f);        // c (a + c)
  const float2 one = dup2(1.f);
#pragma unroll 1
  for (int p0 = grp; p0 < npairs; p0 += kNodeGroups * kNodeChunk) {
    s[0] = s[1] = make_float2(0.f, 0.f);
    const int p1 = min(npairs, p0 + kNodeGroups * kNodeChunk);
#pragma unroll 4
    for (int p = p0; p < p1; p += kNodeGroups) {
      const float4 xy = S.list[2 * p], zw = S.list[2 * p + 1];
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const float2 dx = __fadd2_rn(make_float2(xy.x, xy.y), nx[u]);
        const float2 dy = __fadd2_rn(make_float2(xy.z, xy.w), ny[u]);
        const float2 dz = __fadd2_rn(make_float2(zw.x, zw.y), nz[u]);
        const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
        const float2 rs = rsqrt2(r2), w = make_float2(zw.z, zw.w);
        if (DDD) {
          const float2 arg = __ffma2_rn(__fmul2_rn(r2, rs), nl, sh);
          const float2 E = make_float2(ex2_approx(arg.x), ex2_approx(arg.y));
          s[u] = __ffma2_rn(__fmul2_rn(w, rs), __ffma2_rn(E, __ffma2_rn(E, c2, c1), one), s[u]);
          continue;
        }
        s[u] = __ffma2_rn(w, rs, s[u]);
      }
    }
    add_nodes(S.nodeAcc[threadIdx.x], s[0], s[1]);
  }
}

// Far node k: cos((2 k + 1) pi / 8) h, moved likewise.
__device__ __forceinline__ float far_pos(int k, float h) {
  const float v = (k == 0 || k == 3) ? 0.92387953f : 0.38268343f;
  const float x = 0.5f * rintf(2.f * v * h);
  return k > 1 ? -x : x;
}

// Lagrange weights of an axis' four far nodes p, q, -q, -p at t.
__device__ __forceinline__ void far_weights(double t, float h, double (&w)[kFarNodes1]) {
  const double p = (double)far_pos(0, h), q = (double)far_pos(1, h), d = p * p - q * q;
  const double u = (t * t - q * q) / (2.0 * p * d), v = (p * p - t * t) / (2.0 * q * d);
  w[0] = u * (t + p);
  w[1] = v * (t + q);
  w[2] = v * (q - t);
  w[3] = u * (p - t);
}

// Sum of a tile's far-node atoms (pairs from list) at this lane's two far
// nodes, neighbours along x, so one dy and dz serve both; the warps take the
// pairs in turn.  Saturated dielectric: one rsqrt per term.
__device__ __forceinline__ void far_node_atoms(EmapSmem& S, const float4* list, const int npairs, const float hx,
                                               const float hy, const float hz) {
  int n = 2 * (threadIdx.x & 31);
  asm volatile("" : "+r"(n));  // keeps the node positions out of the caller's loops
  const float2 nx0 = dup2(-far_pos(n & 3, hx)), nx1 = dup2(-far_pos((n & 3) + 1, hx));
  const float2 ny = dup2(-far_pos((n >> 2) & 3, hy)), nz = dup2(-far_pos(n >> 4, hz));
  float2 s0 = make_float2(0.f, 0.f), s1 = s0;
#pragma unroll 4
  for (int p = threadIdx.x >> 5; p < npairs; p += kThreads / 32) {
    const float4 xy = list[2 * p], zw = list[2 * p + 1];
    const float2 dy = __fadd2_rn(make_float2(xy.z, xy.w), ny), dz = __fadd2_rn(make_float2(zw.x, zw.y), nz);
    const float2 yz = __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)), w = make_float2(zw.z, zw.w);
    const float2 x0 = __fadd2_rn(make_float2(xy.x, xy.y), nx0), x1 = __fadd2_rn(make_float2(xy.x, xy.y), nx1);
    s0 = __ffma2_rn(w, rsqrt2(__ffma2_rn(x0, x0, yz)), s0);
    s1 = __ffma2_rn(w, rsqrt2(__ffma2_rn(x1, x1, yz)), s1);
  }
  add_nodes(S.farAcc()[threadIdx.x], s0, s1);
}

// The far nodes' field (sums F4, x fastest) at near node n: exact, a cubic's
// values at the five nodes per axis stand for the cubic itself.
__device__ __forceinline__ double far_field(const double* F4, int n, float hx, float hy, float hz) {
  double wx[kFarNodes1], wy[kFarNodes1], wz[kFarNodes1];
  far_weights((double)node_pos(n % kNodes1, hx), hx, wx);
  far_weights((double)node_pos((n / kNodes1) % kNodes1, hy), hy, wy);
  far_weights((double)node_pos(n / (kNodes1 * kNodes1), hz), hz, wz);
  double f = 0.0;
#pragma unroll
  for (int k = 0; k < kFarNodes1 * kFarNodes1; k++) {
    const double* r = F4 + kFarNodes1 * k;
    f += wz[k >> 2] * wy[k & 3] * (wx[0] * r[0] + wx[1] * r[1] + wx[2] * r[2] + wx[3] * r[3]);
  }
  return f;
}

// The node atoms' field along this thread's row, at the five x nodes, from the
// node sums F (x fastest).
__device__ __forceinline__ void node_row(const double* F, const NodeAxis& ay, const NodeAxis& az, float gy, float gz,
                                         double (&c)[kNodes1]) {
  double wy[kNodes1], wz[kNodes1];
  ay.weights((double)gy, wy);
  az.weights((double)gz, wz);
#pragma unroll
  for (int kz = 0; kz < kNodes1; kz++)
#pragma unroll
    for (int ky = 0; ky < kNodes1; ky++) {
      const double w = wz[kz] * wy[ky];
#pragma unroll
      for (int kx = 0; kx < kNodes1; kx++) c[kx] = fma(w, F[(kz * kNodes1 + ky) * kNodes1 + kx], c[kx]);
    }
}

// One near atom against this thread's points, bins decided exactly near an
// edge.  GUARD: cap 1/r at 2 and clamp the bin at the table's end; without it
// the caller has shown that no point of the warp lies within 0.51 A of the
// atom and that no bin can pass the table's end (the CTA box is small enough),
// so neither would change a value.
template <bool DDD, int MODE, bool GUARD>
__device__ __forceinline__ void near_exact(const EmapSmem& S, const EmapParams& P, const int slot, const int j,
                                           const float2 dyz2, const float2 ax, const float2 aw,
                                           const float2 (&gxn)[kNX / 2], const int iy, const int iz, const int xb,
                                           const int xs, float2 (&sum)[kNX / 2], float2 (&cmp)[kNX / 2]) {
  const float cap = 0.02f;        // min(1/r, 2) in units of 1/(100 r)
  const float kBias = 8388608.f;  // 2^23
  const double h = P.h;
  float2 rsv[kNX / 2];
  float2 kn[kNX / 2];   // 2^23 + the integer nearest 100 r
  float2 d[kNX / 2];    // 100 r minus that integer
  uint32_t bits[kNX];   // 2^23 + bin, as float bits
#pragma unroll
  for (int k = 0; k < kNX / 2; k++) {
    const float2 dx = __fadd2_rn(ax, gxn[k]);
    const float2 r2 = __ffma2_rn(dx, dx, dyz2);
    rsv[k] = rsqrt2(r2);
    if (DDD) {
      float2 f = __ffma2_rd(r2, rsv[k], dup2(kBias));
      if (GUARD) {
        f.x = fminf(f.x, kBias + (float)(kTabLen - 1));
        f.y = fminf(f.y, kBias + (float)(kTabLen - 1));
      }
      bits[2 * k] = __float_as_uint(f.x);
      bits[2 * k + 1] = __float_as_uint(f.y);
      kn[k] = __ffma2_rn(r2, rsv[k], dup2(kBias));
      d[k] = __ffma2_rn(r2, rsv[k], __ffma2_rn(kn[k], dup2(-1.f), dup2(kBias)));
    }
  }
  // Within delta of a bin edge <=> 100 r is within delta of an integer.
  bool any = false;
  if (DDD) {
    static_assert(kNX == 8, "eight points");
    const float m = min3_abs(min3_abs(d[0].x, d[0].y, d[1].x), min3_abs(d[1].y, d[2].x, d[2].y),
                             fminf(fabsf(d[3].x), fabsf(d[3].y)));
    any = m < P.delta;
  }
  if (DDD && __any_sync(0xffffffffu, any)) {
    if (any) {
      const double4 a64 = S.ring[slot][S.nearIdx[j]];
      const double gy64 = __dmul_rn((double)(iy - P.n2y), h), gz64 = __dmul_rn((double)(iz - P.n2z), h);
      const double ddz = __dsub_rn(a64.z, gz64), ddy = __dsub_rn(a64.y, gy64);
      const double dydz = __dadd_rn(__dmul_rn(ddy, ddy), __dmul_rn(ddz, ddz));
#pragma unroll
      for (int k = 0; k < kNX; k++) {
        if (fabsf(lo_hi(d[k >> 1], k)) < P.delta) {
          // The reference's bin is kmid - 1 or kmid, kmid the integer nearest 100 r.
          const int kmid = min(__float_as_int(lo_hi(kn[k >> 1], k)) - 0x4B000000, kTabLen - 1);
          const double gx64 = __dmul_rn((double)(xb + k * xs - P.n2x), h);
          const double ddx = __dsub_rn(a64.x, gx64);
          const double r2d = __dadd_rn(__dmul_rn(ddx, ddx), dydz);
          const int b = (kmid == 0) ? 0 : ((r2d >= P.thr[kmid]) ? kmid : kmid - 1);
          bits[k] = 0x4B000000u + (uint32_t)b;
        }
      }
    }
  }
  const uint32_t tabB = smem_u32(S.tab) - 0x2C000000u;  // address(tab) - 4 * bits(2^23)
#pragma unroll
  for (int k = 0; k < kNX / 2; k++) {
    const float2 rc = GUARD ? make_float2(fminf(rsv[k].x, cap), fminf(rsv[k].y, cap)) : rsv[k];
    float2 wr = aw, t = rc;  // the term is wr * t
    if (DDD) {
      wr = __fmul2_rn(aw, rc);
      asm("ld.shared.f32 %0, [%1];" : "=f"(t.x) : "r"(tabB + (bits[2 * k] << 2)));
      asm("ld.shared.f32 %0, [%1];" : "=f"(t.y) : "r"(tabB + (bits[2 * k + 1] << 2)));
    }
    if (MODE == kEmapKahan)
      kahan2_product(sum[k], cmp[k], wr, t);
    else
      sum[k] = __fadd2_rn(sum[k], __fmul2_rn(wr, t));
  }
}

constexpr int kAxisAt = (8 * (kNodes + kFarNodes) + (int)sizeof(NodeAxis) - 1) / (int)sizeof(NodeAxis);
static_assert((kAxisAt + 3) * sizeof(NodeAxis) <= sizeof(EmapSmem::list), "epilogue");

// One work unit: CTA box `blk` of job P against atom split `split`.  Called
// once per CTA by emap_kernel, and repeatedly by the persistent batch kernel.
// NODES: far atoms are summed at the box's nodes (else rnodeMin is infinite).
template <bool DDD, int MODE, bool NODES>
__device__ __forceinline__ void emap_unit(const EmapParams& P, const int blk, const int split, EmapSmem& S) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const EmapBlock B = P.blocks[blk];
  const int a0 = split * P.chunk;
  const int a1 = min(P.n_atoms, a0 + P.chunk);
  const int ntiles = (a1 - a0 + kTile - 1) / kTile;

  // This thread's points, in the CTA-local frame scaled by 100.
  const bool active = tid < B.nitems;
  const bool busy = warp * 32 < B.nitems;  // a warp without items only helps with the atom handling and the nodes
  int xc = 0, iy = 0, iz = 0;
  const int item = B.tileMode ? tile_item(B, active ? tid : 0) : P.items[B.item0 + (active ? tid : 0)];
  unpack_item(item, xc, iy, iz);
  // x of point k = xb + k * xs: NX consecutive points, or every other point of
  // the 2 NX points of an interleaved column pair.
  const bool il = (item & kItemInterleaved) != 0;
  const int xb = il ? (xc >> 1) * (2 * kNX) + (xc & 1) : xc * kNX;
  const int xs = il ? 2 : 1;
  // A point past the grid's end stands on the last one (and is not written): the
  // box holds every point that is evaluated, on which the table reads' clamps rely.
  const double h = P.h;
  float gx[kNX];
#pragma unroll
  for (int k = 0; k < kNX; k++)
    gx[k] = (float)(((double)(min(xb + k * xs, P.nx - 1) - P.n2x) * h - B.ox) * 100.0);
  const float gy = (float)(((double)(iy - P.n2y) * h - B.oy) * 100.0);
  const float gz = (float)(((double)(iz - P.n2z) * h - B.oz) * 100.0);
  float2 gxn[kNX / 2];
#pragma unroll
  for (int k = 0; k < kNX / 2; k++) gxn[k] = make_float2(-gx[2 * k], -gx[2 * k + 1]);

  // Atoms this far (0.01 A) from the box are summed at its nodes, and at its far nodes.
  const float2 radius = NODES && DDD && P.radius ? P.radius[blk] : make_float2(0.f, 0.f);
  const float rnode = !NODES ? __int_as_float(0x7F800000)
                      : DDD && P.radius ? radius.x : fmaxf(P.rnodeHalfWidths * B.rnode, P.rnodeMin);
  const bool clampMid = B.clampMid;  // mid-list bins may pass the table's end
  // No mid atom is this far from a point of the box.
  const float midEndR = rnode + 2.f * sqrtf(B.hx * B.hx + B.hy * B.hy + B.hz * B.hz);
  int nodeSeen = 0;  // uniform; bit 0: node atoms, bit 1: far-node atoms
  // The part of the packed tail that this box's mid atoms read: 16-bit entries
  // up to the farthest bin only, if the node atoms begin before the 8-bit ones.
  const int tailVecs = NODES && DDD && midEndR < 8100.f && rnode * rnode <= P.r8sq
                           ? min(P.packedVecs, max(0, (int)midEndR + 3 - P.b16) / 8 + 1)
                           : P.packedVecs;
  // Far nodes: where the node atoms begin before the saturated point sums, so
  // that kClsFar holds far-node atoms or none (else kClsFar is summed at the points).
  const bool farNodes = NODES && DDD && P.radius && rnode * rnode <= B.rfar2 && tailVecs <= kFarAccVecs;
  if (NODES) {
    if (tid == 0) {
      S.rnode2 = rnode * rnode;
      S.rfn2 = farNodes ? radius.y * radius.y : __int_as_float(0x7F800000);
    }
    S.nodeAcc[tid] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (farNodes) S.farAcc()[tid] = make_float4(0.f, 0.f, 0.f, 0.f);
  }

  // Packed tail tables for this box: only when no bin can pass the table's end.
  const bool pk = DDD && P.packed != nullptr && !clampMid;
  if (DDD) {
    const float4* src = reinterpret_cast<const float4*>(P.table);
    float4* dst = reinterpret_cast<float4*>(S.tab);
    for (int i = tid; i < kTabLen / 4; i += kThreads) dst[i] = src[i];
    if (pk) {
      uint4* pdst = reinterpret_cast<uint4*>(S.packed);
      for (int i = tid; i < tailVecs; i += kThreads) pdst[i] = P.packed[i];
    }
  }
  // This warp's box: the extent of its active lanes' points (an empty box,
  // lo > hi, when no lane has an item), widened by 1 (0.01 A).
  {
    float lo[3] = {3.0e38f, 3.0e38f, 3.0e38f}, hi[3] = {-3.0e38f, -3.0e38f, -3.0e38f};
    if (active) {
      lo[0] = fminf(gx[0], gx[kNX - 1]);
      hi[0] = fmaxf(gx[0], gx[kNX - 1]);
      lo[1] = hi[1] = gy;
      lo[2] = hi[2] = gz;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int d = 0; d < 3; d++) {
        lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
        hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
      }
    if (lane == 0) {
      S.wlo[warp] = make_float4(lo[0] - 1.f, lo[1] - 1.f, lo[2] - 1.f, 0.f);
      S.whi[warp] = make_float4(hi[0] + 1.f, hi[1] + 1.f, hi[2] + 1.f, 0.f);
    }
  }
  if (tid == 0) {
    mbar_init(&S.bar[0], 1);
    mbar_init(&S.bar[1], 1);
    mbar_init(&S.barIdle, 1);
    fence_barrier_init();
  }
  __syncthreads();
  const float gFar = DDD ? S.tab[kTabLen - 1] : 1.f;
  if (tid == 0 && ntiles > 0) {
    unsigned n0 = (unsigned)min(kTile, a1 - a0);
    mbar_arrive_expect_tx(&S.bar[0], n0 * 32u);
    tma_load_1d(S.ring[0], P.atoms + a0, n0 * 32u, &S.bar[0]);
  }

  float2 sum[kNX / 2], cmp[kNX / 2];
  double wsum = 0.0;  // FP64 sum of the weights this thread converted (checksum)
#pragma unroll
  for (int k = 0; k < kNX / 2; k++) { sum[k] = make_float2(0.f, 0.f); cmp[k] = make_float2(0.f, 0.f); }

  const float kBias = 8388608.f;  // 2^23: adding it with round-down leaves floor() in the low bits

  for (int t = 0; t < ntiles; t++) {
    const int slot = t & 1;
    const int t0 = a0 + t * kTile;
    const int nt = min(kTile, a1 - t0);
    if (tid == 0 && t + 1 < ntiles) {
      // The other slot was released by the __syncthreads() that ended tile t-1.
      const int t1 = t0 + kTile;
      unsigned n1 = (unsigned)min(kTile, a1 - t1);
      fence_proxy_async();
      mbar_arrive_expect_tx(&S.bar[slot ^ 1], n1 * 32u);
      tma_load_1d(S.ring[slot ^ 1], P.atoms + t1, n1 * 32u, &S.bar[slot ^ 1]);
    }
    bool ok = mbar_wait_bounded(&S.bar[slot], (unsigned)(t >> 1) & 1u, P.status);
    // Test hook: after the first tile has landed, wait a few polls on a
    // barrier that nothing arrives on; the wait expires like a lost copy would.
    if (P.testIdleWait > 0 && t == 0) ok = mbar_wait_limit(&S.barIdle, 0u, P.status, P.testIdleWait) && ok;
    if (__syncthreads_or(!ok)) {
      // Give the copies still in flight (this tile's and the prefetched next
      // one) a bounded chance to land before shared memory is released.
      if (tid == 0) {
        mbar_wait_bounded(&S.bar[slot], (unsigned)(t >> 1) & 1u, P.status);
        if (t + 1 < ntiles) mbar_wait_bounded(&S.bar[slot ^ 1], (unsigned)((t + 1) >> 1) & 1u, P.status);
      }
      return;
    }

    // Classify and convert this tile's atoms (one atom per thread).
    int cls = -1;
    unsigned nearBits = 0xFFFFu;
    float4 loc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (tid < nt) {
      double4 a = S.ring[slot][tid];
      wsum += a.w;
      loc.x = (float)((a.x - B.ox) * 100.0);
      loc.y = (float)((a.y - B.oy) * 100.0);
      loc.z = (float)((a.z - B.oz) * 100.0);
      loc.w = (float)(a.w * 100.0);
      const float dx = fmaxf(fabsf(loc.x) - B.hx, 0.f), dy = fmaxf(fabsf(loc.y) - B.hy, 0.f),
                  dz = fmaxf(fabsf(loc.z) - B.hz, 0.f);
      const float d2 = dx * dx + dy * dy + dz * dz;
      if (NODES && d2 >= S.rnode2) {
        cls = DDD && d2 >= S.rfn2 ? kClsFar : kClsNode;
        loc.w *= gFar;
      } else if (d2 < P.rnear2) {
        cls = kClsNear;
        // The warps whose own points it is near: the others evaluate it as a mid atom.
        unsigned m = 0;
#pragma unroll
        for (int w = 0; w < kThreads / 32; w++) {
          const float4 wl = S.wlo[w], wh = S.whi[w];
          const float ex = fmaxf(fmaxf(wl.x - loc.x, loc.x - wh.x), 0.f);
          const float ey = fmaxf(fmaxf(wl.y - loc.y, loc.y - wh.y), 0.f);
          const float ez = fmaxf(fmaxf(wl.z - loc.z, loc.z - wh.z), 0.f);
          const float e2 = ex * ex + ey * ey + ez * ez;
          m |= ((e2 < P.rnear2 ? 1u : 0u) << w) | ((e2 < 51.f * 51.f ? 1u : 0u) << (8 + w));
        }
        nearBits = m;
      } else if (DDD && d2 < B.rfar2) {
        cls = kClsMid;
        if (pk && d2 >= P.r16sq) {
          cls = d2 >= P.r8sq ? kClsMid8 : kClsMid16;
          loc.w *= gFar * (1.0f / 65536.f);
        }
      } else {
        cls = kClsFar;
        loc.w *= gFar;
      }
    }
    const unsigned lt = (1u << lane) - 1u;
    unsigned myBallot = 0;
#pragma unroll
    for (int c = NODES ? kClsNode : kClsNear; c < kNumCls; c++) {
      const unsigned b = __ballot_sync(0xffffffffu, cls == c);
      if (cls == c) myBallot = b;
      if (lane == 0) S.cnt[c][warp] = __popc(b);
    }
    __syncthreads();
    // Start of each class in the list, and of this warp's atoms within it.
    int base[kNumCls];
    int run = 0, myPos = 0, nodeCnt = 0, midEnd = 0;
#pragma unroll
    for (int c = NODES ? kClsNode : kClsNear; c < kNumCls; c++) {
      if (c == kClsFar) {
        midEnd = run;
        if (NODES && DDD) run = (run + 1) & ~1;
      }
      base[c] = run;
      int off = 0;
#pragma unroll
      for (int w = 0; w < kThreads / 32; w++) {
        const int v = S.cnt[c][w];
        off += (w < warp) ? v : 0;
        run += v;
      }
      if (cls == c) myPos = base[c] + off + __popc(myBallot & lt);
      if (c == kClsNode) {  // whole pairs
        nodeCnt = run;
        run = (run + 1) & ~1;
      }
    }
    const int nNode = NODES ? base[kClsNear] : 0;
    if (NODES && (cls == kClsNode || (farNodes && cls == kClsFar))) {
      float* pr = reinterpret_cast<float*>(S.list) + 8 * (myPos >> 1) + (myPos & 1);
      pr[0] = loc.x;
      pr[2] = loc.y;
      pr[4] = loc.z;
      pr[6] = loc.w;
    } else if (cls >= 0) {
      S.list[myPos] = loc;
      if (cls == kClsNear) {
        S.nearIdx[myPos] = (short)tid;
        S.nearMask[myPos] = (unsigned short)nearBits;
      }
    }
    if (NODES && ((tid == 0 && (nodeCnt & 1)) || (farNodes && tid == 1 && (run & 1)))) {
      // An odd last pair is completed by an atom of no weight far away.
      float* pr = reinterpret_cast<float*>(S.list) + 8 * ((tid == 0 ? nodeCnt : run) >> 1) + 1;
      pr[0] = 1.0e7f;
      pr[2] = 0.f;
      pr[4] = 0.f;
      pr[6] = 0.f;
    }
    __syncthreads();
    if (farNodes && run > base[kClsFar]) {
      far_node_atoms(S, S.list + base[kClsFar], (run - base[kClsFar] + 1) >> 1, B.hx, B.hy, B.hz);
      nodeSeen |= 2;
    }
    if (NODES && nNode > 0) {
      node_atoms<DDD>(S, nNode >> 1, B.hx, B.hy, B.hz);
      nodeSeen |= 1;
    }

    // Mid atoms: table read, or a packed tail table.
    if (DDD && busy) {
      const uint32_t tabBiased = smem_u32(S.tab) - 0x2C000000u;
      const int nMid = base[kClsMid16] - base[kClsMid];
      if (clampMid)
        mid_atoms<MODE, true>(S.list + base[kClsMid], tabBiased, nMid, gxn, gy, gz, sum, cmp);
      else
        mid_atoms<MODE, false>(S.list + base[kClsMid], tabBiased, nMid, gxn, gy, gz, sum, cmp);
      if (pk) {
        const uint32_t p16 = smem_u32(S.packed) - 2u * (0x4B000000u + (uint32_t)P.b16);
        const uint32_t p8 = smem_u32(S.packed) + 16u * (uint32_t)P.vec8 - (0x4B000000u + (uint32_t)P.b8);
        mid_packed_atoms<MODE, 2>(S.list + base[kClsMid16], p16, base[kClsMid8] - base[kClsMid16], gxn, gy, gz, sum,
                                  cmp, P.kScale);
        mid_packed_atoms<MODE, 1>(S.list + base[kClsMid8], p8, midEnd - base[kClsMid8], gxn, gy, gz, sum,
                                  cmp, P.kScale);
      }
    }

    // Far atoms: saturated dielectric (or the constant dielectric), no table.
    const int nFar = busy && !farNodes ? run - base[kClsFar] : 0;
    const float4* farA = S.list + base[kClsFar];
#pragma unroll 1
    for (int j0 = 0; j0 < nFar; j0 += kChunk) {
      float2 cs[kNX / 2];
#pragma unroll
      for (int k = 0; k < kNX / 2; k++)
        cs[k] = (MODE == kEmapKahan) ? make_float2(0.f, 0.f) : sum[k];
      const int j1 = min(nFar, j0 + kChunk);
#pragma unroll 8
      for (int j = j0; j < j1; j++) {
        const float4 a = farA[j];
        const float dy = a.y - gy, dz = a.z - gz;
        const float2 dyz2 = dup2(fmaf(dz, dz, dy * dy));
        const float2 ax = dup2(a.x), aw = dup2(a.w);
#pragma unroll
        for (int k = 0; k < kNX / 2; k++) {
          const float2 dx = __fadd2_rn(ax, gxn[k]);
          cs[k] = __ffma2_rn(aw, rsqrt2(__ffma2_rn(dx, dx, dyz2)), cs[k]);
        }
      }
      add_chunk<MODE>(sum, cmp, cs);
    }

    // Near atoms: clamp 1/r at 2 and decide bins near an edge exactly.
#pragma unroll 1
    for (int j = busy ? base[kClsNear] : base[kClsMid]; j < base[kClsMid]; j++) {
      const float4 a = S.list[j];
      const float dy = a.y - gy, dz = a.z - gz;
      // The 1e-30 keeps r2 > 0 (an atom on a grid point) without a per-point max.
      const float2 dyz2 = dup2(fmaf(dz, dz, dy * dy) + 1e-30f);
      const float2 ax = dup2(a.x), aw = dup2(a.w);
      if (DDD && !((S.nearMask[j] >> warp) & 1u)) {
        // At least rNear from every point of this warp (uniform): the mid-list
        // arithmetic (no cap, round-down bin), each term compensated.  The
        // clamp keeps the bin inside the table for any box size.
        const uint32_t tabB = smem_u32(S.tab) - 0x2C000000u;
#pragma unroll
        for (int k = 0; k < kNX / 2; k++) {
          const float2 dx = __fadd2_rn(ax, gxn[k]);
          const float2 r2 = __ffma2_rn(dx, dx, dyz2);
          const float2 rs = rsqrt2(r2);
          float2 f = __ffma2_rd(r2, rs, dup2(kBias));
          f.x = fminf(f.x, kBias + (float)(kTabLen - 1));
          f.y = fminf(f.y, kBias + (float)(kTabLen - 1));
          const float2 t = make_float2(lds_bin(tabB, f.x), lds_bin(tabB, f.y));
          const float2 wr = __fmul2_rn(aw, rs);
          if (MODE == kEmapKahan)
            kahan2_product(sum[k], cmp[k], wr, t);
          else
            sum[k] = __fadd2_rn(sum[k], __fmul2_rn(wr, t));
        }
        continue;
      }
      if (!clampMid && !((S.nearMask[j] >> (8 + warp)) & 1u))  // uniform
        near_exact<DDD, MODE, false>(S, P, slot, j, dyz2, ax, aw, gxn, iy, iz, xb, xs, sum, cmp);
      else
        near_exact<DDD, MODE, true>(S, P, slot, j, dyz2, ax, aw, gxn, iy, iz, xb, xs, sum, cmp);
    }
    __syncthreads();  // ring slot and atom lists are free again
  }

  // Net-charge checksum: the first CTA of each atom split reports, in FP64,
  // the sum of the weights of every atom that went through its tile ring.
  if (blk == 0 && P.checksum) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) wsum += __shfl_xor_sync(0xffffffffu, wsum, o);
    if (lane == 0) S.wpart[warp] = wsum;
    __syncthreads();
    if (tid == 0) {
      double s = 0.0;
      for (int w = 0; w < kThreads / 32; w++) s += S.wpart[w];
      P.checksum[split] = s;
    }
  }

  // The node atoms' part: their sums at the nodes, interpolated to the points.
  double row5[kNodes1] = {0.0, 0.0, 0.0, 0.0, 0.0};
  if (NODES && nodeSeen) {
    double* F = reinterpret_cast<double*>(S.list);
    double* F4 = F + kNodes;  // far nodes' sums
    NodeAxis* axis = reinterpret_cast<NodeAxis*>(S.list) + kAxisAt;
    if (tid < 3) axis[tid].set(tid == 0 ? B.hx : tid == 1 ? B.hy : B.hz);
    if (nodeSeen & 2) {
      if (tid < kFarNodes) {
        double f = 0.0;
#pragma unroll
        for (int w = 0; w < kThreads / 32; w++) {
          const float4 a = S.farAcc()[32 * w + (tid >> 1)];
          f += (tid & 1) ? (double)a.z - (double)a.w : (double)a.x - (double)a.y;
        }
        F4[tid] = f;
      }
      __syncthreads();
    }
    if (tid < kNodes) {
      double f = (nodeSeen & 2) ? far_field(F4, tid, B.hx, B.hy, B.hz) : 0.0;
#pragma unroll
      for (int grp = 0; grp < kNodeGroups; grp++) {
        const float4 a = S.nodeAcc[64 * grp + (tid >> 1)];
        f += (tid & 1) ? (double)a.z - (double)a.w : (double)a.x - (double)a.y;
      }
      F[tid] = f;
    }
    __syncthreads();
    node_row(F, axis[1], axis[2], gy, gz, row5);
  }

  if (!active) return;
  const int64_t row = ((int64_t)iz * P.ny + iy) * P.nx;
#pragma unroll
  for (int k = 0; k < kNX; k++) {
    const int x = xb + k * xs;
    if (x >= P.nx) break;
    double v = (MODE == kEmapKahan) ? (double)lo_hi(sum[k >> 1], k) + (double)lo_hi(cmp[k >> 1], k)
                                    : (double)lo_hi(sum[k >> 1], k);
    if (NODES && nodeSeen) {
      double wx[kNodes1];
      reinterpret_cast<const NodeAxis*>(S.list)[kAxisAt].weights(-(double)lo_hi(gxn[k >> 1], k), wx);
#pragma unroll
      for (int kx = 0; kx < kNodes1; kx++) v = fma(wx[kx], row5[kx], v);
    }
    if (P.nsplit == 1)
      P.out[row + x] = (float)v;
    else
      P.partial[(int64_t)split * P.npoints + row + x] = v;
  }
}

template <bool DDD, int MODE, bool NODES>
__global__ void __launch_bounds__(kThreads, kEmapCtasPerSm) emap_kernel(const __grid_constant__ EmapParams P) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  EmapSmem& S = *reinterpret_cast<EmapSmem*>(smem_raw);
  emap_unit<DDD, MODE, NODES>(P, blockIdx.x % P.nblocks, blockIdx.x / P.nblocks, S);
}

// Persistent kernel over the work units of many jobs (a batch of receptors):
// every CTA takes the next unit (job, CTA box) from an atomic counter until
// none is left; the host orders units by decreasing cost.  Jobs run without
// an atom split and with the distance-dependent dielectric.  Two CTAs per SM:
// at three the per-unit job parameters spill and the batch gains nothing.
template <int MODE>
__global__ void __launch_bounds__(kThreads, 2)
    emap_batch_kernel(const EmapParams* __restrict__ jobs, const int2* __restrict__ units, int nunits, int* counter) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  EmapSmem& S = *reinterpret_cast<EmapSmem*>(smem_raw);
  for (;;) {
    __syncthreads();  // the previous unit is finished by every thread
    if (threadIdx.x == 0) S.unit = atomicAdd(counter, 1);
    __syncthreads();
    const int u = S.unit;
    if (u >= nunits) return;
    const int2 w = units[u];
    emap_unit<true, MODE, MODE == kEmapKahan>(jobs[w.x], w.y, 0, S);
  }
}

// Persistent direct e-map over a device-side list of CTA boxes.
template <int MODE>
__global__ void __launch_bounds__(kThreads, kEmapCtasPerSm)
    emap_list_kernel(const __grid_constant__ EmapParams P, const int* __restrict__ list, const int* __restrict__ count,
                     int* counter) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  EmapSmem& S = *reinterpret_cast<EmapSmem*>(smem_raw);
  const int n = min(*count, P.nblocks);
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) S.unit = atomicAdd(counter, 1);
    __syncthreads();
    const int u = S.unit;
    if (u >= n) return;
    const int blk = list[u];
    if (blk < 0 || blk >= P.nblocks) {
      if (threadIdx.x == 0) atomicOr(P.status, ST_BAD_INPUT);
      continue;
    }
    emap_unit<true, MODE, false>(P, blk, 0, S);
  }
}

cudaError_t emap_list_launch(const EmapParams& P, const int* list, const int* count, int* counter, int grid,
                             cudaStream_t st) {
  const size_t smem = sizeof(EmapSmem);
  cudaError_t e = cudaFuncSetAttribute(emap_list_kernel<kEmapKahan>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(counter, 0, sizeof(int), st);
  if (e != cudaSuccess) return e;
  emap_list_kernel<kEmapKahan><<<grid, kThreads, smem, st>>>(P, list, count, counter);
  return cudaGetLastError();
}

// Sum the atom-split partials in split order (FP64).
__global__ void emap_reduce_kernel(const double* __restrict__ partial, int nsplit, int64_t n, float* __restrict__ out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int k = 0; k < nsplit; k++) s += partial[(int64_t)k * n + i];
    out[i] = (float)s;
  }
}

// Volume within d of a box of half extents h, and that body's surface area.
__device__ __forceinline__ float volume_within(const float3 h, float d) {
  return 8.f * h.x * h.y * h.z + 8.f * (h.x * h.y + h.y * h.z + h.z * h.x) * d +
         6.2831853f * (h.x + h.y + h.z) * d * d + 4.1887902f * d * d * d;
}
__device__ __forceinline__ float area_at(const float3 h, float d) {
  return 8.f * (h.x * h.y + h.y * h.z + h.z * h.x) + 12.566371f * (h.x + h.y + h.z) * d + 12.566371f * d * d;
}

// The node radii of NB boxes of a job with the distance-dependent dielectric.
//
// A node atom enters without the table's 0.01 A steps, which leaves out an
// error energy of w^2 exp(-2 lambda r) times a constant (4.2e-6 of a term, rms,
// at 24 A).  Exact bins reach 0.75 A further than they would have to without
// node sums, which removes an energy that grows with the density of squared
// weights there.  Where that density is the same at both distances, as inside a
// receptor, the second is 1.8 times the first for R = 24 A.  Beside a receptor
// few atoms are near and many far.  So R is the least radius from 24 A on for
// which the density of squared weights within 3.5 A of the exact radius is at
// least that of the node atoms', weighted by their energy.  Where the near weights
// lie to one side of the box (their mean unit vector is longer than kRadiusLean;
// half a shell has 0.5), some of its points have far fewer near atoms than the
// box, and the density must be kRadiusMargin times as large: the energy left out is
// then a fifth of the one removed.  Past 36 A the steps are below FP32 rounding.
//
// Errors against FP64 (relative 2-norm), 20,000 atoms (43 A) and 41^3 points 0,
// 50, 55, 63 and 75 A from the middle, over those without node sums and with
// exact bins to 11 A: 0.91, 0.90, 0.93, 0.95 and 0.82; with R = 24 A everywhere
// 0.91, 1.04, 1.24, 2.19 and 0.92.  Time for 20,000 atoms on 161^3 points 10.9 ms,
// with R = 24 A 10.7, with the margin everywhere 11.2; 60,000 on 255^3 51.6, 50.5
// and 53.3; 8,000 on 125 x 97 x 83 2.53, 2.48 and 2.54.
template <int NB>
__device__ __forceinline__ void box_radii(const EmapParams& P, const int blk0) {
  // Energies from each radius on, the near squared weights, and those times
  // their unit vectors from the box.
  constexpr int kSums = kRadiusSteps + 4;
  __shared__ float part[kThreads / 32][NB][kSums];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float rn = sqrtf(P.rnear2), n0 = rn - 350.f, n1 = rn + 350.f;
  const float nl2 = -9.0998494e-3f;        // -2 lambda / (100 ln 2)
  const float depth = 158.54f;             // 100 / (2 lambda): the energies' e-folding depth
  float3 o[NB], h[NB];
  float inner[NB], s[NB][kSums];
#pragma unroll
  for (int b = 0; b < NB; b++) {
    const EmapBlock& B = P.blocks[min(blk0 + b, P.nblocks - 1)];
    o[b] = make_float3((float)(100.0 * B.ox), (float)(100.0 * B.oy), (float)(100.0 * B.oz));
    h[b] = make_float3(B.hx, B.hy, B.hz);
    inner[b] = fmaxf(P.rnodeHalfWidths * B.rnode, P.rnodeMin);
#pragma unroll
    for (int k = 0; k < kSums; k++) s[b][k] = 0.f;
  }
#pragma unroll 2
  for (int i = tid; i < P.n_atoms; i += kThreads) {
    const double4 a = P.atoms[i];
    const float x = (float)(100.0 * a.x), y = (float)(100.0 * a.y), z = (float)(100.0 * a.z), w = (float)a.w;
#pragma unroll
    for (int b = 0; b < NB; b++) {
      const float dx = fmaxf(fabsf(x - o[b].x) - h[b].x, 0.f), dy = fmaxf(fabsf(y - o[b].y) - h[b].y, 0.f),
                  dz = fmaxf(fabsf(z - o[b].z) - h[b].z, 0.f);
      const float d = sqrtf(dx * dx + dy * dy + dz * dz), u = d - inner[b], step = kRadiusStep * inner[b];
      if (d >= n0 && d < n1) {
        const float w2 = w * w, wd = __fdividef(w2, d);
        s[b][kRadiusSteps] += w2;
        s[b][kRadiusSteps + 1] += copysignf(dx, x - o[b].x) * wd;
        s[b][kRadiusSteps + 2] += copysignf(dy, y - o[b].y) * wd;
        s[b][kRadiusSteps + 3] += copysignf(dz, z - o[b].z) * wd;
      }
      const float e = w * w * ex2_approx(nl2 * u);
#pragma unroll
      for (int k = 0; k < kRadiusSteps; k++)
        if (u >= k * step && u < kRadiusSteps * step) s[b][k] += e;
    }
  }
#pragma unroll
  for (int b = 0; b < NB; b++)
#pragma unroll
    for (int k = 0; k < kSums; k++) {
#pragma unroll
      for (int m = 16; m > 0; m >>= 1) s[b][k] += __shfl_xor_sync(0xffffffffu, s[b][k], m);
      if (lane == 0) part[warp][b][k] = s[b][k];
    }
  __syncthreads();
  if (tid < NB && blk0 + tid < P.nblocks) {
    const EmapBlock& B = P.blocks[blk0 + tid];
    const float3 hb = make_float3(B.hx, B.hy, B.hz);
    float v[kSums] = {};
    for (int w = 0; w < kThreads / 32; w++)
#pragma unroll
      for (int k = 0; k < kSums; k++) v[k] += part[w][tid][k];
    const float r0 = fmaxf(P.rnodeHalfWidths * B.rnode, P.rnodeMin);
    const float nearVol = volume_within(hb, n1) - volume_within(hb, n0), farVol = depth * area_at(hb, r0 + depth);
    const float vx = v[kRadiusSteps + 1], vy = v[kRadiusSteps + 2], vz = v[kRadiusSteps + 3], vn = v[kRadiusSteps];
    const bool inside = vx * vx + vy * vy + vz * vz < kRadiusLean * kRadiusLean * vn * vn;
    const float limit = vn * farVol, scale = (inside ? 1.f : kRadiusMargin) * nearVol;
    int k = 0;
    while (k < kRadiusSteps && limit < scale * v[k]) k++;
    float t = (float)k;
    if (k > 0 && limit > 0.f) {
      // Between the last radius that fails and the first that does not, where the
      // energy falls off evenly (no faster than for an even density).
      const float fall = fminf(k < kRadiusSteps && v[k] > 0.f ? __logf(v[k - 1] / v[k]) : 1.0e30f,
                               r0 * kRadiusStep / depth);
      t = k - 1 + fminf(1.f, __logf(scale * v[k - 1] / limit) / fall);
    }
    const float r = r0 * (1.f + t * kRadiusStep);
    P.radius[blk0 + tid] = make_float2(r, fmaxf(kFarNodeHalfWidths * B.rnode, fmaxf(kFarNodeRadius, r)));
  }
}

__global__ void __launch_bounds__(kThreads) emap_radius_kernel(const __grid_constant__ EmapParams P) {
  box_radii<kRadiusBoxes>(P, kRadiusBoxes * blockIdx.x);
}

// One unit (job, CTA box) of a batch per CTA.
__global__ void __launch_bounds__(kThreads)
    emap_batch_radius_kernel(const EmapParams* __restrict__ jobs, const int2* __restrict__ units) {
  const int2 w = units[blockIdx.x];
  if (jobs[w.x].radius) box_radii<1>(jobs[w.x], w.y);
}

cudaError_t emap_batch_launch(const EmapParams* jobs, const int2* units, int nunits, int* counter, int grid,
                              cudaStream_t st) {
  const size_t smem = sizeof(EmapSmem);
  cudaError_t e = cudaFuncSetAttribute(emap_batch_kernel<kEmapKahan>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(counter, 0, sizeof(int), st);
  if (e != cudaSuccess) return e;
  emap_batch_radius_kernel<<<nunits, kThreads, 0, st>>>(jobs, units);
  emap_batch_kernel<kEmapKahan><<<grid, kThreads, smem, st>>>(jobs, units, nunits, counter);
  return cudaGetLastError();
}

size_t emap_smem_bytes() { return sizeof(EmapSmem); }

cudaError_t emap_launch(const EmapParams& P, bool ddd, int mode, int grid, cudaStream_t st) {
  const size_t smem = sizeof(EmapSmem);
  cudaError_t e = cudaSuccess;
#define AG_LAUNCH(D, M, N)                                                                                  \
  do {                                                                                                      \
    e = cudaFuncSetAttribute(emap_kernel<D, M, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
    if (e != cudaSuccess) return e;                                                                         \
    emap_kernel<D, M, N><<<grid, kThreads, smem, st>>>(P);                                                  \
  } while (0)
  // Without node sums a kernel without their code: small grids, whose CTAs see
  // one or two tiles each, took 5-8 % longer with it.
  const bool nodes = mode == kEmapKahan && P.rnodeMin < 1.0e30f;
  if (nodes && ddd)
    emap_radius_kernel<<<(P.nblocks + kRadiusBoxes - 1) / kRadiusBoxes, kThreads, 0, st>>>(P);
  if (mode != kEmapKahan) {
    if (ddd) AG_LAUNCH(true, kEmapPlain, false); else AG_LAUNCH(false, kEmapPlain, false);
  } else if (nodes) {
    if (ddd) AG_LAUNCH(true, kEmapKahan, true); else AG_LAUNCH(false, kEmapKahan, true);
  } else {
    if (ddd) AG_LAUNCH(true, kEmapKahan, false); else AG_LAUNCH(false, kEmapKahan, false);
  }
#undef AG_LAUNCH
  e = cudaGetLastError();
  if (e != cudaSuccess || P.nsplit == 1) return e;
  emap_reduce_kernel<<<592, 256, 0, st>>>(P.partial, P.nsplit, P.npoints, P.out);
  return cudaGetLastError();
}

}  // namespace agk
