// yee_fused.cuh -- one or two whole timesteps of the Yee update in one pass
// over memory.
//
// The register kernels (yee_kernels.cuh) stream every field and coefficient
// array through HBM twice a timestep (H, then E): 120 B a cell and step with
// full coefficient arrays.  Here a CTA marches a tile of the (y, z) plane
// through x and carries a cell from step n to n + kSteps before it is written:
//
//   iteration i:  A  H(n+1/2) of plane i      from E(n) of planes i, i+1
//                 B  E(n+1)   of plane i      from H(n+1/2) of planes i-1, i
//      kSteps=2:  C  H(n+3/2) of plane i-1    from E(n+1) of planes i-1, i
//                 D  E(n+2)   of plane i-1    from H(n+3/2) of planes i-2, i-1
//
// and coefficients come from a table of the distinct sets (a material id per
// cell), so a two-step pass moves 48 B of fields and 1-2 B of ids per cell.
// Every value is computed by the operations of yee_kernels.cuh in the same
// order (products and sums rounded separately), so results are the same bits.
//
// Tiles overlap: kSteps rows and one float4 chunk on every inner side are
// loaded and computed but not written (their values near the tile's edge are
// wrong after a step and never reach a written cell).  Neighbouring CTAs read
// the overlap at step n, so the pass reads one set of field (and CPML psi)
// buffers and writes another.
//
// One thread owns one chunk (4 cells along z) of the tile.  Its x-neighbours
// stay in registers or in the ring, z-neighbours come by shuffle (through shared memory
// across a warp's edge), y-neighbours through shared memory.  The planes
// ahead are copied into a shared-memory ring (cp.async) two iterations before
// they are used, so two barriers an iteration are the only waits.
#pragma once

#include "yee_kernels.cuh"

namespace oems {

constexpr int kFusedMaxThreads = 512;
constexpr int kFusedMaxBox = 7;
// floats of one row of warp-edge values (a float per warp), of which there
// are five; what follows them is read 16 bytes at a time
constexpr int kFusedEdge = 20;
static_assert(kFusedEdge > kFusedMaxThreads / 32 && 5 * kFusedEdge % 4 == 0, "aligned tables");

// A part of the grid a pass writes: planes [i0, i1) x rows [j0, j1) x chunks
// [q0, q1), cut into tiles of ty rows x wz chunks (the overlap included; each
// next tile starts sy rows / sz chunks on) and x-runs of xlen planes.  axes:
// the CPML slabs (bit 0 x, 1 y, 2 z) its cells and their overlap may meet;
// each value has its own code, so a part clear of the slabs runs without any
// of the CPML's registers and branches.
struct FusedBox {
  int i0, i1, j0, j1, q0, q1;
  int ja, qa;  // first row / chunk loaded
  int wz, ty, sz, sy, ntz, nty, xlen;
  int axes, item0;
};

struct FusedArgs {
  int nx, ny, nz, nzp, nzq;
  long long plane;   // elements per x-plane
  long long comp;    // elements per field component
  const void* in;    // Ex Ey Ez Hx Hy Hz, `comp` elements apart
  void* out;
  const void* ids;
  const float* table;  // [ntable][12] = ca0..2 cb0..2 da0..2 db0..2
  int ntable;
  int nbox;
  FusedBox box[kFusedMaxBox];
  // CPML: psi of the buffer read; the one written lies psi_out floats on
  CpmlArgs cp;
  long long psi_out;
  int pairs;    // (cell column, slab) pairs a CTA's shared memory has room for
  int poff[6];  // profiles in shared memory: 6 rows of L (x, y faces) or of the psi row width (z)
  // sources, sorted by (plane, row, chunk), list order kept among equals
  int nsrc, src_lo, src_hi;  // planes that hold sources: [src_lo, src_hi)
  const int* src_off;        // [nx + 1]
  const int* src_key;        // row * nzq + chunk
  const int* src_meta;       // element | dir << 2 | soft << 4
  const long long* src_first;
  const long long* src_count;
  const float* samples;
  // taps: field values the probes read, sorted like the sources
  int ntap, tap_lo, tap_hi;
  const int* tap_off;
  const int* tap_key;
  const int* tap_meta;  // element | component << 2
  const int* tap_slot;
  float* taps;          // [step of the span][ntap]
  const long long* d_base;
  int local;            // step of the span this pass starts at
  float h_inv;
};

// Planes of E and H in the ring.  Clear of the slabs the copies run two
// iterations ahead; in the slabs an iteration is long enough that one will
// do, and the room goes to psi.
constexpr int fused_ring_e(bool cpml) { return cpml ? 2 : 3; }
constexpr int fused_ring_h(bool cpml) { return cpml ? 1 : 2; }

// Shared-memory bytes of a CTA of nt threads (elem: bytes per field value).
__host__ __device__ inline size_t fused_smem(int steps, bool cpml, int nt, int elem, int id_bytes, int table_floats,
                                             int prof_floats, int pairs) {
  const size_t ring = (size_t)(3 * (fused_ring_e(cpml) + fused_ring_h(cpml)) * elem + fused_ring_e(cpml) * id_bytes) * nt * 4;
  const size_t ex = (size_t)(steps == 2 ? 10 : 4) * nt * 16, psi = (size_t)pairs * 4 * steps * 16;
  return ring + ex + psi + (5 * kFusedEdge + ((table_floats + 3) & ~3) + prof_floats) * sizeof(float);
}

template <typename T>
struct ChunkIO {
  using Raw = uint2;
  static __device__ __forceinline__ void unpack(const Raw& r, float (&v)[4]) {
    to_arr(FieldIO<T>::unpack(r), v);
  }
  static __device__ __forceinline__ void round(float (&v)[4]) {
    const float2 a = FieldIO<T>::cvt(FieldIO<T>::pack(v[0], v[1])), b = FieldIO<T>::cvt(FieldIO<T>::pack(v[2], v[3]));
    v[0] = a.x;
    v[1] = a.y;
    v[2] = b.x;
    v[3] = b.y;
  }
  static __device__ __forceinline__ void copy(uint32_t dst, const void* src, bool on) {
    const int n = on ? 8 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
  }
};
template <>
struct ChunkIO<float> {
  using Raw = float4;
  static __device__ __forceinline__ void unpack(const Raw& r, float (&v)[4]) { to_arr(r, v); }
  static __device__ __forceinline__ void round(float (&)[4]) {}
  static __device__ __forceinline__ void copy(uint32_t dst, const void* src, bool on) {
    const int n = on ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
  }
};

// What a thread knows of its cell column and of the slabs it crosses.
struct FusedCell {
  int j, k0;
  bool in;          // inside the grid
  bool own;         // written by this tile
  bool jp, jm;      // row j + 1 / j - 1 exists
  unsigned live_h;  // elements below nz
  unsigned live_e;  // ... and k >= 1
  int fy, ly;       // y slab and layer
  int fz;           // z slab
  unsigned mz;      // elements inside it
  bool both;        // the chunk also meets the z-max slab (thin grids)
  int iy, iz, ix;   // places of its psi in shared memory
};

// Elements of the chunk at k0 inside z slab f.
__device__ __forceinline__ unsigned fused_zmask(const FusedArgs& a, int f, int k0) {
  unsigned m = 0;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int l = k0 + e - a.cp.start[f];
    m |= (l >= 0 && l < a.cp.L[f] ? 1u : 0u) << e;
  }
  return m;
}

// psi of a thread's stretched differences -- y slab (dy of comp 0, dy of comp
// 2), z slab (dz of comp 0, dz of comp 1), x slab (dx of comp 1, dx of comp
// 2) -- in shared memory, from their copy (issued as soon as the place is
// free) to the step that writes them out.  Only the thread itself touches
// them, so they need no barrier.  Places: [plane parity][H 0, H 1, E 0, E 1]
// [pair], one pair per (thread, slab) that the tile holds.
template <int kSteps, int kAxes, bool kH>
struct FusedPsi {
  static __device__ __forceinline__ float* at(const FusedArgs& a, const FusedCell& c, int f, int slot, int i, int lx) {
    const CpmlArgs& cp = a.cp;
    const long long o = f < 2 ? ((long long)lx * a.ny + c.j) * a.nzp + c.k0
                        : f < 4 ? ((long long)i * cp.L[f] + c.ly) * a.nzp + c.k0
                                : ((long long)i * a.ny + c.j) * cp.zw[f - 4] + c.k0 - cp.zbase[f - 4];
    return (kH ? cp.psi_h[f][slot] : cp.psi_e[f][slot]) + o;
  }
  static __device__ __forceinline__ float4* place(const FusedArgs& a, float4* psi, int i, int slot, int pair) {
    return psi + ((kSteps == 2 ? (i & 1) * 4 : 0) + (kH ? 0 : 2) + slot) * a.pairs + pair;
  }
  static __device__ __forceinline__ void fetch(const FusedArgs& a, const FusedCell& c, float4* psi, int f, int i, int lx,
                                               int pair) {
#pragma unroll
    for (int s = 0; s < 2; ++s)
      ChunkIO<float>::copy((uint32_t)__cvta_generic_to_shared(place(a, psi, i, s, pair)), at(a, c, f, s, i, lx), true);
  }
  // Starts the copies of plane i's psi.
  static __device__ __forceinline__ void load(const FusedArgs& a, const FusedCell& c, float4* psi, int i) {
    if (!c.in || i >= a.nx) return;
    int lx = 0;
    const int fx = kAxes & 1 ? cpml_face(a.cp, 0, i, lx) : -1;
    if ((kAxes & 2) && c.fy >= 0) fetch(a, c, psi, c.fy, i, lx, c.iy);
    if ((kAxes & 4) && c.fz >= 0) fetch(a, c, psi, c.fz, i, lx, c.iz);
    if ((kAxes & 1) && fx >= 0) fetch(a, c, psi, fx, i, lx, c.ix);
  }
  static __device__ __forceinline__ void row(float (&d)[4], float4& v, float b, float cc, float ik, unsigned m) {
    float q[4];
    to_arr(v, q);
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (m >> e & 1u) d[e] = cpml_stretch(d[e], q[e], b, cc, ik);
    v = to_f4(q);
  }
  static __device__ __forceinline__ void zrow(const FusedArgs& a, const float* prof, int f, int k0, float (&d)[4],
                                              float4& v, unsigned m) {
    const int w = a.cp.zw[f - 4], o = k0 - a.cp.zbase[f - 4];
    const float* pr = prof + a.poff[f] + (kH ? 3 * w : 0) + o;
    float q[4], b[4], cc[4], ik[4];
    to_arr(v, q);
    to_arr(*reinterpret_cast<const float4*>(pr), b);
    to_arr(*reinterpret_cast<const float4*>(pr + w), cc);
    to_arr(*reinterpret_cast<const float4*>(pr + 2 * w), ik);
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (m >> e & 1u) d[e] = cpml_stretch(d[e], q[e], b[e], cc[e], ik[e]);
    v = to_f4(q);
  }
  // One step's new psi: kept for the pass's second step, or written out.
  template <bool kLast>
  static __device__ __forceinline__ void put(const FusedArgs& a, const FusedCell& c, float4* q, int f, int slot, int i,
                                             int lx, bool own, float4 v) {
    if constexpr (!kLast)
      *q = v;
    else if (own)
      st4(at(a, c, f, slot, i, lx) + a.psi_out, v);
  }

  // Stretches the differences d (dy of comp 0, dz of comp 0, dz of comp 1,
  // dx of comp 1, dx of comp 2, dy of comp 2) of plane i; kLast: the last
  // step of the pass.
  template <bool kLast>
  static __device__ __forceinline__ void apply(const FusedArgs& a, const float* prof, float4* psi, const FusedCell& c,
                                               int i, bool own, float (&d)[6][4], unsigned live) {
    int lx = 0;
    const int fx = (kAxes & 1) && c.in ? cpml_face(a.cp, 0, i, lx) : -1;
    if ((kAxes & 2) && c.fy >= 0) {
      const int L = a.cp.L[c.fy];
      const float* pr = prof + a.poff[c.fy] + (kH ? 3 * L : 0) + c.ly;
      const float b = pr[0], cc = pr[L], ik = pr[2 * L];
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        float4* q = place(a, psi, i, s, c.iy);
        float4 v = *q;
        row(d[s ? 5 : 0], v, b, cc, ik, live);
        put<kLast>(a, c, q, c.fy, s, i, lx, own, v);
      }
    }
    if ((kAxes & 4) && c.fz >= 0) {
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        float4* q = place(a, psi, i, s, c.iz);
        float4 v = *q;
        zrow(a, prof, c.fz, c.k0, d[1 + s], v, live & c.mz);
        put<kLast>(a, c, q, c.fz, s, i, lx, own, v);
      }
      if (kSteps == 1 && c.both) {
        // the z-max slab's part of a chunk that meets both (such grids run
        // one step a pass)
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          float* q = at(a, c, 5, s, i, lx);
          float4 v = ld_nc4(q);
          zrow(a, prof, 5, c.k0, d[1 + s], v, live & fused_zmask(a, 5, c.k0));
          if (own) st4(q + a.psi_out, v);
        }
      }
    }
    if ((kAxes & 1) && fx >= 0) {
      const int L = a.cp.L[fx];
      const float* pr = prof + a.poff[fx] + (kH ? 3 * L : 0) + lx;
      const float b = pr[0], cc = pr[L], ik = pr[2 * L];
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        float4* q = place(a, psi, i, s, c.ix);
        float4 v = *q;
        row(d[3 + s], v, b, cc, ik, live);
        put<kLast>(a, c, q, fx, s, i, lx, own, v);
      }
    }
  }
};

// Six coefficients (a0 a1 a2 b0 b1 b2) of element e's material: the E half
// of a table row or the H half.
template <int kIdBytes, bool kH>
__device__ __forceinline__ void fused_coef(const float* tab, uint32_t w0, uint32_t w1, int e, float (&ca)[3],
                                           float (&cb)[3]) {
  const int id = kIdBytes == 1 ? (w0 >> (8 * e)) & 0xff : ((e < 2 ? w0 : w1) >> (16 * (e & 1))) & 0xffff;
  const float* r = tab + id * 12;
  float4 q;
  float2 p;
  if constexpr (kIdBytes == 1) {
    q = *reinterpret_cast<const float4*>(r + (kH ? 8 : 0));
    p = *reinterpret_cast<const float2*>(r + (kH ? 6 : 4));
  } else {
    q = __ldg(reinterpret_cast<const float4*>(r + (kH ? 8 : 0)));
    p = __ldg(reinterpret_cast<const float2*>(r + (kH ? 6 : 4)));
  }
  if constexpr (kH) {
    ca[0] = p.x;
    ca[1] = p.y;
    ca[2] = q.x;
    cb[0] = q.y;
    cb[1] = q.z;
    cb[2] = q.w;
  } else {
    ca[0] = q.x;
    ca[1] = q.y;
    ca[2] = q.z;
    cb[0] = q.w;
    cb[1] = p.x;
    cb[2] = p.y;
  }
}

// u = ca u + cb curl for the elements of `live` (others keep u).  A row of
// the table per element: a second path for warps of one material (one row a
// chunk) issued fewer loads but measured 5-10% slower (256^3, both kernels).
// kCpml: the elements are selected, else restored behind a branch few chunks
// take; each form is the faster one in its kernel (118 against 126 us a step
// without slabs, 204 against 214 with).
template <int kIdBytes, bool kH, bool kCpml>
__device__ __forceinline__ void fused_apply(const float* tab, uint32_t w0, uint32_t w1, const float (&d)[6][4],
                                            unsigned live, float (&u)[3][4]) {
  float v[3][4], ca[3], cb[3];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    fused_coef<kIdBytes, kH>(tab, w0, w1, e, ca, cb);
    const float curl[3] = {__fsub_rn(d[0][e], d[1][e]), __fsub_rn(d[2][e], d[3][e]), __fsub_rn(d[4][e], d[5][e])};
#pragma unroll
    for (int c = 0; c < 3; ++c) v[c][e] = __fadd_rn(__fmul_rn(ca[c], u[c][e]), __fmul_rn(cb[c], curl[c]));
  }
  if (kCpml || live != 15u) {
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
      for (int c = 0; c < 3; ++c)
        if (!(live >> e & 1u)) v[c][e] = u[c][e];
  }
#pragma unroll
  for (int e = 0; e < 4; ++e)
#pragma unroll
    for (int c = 0; c < 3; ++c) u[c][e] = v[c][e];
}

// First entry of [lo, hi) whose key is not below `key`.
__device__ __forceinline__ int fused_find(const int* keys, int lo, int hi, int key) {
  while (lo < hi) {
    const int m = (lo + hi) >> 1;
    if (__ldg(keys + m) < key)
      lo = m + 1;
    else
      hi = m;
  }
  return lo;
}

// Whether plane i holds entries of a table over the planes [lo, hi): only such
// planes pay for the calls below and their copies of the cell's values.  Every
// plane between the first and the last probe did: 128^3 with CPML, a source and
// two probes 50.5 us a step, 38.7 now, and a batch of one step 134 us, 110 now
// (the separate kernels 113); 256^3 with CPML 207 -> 198.  The two loads a plane
// show on the smallest grids only (20^3 5.2 -> 5.7 us a step).
__device__ __forceinline__ bool fused_any(const int* off, int lo, int hi, int i) {
  return i >= lo && i < hi && __ldg(off + i + 1) > __ldg(off + i);
}

// Sources of plane i, pass step `s` (batch step): e = or += the sample, in
// list order.
template <typename T>
__device__ __noinline__ void fused_sources(const FusedArgs& a, int i, int key, long long s, float* e) {
  const int end = __ldg(a.src_off + i + 1);
  for (int x = fused_find(a.src_key, __ldg(a.src_off + i), end, key); x < end && __ldg(a.src_key + x) == key; ++x) {
    if (s >= __ldg(a.src_count + x)) continue;
    const float v = __ldg(a.samples + __ldg(a.src_first + x) + s);
    const int m = __ldg(a.src_meta + x);
    float* p = e + ((m >> 2) & 3) * 4 + (m & 3);
    float r = (m >> 4) ? __fadd_rn(*p, v) : v;
    if constexpr (!FieldIO<T>::kFloat) r = FieldIO<T>::cvt1(FieldIO<T>::round1(r));
    *p = r;
  }
}

// Values of plane i the probes read, after batch-span step `row`.
__device__ __noinline__ void fused_taps(const FusedArgs& a, int i, int key, int row, const float* e, const float* h) {
  const int end = __ldg(a.tap_off + i + 1);
  for (int x = fused_find(a.tap_key, __ldg(a.tap_off + i), end, key); x < end && __ldg(a.tap_key + x) == key; ++x) {
    const int m = __ldg(a.tap_meta + x), c = m >> 2;
    const float v = c < 3 ? e[c * 4 + (m & 3)] : __fmul_rn(h[(c - 3) * 4 + (m & 3)], a.h_inv);
    a.taps[(long long)row * a.ntap + __ldg(a.tap_slot + x)] = v;
  }
}

// f on a copy of v in memory (a call on v itself would keep v out of
// registers for the whole item).
template <typename F>
__device__ __forceinline__ void with_copy(float (&v)[3][4], F f) {
  float m[12];
#pragma unroll
  for (int x = 0; x < 12; ++x) m[x] = v[x / 4][x % 4];
  f(m);
#pragma unroll
  for (int x = 0; x < 12; ++x) v[x / 4][x % 4] = m[x];
}

// Work item w of box B.  Every thread of the CTA calls it.
template <int kSteps, int kIdBytes, int kAxes, typename T>
__device__ __forceinline__ void fused_item(const FusedArgs& a, const FusedBox& B, int w, char* smem, const float* tab,
                                           const float* prof) {
  constexpr bool kCpml = kAxes != 0;
  constexpr int kRingE = fused_ring_e(kCpml), kRingH = fused_ring_h(kCpml);
  using PsiH = FusedPsi<kSteps, kAxes, true>;
  using PsiE = FusedPsi<kSteps, kAxes, false>;
  using CIO = ChunkIO<T>;
  using Raw = typename CIO::Raw;
  const int nt = blockDim.x, t = threadIdx.x, lane = t & 31, warp = t >> 5;
  Raw* ringE = reinterpret_cast<Raw*>(smem);    // [plane][3][nt]
  Raw* ringH = ringE + 3 * kRingE * nt;
  char* ringI = reinterpret_cast<char*>(ringH + 3 * kRingH * nt);  // ids of the planes of ringE
  float4* x1 = reinterpret_cast<float4*>(ringI + kRingE * 4 * kIdBytes * nt);  // H of this step, two planes: hx hz
  float4* x2 = x1 + 4 * nt;         // E(n+1) of two planes: ex ez
  float4* x3 = x2 + 4 * nt;                             // H of the second step: hx hz
  constexpr int kEdge = kFusedEdge;
  float4* psi = x1 + (kSteps == 2 ? 10 : 4) * nt;
  float* edge = reinterpret_cast<float*>(psi + (kCpml ? a.pairs * 4 * kSteps : 0));  // [5][kEdge]

  const int tiles = B.ntz * B.nty, wz = B.wz;
  const int xc = w / tiles, tl = w - xc * tiles;
  const int tj = tl / B.ntz, tz = tl - tj * B.ntz;
  const int i0 = B.i0 + xc * B.xlen, i1 = min(i0 + B.xlen, B.i1);
  const int r = t / wz, cc = t - r * wz;
  FusedCell c;
  c.j = B.ja + tj * B.sy + r;
  const int q = B.qa + tz * B.sz + cc;
  c.k0 = q * 4;
  c.in = r < B.ty && c.j < a.ny && q < a.nzq;
  c.own = c.in && c.j >= B.j0 && c.j < B.j1 && q >= B.q0 && q < B.q1 && (tj == 0 || r >= kSteps) &&
          (tj == B.nty - 1 || r < B.ty - kSteps) && (tz == 0 || cc >= 1) && (tz == B.ntz - 1 || cc < wz - 1);
  c.jp = c.j + 1 < a.ny;
  c.jm = c.j >= 1;
  c.live_h = c.live_e = 0;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    c.live_h |= (c.in && c.k0 + e < a.nz ? 1u : 0u) << e;
    c.live_e |= (c.in && c.jm && c.k0 + e >= 1 && c.k0 + e < a.nz ? 1u : 0u) << e;
  }
  c.fy = c.fz = -1;
  c.ly = 0;
  c.mz = 0;
  c.both = false;
  if (kCpml && c.in) {
    c.fy = cpml_face(a.cp, 1, c.j, c.ly);
    const bool z0 = a.cp.L[4] > 0 && c.k0 < a.cp.L[4], z1 = a.cp.L[5] > 0 && c.k0 + 3 >= a.cp.start[5];
    c.fz = z0 ? 4 : z1 ? 5 : -1;
    c.both = z0 && z1;
    if (c.fz >= 0) c.mz = fused_zmask(a, c.fz, c.k0);
    // the tile's slab rows (min face first), then its slab columns, then (x
    // slabs) every thread
    const int j0 = B.ja + tj * B.sy, q0 = B.qa + tz * B.sz, je = min(j0 + B.ty, a.ny), qe = min(q0 + wz, a.nzq);
    const int y0 = max(min(a.cp.L[2], je) - j0, 0), ys = max(a.cp.L[3] ? a.cp.start[3] : a.ny, j0);
    const int z0n = max(min((a.cp.L[4] + 3) / 4, qe) - q0, 0), zs = max(a.cp.L[5] ? a.cp.zbase[1] / 4 : a.nzq, max(q0, q0 + z0n));
    const int ny = y0 + max(je - ys, 0), nz = z0n + max(qe - zs, 0);
    c.iy = (c.fy == 2 ? r : y0 + c.j - ys) * wz + cc;
    c.iz = ny * wz + (c.fz == 4 ? cc : z0n + q - zs) * B.ty + r;
    c.ix = ny * wz + nz * B.ty + t;
  }
  const int tp = min(t + wz, nt - 1), tm = max(t - wz, 0);  // y-neighbours' slots
  const bool edge_p = lane == 31 && t + 1 < nt, edge_m = lane == 0 && t > 0;
  const bool last_k = c.k0 + 4 >= a.nz;  // the chunk holds the last cell of the row
  // element offset in a plane; what is added to it is the same for the warp
  const unsigned off = c.in ? (unsigned)(c.j * a.nzp + c.k0) : 0u;
  const int key = c.in ? c.j * a.nzq + q : -1;
  const uint32_t sE = (uint32_t)__cvta_generic_to_shared(ringE + t), sH = (uint32_t)__cvta_generic_to_shared(ringH + t);
  const T* in = static_cast<const T*>(a.in);
  T* out = static_cast<T*>(a.out);
  const long long step0 = (a.nsrc ? *a.d_base : 0) + a.local;

  auto copy_plane = [&](uint32_t dst, int p, int comp0, int slot) {
    const T* s = in + (comp0 * a.comp + min(p, a.nx - 1) * a.plane);
    const bool on = c.in && p < a.nx;
#pragma unroll
    for (int m = 0; m < 3; ++m)
      CIO::copy(dst + (uint32_t)((slot * 3 + m) * nt * sizeof(Raw)), s + m * a.comp + off, on);
  };
  const uint32_t sI = (uint32_t)__cvta_generic_to_shared(ringI + t * 4 * kIdBytes);
  auto copy_ids = [&](int p, int slot) {
    const char* s = static_cast<const char*>(a.ids) + (min(p, a.nx - 1) * a.plane + off) * kIdBytes;
    const int n = c.in && p < a.nx ? 4 * kIdBytes : 0;
    const uint32_t dst = sI + slot * 4 * kIdBytes * nt;
    if constexpr (kIdBytes == 1)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(s), "r"(n) : "memory");
    else
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(s), "r"(n) : "memory");
  };
  const int ia = max(i0 - kSteps, 0);
  const int ib = kSteps == 2 ? i1 : i1 - 1;
  copy_plane(sE, ia, 0, 0);
  copy_plane(sE, ia + 1, 0, 1);
  copy_ids(ia, 0);
  copy_ids(ia + 1, 1);
  copy_plane(sH, ia, 3, 0);
  if constexpr (kCpml) {
    PsiH::load(a, c, psi, ia);
    PsiE::load(a, c, psi, ia);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  if constexpr (!kCpml) {
    copy_plane(sE, ia + 2, 0, 2);
    copy_ids(ia + 2, 2);
    copy_plane(sH, ia + 1, 3, 1);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  uint32_t w0 = 0, w1 = 0, v0 = 0, v1 = 0;  // ids of planes i and i - 1
  // what a step needs of the plane before: in registers, or (kLean: the CPML
  // form has none to spare) the y components only, the others read again from
  // the exchange buffers
  constexpr bool kLean = kCpml;
  float hy1p[4], ey1p[4], hy2p[4], hx1p[4], hz1p[4], ex1p[4], ez1p[4], hz2p[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) hy1p[e] = ey1p[e] = hy2p[e] = hx1p[e] = hz1p[e] = ex1p[e] = ez1p[e] = hz2p[e] = 0.f;
  asm volatile("cp.async.wait_group 1;" ::: "memory");
  __syncthreads();

  int se = 0, sh = 0;  // ring slots of plane i
  for (int i = ia; i <= ib; ++i) {
    // all but the newest group: E of planes <= i + 1, H (and psi of H) of
    // plane i; the neighbours' part of E(i) was waited for an iteration (and
    // a barrier) ago
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    const int se1 = se == kRingE - 1 ? 0 : se + 1;
    const int par = i & 1;
    float h1[3][4], e1[3][4];
    const bool go = i < a.nx;
    float4* x1i = x1 + par * 2 * nt;
    const float4* x1p = x1 + (par ^ 1) * 2 * nt;
    const bool own1 = c.own && i >= i0;  // (one-step passes)
    if (go) {
      // ---- A: H(n+1/2) of plane i
      const uint32_t* id = reinterpret_cast<const uint32_t*>(ringI + (se * nt + t) * 4 * kIdBytes);
      w0 = id[0];
      if constexpr (kIdBytes == 2) w1 = id[1];
      const Raw* E0 = ringE + se * 3 * nt;
      const Raw* En = ringE + se1 * 3 * nt;
      const Raw* H0 = ringH + sh * 3 * nt;
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        CIO::unpack(H0[m * nt + t], h1[m]);
        CIO::unpack(E0[m * nt + t], e1[m]);
      }
      float exn = __shfl_down_sync(kFullMask, e1[0][0], 1);
      float eyn = __shfl_down_sync(kFullMask, e1[1][0], 1);
      if (edge_p) {
        float v[4];
        CIO::unpack(E0[t + 1], v);
        exn = v[0];
        CIO::unpack(E0[nt + t + 1], v);
        eyn = v[0];
      }
      float d[6][4], f[4];
      CIO::unpack(E0[2 * nt + tp], f);
#pragma unroll
      for (int e = 0; e < 4; ++e) d[0][e] = __fsub_rn(f[e], e1[2][e]);
      CIO::unpack(E0[tp], f);
#pragma unroll
      for (int e = 0; e < 4; ++e) d[5][e] = __fsub_rn(f[e], e1[0][e]);
      if (!c.jp) {
#pragma unroll
        for (int e = 0; e < 4; ++e) d[0][e] = d[5][e] = 0.f;
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        d[1][e] = __fsub_rn(e < 3 ? e1[1][e < 3 ? e + 1 : 3] : eyn, e1[1][e]);
        d[2][e] = __fsub_rn(e < 3 ? e1[0][e < 3 ? e + 1 : 3] : exn, e1[0][e]);
      }
      if (last_k) {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (c.k0 + e + 1 >= a.nz) d[1][e] = d[2][e] = 0.f;
      }
      if (i + 1 < a.nx) {
        CIO::unpack(En[2 * nt + t], f);
#pragma unroll
        for (int e = 0; e < 4; ++e) d[3][e] = __fsub_rn(f[e], e1[2][e]);
        CIO::unpack(En[nt + t], f);
#pragma unroll
        for (int e = 0; e < 4; ++e) d[4][e] = __fsub_rn(f[e], e1[1][e]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) d[3][e] = d[4][e] = 0.f;
      }
      if constexpr (kCpml) PsiH::template apply<kSteps == 1>(a, prof, psi, c, i, own1, d, c.live_h);
      fused_apply<kIdBytes, true, kCpml>(tab, w0, w1, d, c.live_h, h1);
#pragma unroll
      for (int m = 0; m < 3; ++m) CIO::round(h1[m]);
      x1i[t] = to_f4(h1[0]);
      x1i[nt + t] = to_f4(h1[2]);
      if (lane == 31) edge[par * kEdge + warp] = h1[1][3];
      copy_plane(sH, i + kRingH, 3, sh);
      if constexpr (kCpml && kSteps == 1) PsiH::load(a, c, psi, i + 1);
    }
    __syncthreads();
    if (go) {
      // ---- B: E(n+1) of plane i
      float d[6][4], f[4];
      float hxm = __shfl_up_sync(kFullMask, h1[0][3], 1);
      float hym = __shfl_up_sync(kFullMask, h1[1][3], 1);
      if (edge_m) {
        hxm = x1i[t - 1].w;
        hym = edge[par * kEdge + warp - 1];
      }
      if constexpr (kLean) to_arr(x1p[nt + t], hz1p);
      to_arr(x1i[nt + tm], f);
#pragma unroll
      for (int e = 0; e < 4; ++e) d[0][e] = __fsub_rn(h1[2][e], f[e]);
      to_arr(x1i[tm], f);
#pragma unroll
      for (int e = 0; e < 4; ++e) d[5][e] = __fsub_rn(h1[0][e], f[e]);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        d[1][e] = __fsub_rn(h1[1][e], e ? h1[1][e ? e - 1 : 0] : hym);
        d[2][e] = __fsub_rn(h1[0][e], e ? h1[0][e ? e - 1 : 0] : hxm);
        d[3][e] = __fsub_rn(h1[2][e], hz1p[e]);
        d[4][e] = __fsub_rn(h1[1][e], hy1p[e]);
      }
      const unsigned live = i >= 1 ? c.live_e : 0u;
      if constexpr (kCpml) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");  // psi of E
        PsiE::template apply<kSteps == 1>(a, prof, psi, c, i, own1, d, live);
      }
      fused_apply<kIdBytes, false, kCpml>(tab, w0, w1, d, live, e1);
#pragma unroll
      for (int m = 0; m < 3; ++m) CIO::round(e1[m]);
      if (fused_any(a.src_off, a.src_lo, a.src_hi, i)) with_copy(e1, [&](float* e) { fused_sources<T>(a, i, key, step0, e); });
      if (c.own && i >= i0 && i < i1 && fused_any(a.tap_off, a.tap_lo, a.tap_hi, i))
        with_copy(e1, [&](float* e) { with_copy(h1, [&](float* h) { fused_taps(a, i, key, a.local, e, h); }); });
      if constexpr (kSteps == 1) {
        if (c.own && i >= i0) {
          T* o = out + i * a.plane;
#pragma unroll
          for (int m = 0; m < 3; ++m) {
            FieldIO<T>::st4(reinterpret_cast<float*>(o + m * a.comp), off, to_f4(e1[m]));
            FieldIO<T>::st4(reinterpret_cast<float*>(o + (3 + m) * a.comp), off, to_f4(h1[m]));
          }
        }
      }
    }
    copy_plane(sE, i + kRingE, 0, se);
    copy_ids(i + kRingE, se);
    if constexpr (!kCpml || kSteps == 1) asm volatile("cp.async.commit_group;" ::: "memory");
    if constexpr (kCpml && kSteps == 1) {
      PsiE::load(a, c, psi, i + 1);
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    if constexpr (kSteps == 2) {
      // ---- C: H(n+3/2) of plane i - 1
      const int p = i - 1;
      const bool run_c = p >= ia && p >= i0 - 1;
      float h2[3][4];
      float4* x2o = x2 + (par ^ 1) * 2 * nt;
      float4* x2n = x2 + par * 2 * nt;
      float* edge2o = edge + (2 + (par ^ 1)) * kEdge;
      if (run_c) {
        float d[6][4], f[4], e1p[3][4];
        if constexpr (kLean) {
          to_arr(x2o[t], ex1p);
          to_arr(x2o[nt + t], ez1p);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          e1p[0][e] = ex1p[e];
          e1p[1][e] = ey1p[e];
          e1p[2][e] = ez1p[e];
        }
        float exn = __shfl_down_sync(kFullMask, e1p[0][0], 1);
        float eyn = __shfl_down_sync(kFullMask, e1p[1][0], 1);
        if (edge_p) {
          exn = x2o[t + 1].x;
          eyn = edge2o[warp + 1];
        }
        to_arr(x2o[nt + tp], f);
#pragma unroll
        for (int e = 0; e < 4; ++e) d[0][e] = __fsub_rn(f[e], e1p[2][e]);
        to_arr(x2o[tp], f);
#pragma unroll
        for (int e = 0; e < 4; ++e) d[5][e] = __fsub_rn(f[e], e1p[0][e]);
        if (!c.jp) {
#pragma unroll
          for (int e = 0; e < 4; ++e) d[0][e] = d[5][e] = 0.f;
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          d[1][e] = __fsub_rn(e < 3 ? e1p[1][e < 3 ? e + 1 : 3] : eyn, e1p[1][e]);
          d[2][e] = __fsub_rn(e < 3 ? e1p[0][e < 3 ? e + 1 : 3] : exn, e1p[0][e]);
        }
        if (last_k) {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (c.k0 + e + 1 >= a.nz) d[1][e] = d[2][e] = 0.f;
        }
        if (go) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            d[3][e] = __fsub_rn(e1[2][e], e1p[2][e]);
            d[4][e] = __fsub_rn(e1[1][e], e1p[1][e]);
          }
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) d[3][e] = d[4][e] = 0.f;
        }
        if constexpr (kCpml) PsiH::template apply<true>(a, prof, psi, c, p, c.own && p >= i0, d, c.live_h);
        if constexpr (kLean) {
          to_arr(x1p[t], hx1p);
          to_arr(x1p[nt + t], hz1p);
          to_arr(x3[nt + t], hz2p);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          h2[0][e] = hx1p[e];
          h2[1][e] = hy1p[e];
          h2[2][e] = hz1p[e];
        }
        fused_apply<kIdBytes, true, kCpml>(tab, v0, v1, d, c.live_h, h2);
#pragma unroll
        for (int m = 0; m < 3; ++m) CIO::round(h2[m]);
        x3[t] = to_f4(h2[0]);
        x3[nt + t] = to_f4(h2[2]);
        if (lane == 31) edge[4 * kEdge + warp] = h2[1][3];
      }
      if constexpr (kCpml) {
        PsiH::load(a, c, psi, i + 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
      }
      if (go) {
        x2n[t] = to_f4(e1[0]);
        x2n[nt + t] = to_f4(e1[2]);
        if (lane == 0) edge[(2 + par) * kEdge + warp] = e1[1][0];
      }
      __syncthreads();
      // ---- D: E(n+2) of plane i - 1
      if (p >= i0) {
        float d[6][4], f[4], e2[3][4];
        if constexpr (kLean) {
          to_arr(x2o[t], ex1p);
          to_arr(x2o[nt + t], ez1p);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          e2[0][e] = ex1p[e];
          e2[1][e] = ey1p[e];
          e2[2][e] = ez1p[e];
        }
        float hxm = __shfl_up_sync(kFullMask, h2[0][3], 1);
        float hym = __shfl_up_sync(kFullMask, h2[1][3], 1);
        if (edge_m) {
          hxm = x3[t - 1].w;
          hym = edge[4 * kEdge + warp - 1];
        }
        to_arr(x3[nt + tm], f);
#pragma unroll
        for (int e = 0; e < 4; ++e) d[0][e] = __fsub_rn(h2[2][e], f[e]);
        to_arr(x3[tm], f);
#pragma unroll
        for (int e = 0; e < 4; ++e) d[5][e] = __fsub_rn(h2[0][e], f[e]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          d[1][e] = __fsub_rn(h2[1][e], e ? h2[1][e ? e - 1 : 0] : hym);
          d[2][e] = __fsub_rn(h2[0][e], e ? h2[0][e ? e - 1 : 0] : hxm);
          d[3][e] = __fsub_rn(h2[2][e], hz2p[e]);
          d[4][e] = __fsub_rn(h2[1][e], hy2p[e]);
        }
        const unsigned live = p >= 1 ? c.live_e : 0u;
        if constexpr (kCpml) PsiE::template apply<true>(a, prof, psi, c, p, c.own, d, live);
        fused_apply<kIdBytes, false, kCpml>(tab, v0, v1, d, live, e2);
#pragma unroll
        for (int m = 0; m < 3; ++m) CIO::round(e2[m]);
        if (fused_any(a.src_off, a.src_lo, a.src_hi, p)) with_copy(e2, [&](float* e) { fused_sources<T>(a, p, key, step0 + 1, e); });
        if (c.own && fused_any(a.tap_off, a.tap_lo, a.tap_hi, p))
          with_copy(e2, [&](float* e) { with_copy(h2, [&](float* h) { fused_taps(a, p, key, a.local + 1, e, h); }); });
        if (c.own) {
          T* o = out + p * a.plane;
#pragma unroll
          for (int m = 0; m < 3; ++m) {
            FieldIO<T>::st4(reinterpret_cast<float*>(o + m * a.comp), off, to_f4(e2[m]));
            FieldIO<T>::st4(reinterpret_cast<float*>(o + (3 + m) * a.comp), off, to_f4(h2[m]));
          }
        }
      }
      if constexpr (kCpml) {
        PsiE::load(a, c, psi, i + 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        hy2p[e] = h2[1][e];
        ey1p[e] = e1[1][e];
        if constexpr (!kLean) {
          hz2p[e] = h2[2][e];
          ex1p[e] = e1[0][e];
          ez1p[e] = e1[2][e];
        }
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      hy1p[e] = h1[1][e];
      if constexpr (!kLean) {
        hx1p[e] = h1[0][e];
        hz1p[e] = h1[2][e];
      }
    }
    v0 = w0;
    v1 = w1;
    se = se1;
    sh = sh == kRingH - 1 ? 0 : sh + 1;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// The table (1-byte ids) and the CPML profiles behind the exchange buffers.
template <int kSteps, int kIdBytes, bool kCpml, typename T>
__device__ __forceinline__ void fused_stage(const FusedArgs& a, char* smem, const float*& tab, const float*& prof) {
  const int nt = blockDim.x;
  float* p = reinterpret_cast<float*>(smem + fused_smem(kSteps, kCpml, nt, sizeof(T), kIdBytes, 0, 0, kCpml ? a.pairs : 0));
  tab = a.table;
  if constexpr (kIdBytes == 1) {
    for (int t = threadIdx.x; t < a.ntable * 12; t += nt) p[t] = __ldg(a.table + t);
    tab = p;
    p += (a.ntable * 12 + 3) & ~3;
  }
  prof = p;
  if constexpr (kCpml) {
    // z profiles by the psi row's cell (0 outside the slab), so a chunk's four are one load
    for (int f = 0; f < 6; ++f) {
      const int L = a.cp.L[f], w = f < 4 ? L : a.cp.zw[f - 4], o = f < 4 ? 0 : a.cp.zbase[f - 4] - a.cp.start[f];
      for (int t = threadIdx.x; t < 6 * w; t += nt) {
        const int r = t / w, l = t - r * w + o;
        p[a.poff[f] + t] = l >= 0 && l < L ? __ldg(a.cp.prof + a.cp.prof_off[f] + r * L + l) : 0.f;
      }
    }
  }
  __syncthreads();
}

// A CTA per work item; the boxes with the longest items come first.  The
// boxes that meet no slab and those that do are separate launches.
template <int kSteps, int kIdBytes, bool kCpml, typename T>
__global__ void __launch_bounds__(kFusedMaxThreads, 1) k_fused(const __grid_constant__ FusedArgs a) {
  extern __shared__ __align__(16) char fused_mem[];
  const float *tab, *prof;
  // the next pass may take this one's place on an SM as CTAs end; its own
  // wait below keeps it from the fields until all of them have
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  fused_stage<kSteps, kIdBytes, kCpml, T>(a, fused_mem, tab, prof);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  int b = 0;
  while (b + 1 < a.nbox && (int)blockIdx.x >= a.box[b + 1].item0) ++b;
  const FusedBox& B = a.box[b];
  const int w = blockIdx.x - B.item0;
  if constexpr (!kCpml) {
    fused_item<kSteps, kIdBytes, 0, T>(a, B, w, fused_mem, tab, prof);
  } else {
    if (B.axes == 4)
      fused_item<kSteps, kIdBytes, 4, T>(a, B, w, fused_mem, tab, prof);
    else if (B.axes == 6)
      fused_item<kSteps, kIdBytes, 6, T>(a, B, w, fused_mem, tab, prof);
    else
      fused_item<kSteps, kIdBytes, 7, T>(a, B, w, fused_mem, tab, prof);
  }
}

// Probe values of a span's steps from its taps (the sums of k_post_step).
struct ProbeSumArgs {
  int nprobe, ntap, steps;
  const int* probe_off;
  const int* probe_mode;
  const double* term_w;
  const float* taps;
  double* traces;  // [batch step][probe]
  const long long* d_base;
};

__global__ void k_probe_sums(const ProbeSumArgs a) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)a.steps * a.nprobe) return;
  const long long s = t / a.nprobe;
  const int p = (int)(t - s * a.nprobe);
  const float* v = a.taps + s * a.ntap;
  double val;
  if (a.probe_mode[p] == 0) {
    float acc = 0.0f;
    for (int x = a.probe_off[p]; x < a.probe_off[p + 1]; ++x)
      acc = a.term_w[x] >= 0.0 ? __fadd_rn(acc, v[x]) : __fsub_rn(acc, v[x]);
    val = (double)acc;
  } else {
    double acc = 0.0;
    for (int x = a.probe_off[p]; x < a.probe_off[p + 1]; ++x) acc = __dadd_rn(acc, __dmul_rn(a.term_w[x], (double)v[x]));
    val = acc;
  }
  a.traces[(*a.d_base + s) * a.nprobe + p] = val;
}

// ---- distinct coefficient sets ------------------------------------------
// An open-addressing table of 64-bit hashes; each slot keeps the lowest cell
// that hashed to it, whose 12 coefficients stand for the set.  k_coef_ids
// compares every cell's bits with its set's, so two sets with one hash are
// noticed (and the grid then keeps its full arrays).
constexpr int kCoefSlots = 1 << 18;
constexpr int kCoefMax = 65536;

struct CoefArgs {
  const float* c;  // [12][comp]
  long long comp;
  int nz, nzp;
  long long rows;
  unsigned long long* key;  // [kCoefSlots], 0 = empty
  long long* rep;           // [kCoefSlots]
  int* list;                // occupied slots
  int* count;               // [0] occupied slots, [1] failures
  const int* id_of;         // [kCoefSlots]
  void* ids;
  int id_bytes;
};

__device__ __forceinline__ unsigned long long coef_hash(const float* c, long long comp, long long q) {
  unsigned long long h = 0x9e3779b97f4a7c15ull;
#pragma unroll
  for (int a = 0; a < 12; ++a) {
    h ^= (unsigned long long)__float_as_uint(__ldg(c + a * comp + q));
    h *= 0xff51afd7ed558ccdull;
    h ^= h >> 32;
  }
  return h ? h : 1;
}

__global__ void k_coef_sets(const CoefArgs a) {
  const long long n = a.rows * a.nz;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
    if (*(volatile int*)(a.count + 1)) return;
    const long long row = t / a.nz, q = row * a.nzp + (t - row * a.nz);
    const unsigned long long h = coef_hash(a.c, a.comp, q);
    unsigned s = (unsigned)(h >> 20) & (kCoefSlots - 1);
    for (int probe = 0;; ++probe) {
      unsigned long long k = *(volatile unsigned long long*)(a.key + s);
      if (k == 0) {
        k = atomicCAS(a.key + s, 0ull, h);
        if (k == 0) {
          const int m = atomicAdd(a.count, 1);
          if (m < kCoefMax)
            a.list[m] = (int)s;
          else
            atomicExch(a.count + 1, 1);
          k = h;
        }
      }
      if (k == h) break;
      if (probe >= 1024) {
        atomicExch(a.count + 1, 1);
        return;
      }
      s = (s + 1) & (kCoefSlots - 1);
    }
    if (q < *(volatile long long*)(a.rep + s)) atomicMin(a.rep + s, q);
  }
}

__global__ void k_coef_ids(const CoefArgs a) {
  const long long n = a.rows * a.nz;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
    const long long row = t / a.nz, q = row * a.nzp + (t - row * a.nz);
    const unsigned long long h = coef_hash(a.c, a.comp, q);
    unsigned s = (unsigned)(h >> 20) & (kCoefSlots - 1);
    for (int probe = 0; probe <= 1024 && a.key[s] != h; ++probe) s = (s + 1) & (kCoefSlots - 1);
    const long long r = a.rep[s];
    bool same = a.key[s] == h;
#pragma unroll
    for (int c = 0; c < 12; ++c)
      same = same && __float_as_uint(__ldg(a.c + c * a.comp + q)) == __float_as_uint(__ldg(a.c + c * a.comp + r));
    if (!same) atomicExch(a.count + 1, 1);
    const int id = a.id_of[s];
    if (a.id_bytes == 1)
      static_cast<uint8_t*>(a.ids)[q] = (uint8_t)id;
    else
      static_cast<uint16_t*>(a.ids)[q] = (uint16_t)id;
  }
}

// First cell of each occupied slot; ids of the slots in their final order.
__global__ void k_coef_first(const int* list, const long long* rep, int n, long long* first) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) first[t] = rep[list[t]];
}
__global__ void k_coef_number(const int* list, int n, int* id_of) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) id_of[list[t]] = t;
}

// table[id] = the coefficients of cell reps[id].
__global__ void k_coef_table(const float* c, long long comp, const long long* reps, int n, float* table) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n * 12) table[t] = c[(t % 12) * comp + reps[t / 12]];
}

}  // namespace oems
