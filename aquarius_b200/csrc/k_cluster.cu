// The whole pressure solve of one scene in one thread-block cluster: every
// sweep and residual check runs on chip, with the iterate in the cluster's
// shared memory.
//
// Arithmetic: jacobiImpl (Fluid/Fluid_3D_kernels.cu:460-505) in the race-free
// reading of k_jacobi.cu, cell for cell the same operations in the same order
// (x+1, x-1, y+1, y-1, z+1, z-1, rhs, divided by 6), so every iterate equals
// the other plans' bit for bit.
//
// What bounds small grids: a sweep of a few thousand to a hundred thousand
// fluid cells is microseconds of latency per launch and almost no work.  One
// sweep per launch takes 1.6 us at 16^3 (row list) and 6.1 us at 50^3 (tiled
// kernel, z not a multiple of 4); a cluster barrier with a read of another
// CTA's shared memory takes 0.4 us at 16 CTAs (0.05 us at one CTA).  Measured
// here, a sweep: 16^3 0.39 us (one CTA), 50^3 with 27k fluid cells 0.80 us,
// 64^3 with 111k 1.50 us (row list 2.05), 90x61x75 with 132k 2.10 us (tiled
// 6.2).  What bounds it now is the latency of a unit's dependent instructions
// (few warps per scheduler) and the barrier.
//
// Layout: the unknowns are units of 2 x 1 x 4 cells (two z-quads, A and B, at
// x and x+1) that hold fluid, in the order of their (x, y, z), numbered by a
// scan over the cluster.  CTA r owns the r-th equal share, so the load is even
// whatever the shape of the fluid.  A share's pressures lie in two
// shared-memory buffers (read one, write the other: one cluster barrier per
// sweep); a thread owns up to kU units, with their rhs, fluid marks and the
// addresses of their neighbours in registers.  Shared memory carries 36
// clocks of a unit's 8 cells per warp (16-byte rows, against 52 for two
// separate quads), the FP32 pipe about as much: the sums of a pair of cells
// are one packed add.  Neighbours in another CTA are read through distributed
// shared memory, units without fluid are one zero unit, and a wall (Neumann)
// is an address inside the unit itself.  Sides need not be even or multiples
// of 4: cells of a unit beyond the wall carry copies of the last cell inside,
// which are exactly the clamped neighbours the wall asks for.
//
// FP64 residuals are summed per 32 consecutive units, then over those partial
// sums in index order, so a solve's decisions do not depend on the cluster
// size (a scene in a batch stops where it stops alone).
//
// A fluid may spread over more units than the cluster's shared memory holds (a
// droplet occupies a whole unit).  The cluster then leaves the system as it is
// and sets a mark, from which a graph condition runs the solve's other branch, the
// sweeps over the whole machine.
#include <algorithm>
#include <type_traits>

#include "aq_kernels.cuh"

namespace aqb {
namespace {

constexpr int kT = 512;                    // threads per CTA
constexpr int kU = 4;                      // units per thread
constexpr int kCap = 2048;                 // units per CTA (a multiple of 32): 16 CTAs hold any 64^3 fluid
constexpr int kZero = kCap;                // the zero unit of a buffer
constexpr int kSlots = kCap + 16;          // units per buffer
constexpr int kHalf = kSlots * 16;         // bytes from quad A to quad B
constexpr int kBufBytes = 2 * kHalf;
constexpr int kSmem = 2 * kBufBytes;
constexpr int kScanBits = 32;              // scan passes a thread remembers as one bit each
constexpr int kSmallUnits = 1024;          // grids up to this many units (fluid or not) take one CTA
static_assert(kCap <= kT * kU && kCap % 32 == 0, "a CTA's share must fit its threads");

struct ClusterScene {
  Dims d;
  float* pa;
  const float* rhs;
  const int8_t* type;
  int *umap, *list;  // unit -> index among the fluid units (-1: none), and back
  double* part;      // residual partials, one per 32 fluid units
  SolveState* ss;
};

struct SolveArgs {
  int fixed_sweeps, check, max_iters;  // fixed_sweeps 0: residual mode
  double tol;
  double* r2_only;  // if set: where ||b - A p||^2 goes, and the solve state stays as it is
  int* spilled;     // set to 1 where the fluid's units do not fit (null: they always do)
};

// What every thread of the cluster knows of the running solve.
struct Solve {
  unsigned me, nr;  // CTA and cluster size
  int n, per;       // fluid units, and of them to a CTA
  double b2;
  int it0;
  int done, checks;
  double r2, rel;
};

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cluster_size() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// Orders the cluster's shared and global memory accesses across it.
__device__ __forceinline__ void cluster_sync(unsigned nr) {
  if (nr == 1) {
    __syncthreads();
    return;
  }
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned mapa(unsigned addr, unsigned rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}

// Four cells along z as two packed pairs.
struct Quad {
  u64 lo, hi;
};
__device__ __forceinline__ Quad pack4(const float4& v) { return {pack2(v.x, v.y), pack2(v.z, v.w)}; }
__device__ __forceinline__ float4 unpack4(const Quad& q) {
  const float2 a = unpack2(q.lo), b = unpack2(q.hi);
  return make_float4(a.x, a.y, b.x, b.y);
}
// Loads and stores at an address of buffer 0, OFF bytes on.  They are
// volatile, so they keep their place between the barriers; no other access
// touches the buffers.
template <int OFF, bool FAR>
__device__ __forceinline__ Quad ld4(unsigned a) {
  Quad v;
  if (FAR)
    asm volatile("ld.shared::cluster.v2.b64 {%0,%1}, [%2+%3];" : "=l"(v.lo), "=l"(v.hi) : "r"(a), "n"(OFF));
  else
    asm volatile("ld.shared.v2.b64 {%0,%1}, [%2+%3];" : "=l"(v.lo), "=l"(v.hi) : "r"(a), "n"(OFF));
  return v;
}
template <int OFF, bool FAR>
__device__ __forceinline__ float ld1(unsigned a) {
  float v;
  if (FAR)
    asm volatile("ld.shared::cluster.f32 %0, [%1+%2];" : "=f"(v) : "r"(a), "n"(OFF));
  else
    asm volatile("ld.shared.f32 %0, [%1+%2];" : "=f"(v) : "r"(a), "n"(OFF));
  return v;
}
template <int OFF>
__device__ __forceinline__ void st4(unsigned a, const Quad& v) {
  asm volatile("st.shared.v2.b64 [%0+%3], {%1,%2};" ::"r"(a), "l"(v.lo), "l"(v.hi), "n"(OFF));
}

// Flags of a unit: bits 0-3 the fluid cells of quad A, 4-7 of quad B.
constexpr unsigned kCopyB = 1u << 8;     // B is beyond the wall: a copy of A
constexpr unsigned kLenShift = 9;        // 2 bits: cells of a short last quad, 0 all four
constexpr unsigned kFarX = 1u << 11;     // x - 1 or x + 2 is in another CTA
constexpr unsigned kFarYZ = 1u << 12;    // a y or z neighbour is
constexpr unsigned kValid = 1u << 13;

// Addresses in buffer 0 of a unit's neighbours: quad B of the unit at x - 1,
// quad A of the one at x + 2, quads A of y + 1 and y - 1 (B is kHalf on), and
// the single values of z + 4 and z - 1 beside quad A.  The two x addresses are
// shared::cluster ones when one of them is in another CTA, and so are the
// four y and z addresses; otherwise they are plain shared addresses.
struct Near {
  unsigned xm, xp, yp, ym, zh, zl;
};

struct UnitIn {
  Quad a, b;  // the unit itself
  Quad xm, xp, ypa, yma, ypb, ymb;
  float zha, zla, zhb, zlb;
};

template <int BUF, bool FAR>
__device__ __forceinline__ void load_x(UnitIn& u, const Near& at) {
  constexpr int O = BUF * kBufBytes;
  u.xp = ld4<O, FAR>(at.xp);
  u.xm = ld4<O, FAR>(at.xm);
}
template <int BUF, bool FAR>
__device__ __forceinline__ void load_yz(UnitIn& u, const Near& at) {
  constexpr int O = BUF * kBufBytes;
  u.ypa = ld4<O, FAR>(at.yp);
  u.yma = ld4<O, FAR>(at.ym);
  u.ypb = ld4<O + kHalf, FAR>(at.yp);
  u.ymb = ld4<O + kHalf, FAR>(at.ym);
  u.zha = ld1<O, FAR>(at.zh);
  u.zla = ld1<O, FAR>(at.zl);
  u.zhb = ld1<O + kHalf, FAR>(at.zh);
  u.zlb = ld1<O + kHalf, FAR>(at.zl);
}
template <int BUF>
__device__ __forceinline__ void load_unit(UnitIn& u, const Near& at, unsigned fl) {
  if (!(fl & kFarX)) load_x<BUF, false>(u, at);
  else load_x<BUF, true>(u, at);
  if (!(fl & kFarYZ)) load_yz<BUF, false>(u, at);
  else load_yz<BUF, true>(u, at);
}

constexpr float kSixth = 0x1.555556p-3f;  // RN(1/6)

// 1/6 where bit k of the fluid marks is set, else 0.
__device__ __forceinline__ Quad sixths(unsigned marks) {
  return pack4(make_float4(marks & 1u ? kSixth : 0.f, marks & 2u ? kSixth : 0.f, marks & 4u ? kSixth : 0.f,
                           marks & 8u ? kSixth : 0.f));
}

// The seven-term sums of a quad in the reference's order.
__device__ __forceinline__ Quad sum_quad(const Quad& xp, const Quad& xm, const Quad& yp, const Quad& ym, const Quad& c,
                                         float zh, float zl, const Quad& rhs) {
  u64 lo = add2(xp.lo, xm.lo), hi = add2(xp.hi, xm.hi);
  lo = add2(lo, yp.lo);
  hi = add2(hi, yp.hi);
  lo = add2(lo, ym.lo);
  hi = add2(hi, ym.hi);
  const float2 c0 = unpack2(c.lo), c1 = unpack2(c.hi);
  float2 s0 = unpack2(lo), s1 = unpack2(hi);
  s0.x += c0.y; s0.y += c1.x; s1.x += c1.y; s1.y += zh;
  s0.x += zl;   s0.y += c0.x; s1.x += c0.y; s1.y += c1.x;
  return {add2(pack2(s0.x, s0.y), rhs.lo), add2(pack2(s1.x, s1.y), rhs.hi)};
}
// One Jacobi update of a quad.  s / 6 is the corrected reciprocal product
// (Markstein's; aq_selfcheck_division compares it with the IEEE divide over
// all floats): exact for 0 and for finite |s| >= 2^-123, other sums divide.
// r is 1/6 on fluid cells and 0 elsewhere, which makes the quotient of a
// finite sum 0 there.  The sign of a zero may be another one than the divide's
// (packed operands cannot be negated for nothing): a sum with a nonzero term
// does not see it, and the solve's end stores zeros as +0.
__device__ __forceinline__ Quad update_quad(const Quad& xp, const Quad& xm, const Quad& yp, const Quad& ym,
                                            const Quad& c, float zh, float zl, const Quad& rhs, const Quad& r) {
  const Quad s = sum_quad(xp, xm, yp, ym, c, zh, zl, rhs);
  const float4 v = unpack4(s);
  // 2 bits - 1 orders magnitudes, with 0 above all of them; the total is
  // finite only if all four sums are
  const unsigned k0 = 2u * __float_as_uint(v.x) - 1u, k1 = 2u * __float_as_uint(v.y) - 1u;
  const unsigned k2 = 2u * __float_as_uint(v.z) - 1u, k3 = 2u * __float_as_uint(v.w) - 1u;
  const float2 t = unpack2(add2(s.lo, s.hi));
  if (min(min(k0, k1), min(k2, k3)) >= 0x07ffffffu && fabsf(t.x + t.y) <= 3.402823466e38f) {  // 2 bits(2^-123) - 1
    const u64 m6 = pack2(-6.f, -6.f);
    const u64 q0 = mul2(s.lo, r.lo), q1 = mul2(s.hi, r.hi);
    return {fma2(fma2(q0, m6, s.lo), r.lo, q0), fma2(fma2(q1, m6, s.hi), r.hi, q1)};
  }
  const float4 m = unpack4(r);
  return pack4(make_float4(m.x != 0.f ? __fdiv_rn(v.x, 6.f) : 0.f, m.y != 0.f ? __fdiv_rn(v.y, 6.f) : 0.f,
                           m.z != 0.f ? __fdiv_rn(v.z, 6.f) : 0.f, m.w != 0.f ? __fdiv_rn(v.w, 6.f) : 0.f));
}

// One Jacobi update of a unit's quads into u.a and u.b.
__device__ __forceinline__ void update_unit(UnitIn& u, const Quad& rha, const Quad& rhb, const Quad& ra,
                                            const Quad& rb) {
  const Quad a = update_quad(u.b, u.xm, u.ypa, u.yma, u.a, u.zha, u.zla, rha, ra);
  u.b = update_quad(u.xp, u.a, u.ypb, u.ymb, u.b, u.zhb, u.zlb, rhb, rb);
  u.a = a;
}

// Cells beyond the row's end copy the last one inside.
__device__ __forceinline__ Quad copy_tail(const Quad& q, unsigned len) {
  float4 v = unpack4(q);
  if (len < 2u) v.y = v.x;
  if (len < 3u) v.z = v.y;
  v.w = v.z;
  return pack4(v);
}

// (b - A p)^2 summed over a quad's fluid cells, in FP64 (as resid_row).
__device__ __forceinline__ double resid_quad(const Quad& xpq, const Quad& xmq, const Quad& ypq, const Quad& ymq,
                                             const Quad& cq, float zh, float zl, const Quad& rhs, unsigned marks) {
  const float4 xpv = unpack4(xpq), xmv = unpack4(xmq), ypv = unpack4(ypq), ymv = unpack4(ymq), cv = unpack4(cq),
               bv = unpack4(rhs);
  const float c[4] = {cv.x, cv.y, cv.z, cv.w};
  const float zp[4] = {cv.y, cv.z, cv.w, zh}, zm[4] = {zl, cv.x, cv.y, cv.z};
  const float xp[4] = {xpv.x, xpv.y, xpv.z, xpv.w}, xm[4] = {xmv.x, xmv.y, xmv.z, xmv.w};
  const float yp[4] = {ypv.x, ypv.y, ypv.z, ypv.w}, ym[4] = {ymv.x, ymv.y, ymv.z, ymv.w};
  const float rb[4] = {bv.x, bv.y, bv.z, bv.w};
  double acc = 0.0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (!((marks >> k) & 1u)) continue;
    double s = (double)xp[k];
    s += (double)xm[k];
    s += (double)yp[k];
    s += (double)ym[k];
    s += (double)zp[k];
    s += (double)zm[k];
    const double r = (double)rb[k] + s - 6.0 * (double)c[k];
    acc += r * r;
  }
  return acc;
}
__device__ __forceinline__ double resid_unit(const UnitIn& u, const Quad& ra, const Quad& rb, unsigned fl) {
  const double a = resid_quad(u.b, u.xm, u.ypa, u.yma, u.a, u.zha, u.zla, ra, fl & 15u);
  return a + resid_quad(u.xp, u.a, u.ypb, u.ymb, u.b, u.zhb, u.zlb, rb, (fl >> 4) & 15u);
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Unit `u` of the grid: its place, its first cell, the cells of its quads.
struct UnitPos {
  int x, y, zq, cell, len;
  bool two;  // quad B is inside
};
__device__ __forceinline__ UnitPos unit_pos(const Dims& d, int nq, int u) {
  UnitPos p;
  const int row = u / nq, xx = row / d.sy;
  p.zq = u - row * nq;
  p.x = 2 * xx;
  p.y = row - xx * d.sy;
  p.cell = (p.x * d.sy + p.y) * d.sz + 4 * p.zq;
  p.len = min(4, d.sz - 4 * p.zq);
  p.two = p.x + 1 < d.sx;
  return p;
}
__device__ __forceinline__ unsigned quad_fluid(const int8_t* __restrict__ type, int cell, int len, bool vec) {
  unsigned m = 0;
  if (vec) {
    const char4 t = *reinterpret_cast<const char4*>(type + cell);
    m = (t.x == kFluid ? 1u : 0u) | (t.y == kFluid ? 2u : 0u) | (t.z == kFluid ? 4u : 0u) | (t.w == kFluid ? 8u : 0u);
  } else {
    for (int k = 0; k < len; ++k) m |= (type[cell + k] == kFluid ? 1u : 0u) << k;
  }
  return m;
}
__device__ __forceinline__ unsigned unit_fluid(const Dims& d, const int8_t* __restrict__ type, const UnitPos& p,
                                               bool vec) {
  unsigned m = quad_fluid(type, p.cell, p.len, vec);
  if (p.two) m |= quad_fluid(type, p.cell + d.sy * d.sz, p.len, vec) << 4;
  return m;
}
// A quad's values; cells beyond the row's end copy the last one.
__device__ __forceinline__ Quad load_cells(const float* __restrict__ v, int cell, int len) {
  float4 r;
  r.x = __ldcg(v + cell);
  r.y = len > 1 ? __ldcg(v + cell + 1) : r.x;
  r.z = len > 2 ? __ldcg(v + cell + 2) : r.y;
  r.w = len > 3 ? __ldcg(v + cell + 3) : r.z;
  return pack4(r);
}
// -0 is stored as +0, which the other plans write.
__device__ __forceinline__ void store_cells(float* __restrict__ v, int cell, int len, const Quad& q) {
  const float4 o = unpack4({add2(q.lo, 0ull), add2(q.hi, 0ull)});
  v[cell] = o.x;
  if (len > 1) v[cell + 1] = o.y;
  if (len > 2) v[cell + 2] = o.z;
  if (len > 3) v[cell + 3] = o.w;
}

// The sum of n residual partials in a fixed order; the same in every thread.
__device__ __forceinline__ double sum_parts(const double* part, int n, double* s_red) {
  double a = 0.0;
  for (int i = threadIdx.x; i < n; i += kT) a += __ldcg(part + i);
  __syncthreads();
  s_red[threadIdx.x] = a;
  __syncthreads();
  for (int o = kT / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) s_red[threadIdx.x] += s_red[threadIdx.x + o];
    __syncthreads();
  }
  return s_red[0];
}

// Blocks of sweeps, each followed by a residual, until the solve's end.
// sweeps(k): k sweeps; residual(): the CTA's partials of the iterate.
template <class SW, class RE>
__device__ __forceinline__ void solve_loop(const ClusterScene& S, const SolveArgs& a, Solve& v, double* s_red,
                                           SW&& sweeps, RE&& residual) {
  for (;;) {
    const int todo = a.fixed_sweeps > 0 ? a.fixed_sweeps : a.check;
    if (v.n > 0) sweeps(todo);
    v.done += todo;
    residual();
    cluster_sync(v.nr);
    v.r2 = sum_parts(S.part, (v.n + 31) / 32, s_red);
    v.rel = rel_residual_of(v.r2, v.b2);
    ++v.checks;
    if (a.fixed_sweeps > 0 || !(v.rel > a.tol) || !isfinite(v.rel) || v.it0 + v.done >= a.max_iters) break;
    cluster_sync(v.nr);  // the partials are read before the next check rewrites them
  }
}

// The solve with at most U units to a thread.  RAGGED: sx is odd or sz not a
// multiple of 4, so units may reach beyond the walls.
template <int U, bool RAGGED>
__device__ __forceinline__ void solve_shared(const ClusterScene& S, const SolveArgs& a, Solve& v, double* s_red,
                                             unsigned smem) {
  // 31 registers a unit with its iterate and its reciprocals, 15 with neither; two
  // units with both leave no room to overlap them (64 x 24 x 64, 90k fluid cells:
  // 1.41 us a sweep, 1.28 with the reciprocals made anew)
  constexpr bool KEEP_C = U <= 3, KEEP_R = U <= 1;
  const Dims& d = S.d;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nq = (d.sz + 3) / 4, plane = d.sy * d.sz;
  const bool vec = d.sz % 4 == 0;
  const unsigned me = v.me, nr = v.nr;
  const int per = v.per;
  const int first = (int)me * per, nloc = max(0, min(v.n - first, per));
  const unsigned own = smem + tid * 16;
  const Quad none = {0ull, 0ull};
  Quad rha[U], rhb[U], ca[KEEP_C ? U : 1], cb[KEEP_C ? U : 1], ra[KEEP_R ? U : 1], rb[KEEP_R ? U : 1];
  Near at[U];
  unsigned fl[U];
  if (tid == 0) {
    st4<0>(smem + kZero * 16, none);
    st4<kHalf>(smem + kZero * 16, none);
    st4<kBufBytes>(smem + kZero * 16, none);
    st4<kBufBytes + kHalf>(smem + kZero * 16, none);
  }
#pragma unroll
  for (int j = 0; j < U; ++j) {
    const int s = tid + j * kT;
    const unsigned zero = smem + kZero * 16, self = smem + s * 16;
    unsigned f = 0u;
    Quad va = none, vb = none;
    rha[j] = rhb[j] = none;
    at[j] = {zero, zero, zero, zero, zero, zero};
    if (s < nloc) {
      const int u = __ldcg(S.list + first + s);
      const UnitPos p = unit_pos(d, nq, u);
      int k[6];  // neighbours' indices: -1 no fluid, -2 wall
      k[0] = p.x > 0 ? __ldcg(S.umap + u - d.sy * nq) : -2;
      k[1] = p.x + 2 < d.sx ? __ldcg(S.umap + u + d.sy * nq) : -2;
      k[2] = p.y + 1 < d.sy ? __ldcg(S.umap + u + nq) : -2;
      k[3] = p.y > 0 ? __ldcg(S.umap + u - nq) : -2;
      k[4] = p.zq + 1 < nq ? __ldcg(S.umap + u + 1) : -2;
      k[5] = p.zq > 0 ? __ldcg(S.umap + u - 1) : -2;
      f = kValid | unit_fluid(d, S.type, p, vec);
      if (!p.two) f |= kCopyB;
      if (p.len < 4) f |= (unsigned)p.len << kLenShift;
#pragma unroll
      for (int e = 0; e < 6; ++e)
        if (k[e] >= 0 && k[e] / per != (int)me) f |= e < 2 ? kFarX : kFarYZ;
      // `in`: offset in the neighbour, `wall`: offset in the unit itself
      auto place = [&](int index, unsigned far, unsigned in, unsigned wall) {
        const unsigned x = index >= 0 ? smem + (unsigned)(index % per) * 16u + in
                                      : (index == -1 ? zero + in : self + wall);
        return f & far ? mapa(x, index >= 0 ? (unsigned)(index / per) : me) : x;
      };
      at[j].xm = place(k[0], kFarX, kHalf, 0u);
      at[j].xp = place(k[1], kFarX, 0u, kHalf);
      at[j].yp = place(k[2], kFarYZ, 0u, 0u);
      at[j].ym = place(k[3], kFarYZ, 0u, 0u);
      at[j].zh = place(k[4], kFarYZ, 0u, 12u);
      at[j].zl = place(k[5], kFarYZ, 12u, 0u);
      rha[j] = load_cells(S.rhs, p.cell, p.len);
      va = load_cells(S.pa, p.cell, p.len);
      rhb[j] = p.two ? load_cells(S.rhs, p.cell + plane, p.len) : rha[j];
      vb = p.two ? load_cells(S.pa, p.cell + plane, p.len) : va;
    }
    fl[j] = f;
    if (KEEP_C) {
      ca[KEEP_C ? j : 0] = va;
      cb[KEEP_C ? j : 0] = vb;
    }
    if (KEEP_R) {
      ra[KEEP_R ? j : 0] = sixths(f & 15u);
      rb[KEEP_R ? j : 0] = sixths((f >> 4) & 15u);
    }
    if (s < kZero) {
      st4<0>(own + j * kT * 16, va);
      st4<kHalf>(own + j * kT * 16, vb);
    }
  }
  cluster_sync(nr);

  auto load = [&](auto tag, int j, UnitIn& u) {
    constexpr int B = decltype(tag)::value;
    u.a = KEEP_C ? ca[KEEP_C ? j : 0] : ld4<B * kBufBytes, false>(own + j * kT * 16);
    u.b = KEEP_C ? cb[KEEP_C ? j : 0] : ld4<B * kBufBytes + kHalf, false>(own + j * kT * 16);
    load_unit<B>(u, at[j], fl[j]);
  };
  // one sweep from buffer B to the other
  auto sweep = [&](auto tag) {
    constexpr int O = (decltype(tag)::value ^ 1) * kBufBytes;
#pragma unroll
    for (int j = 0; j < U; ++j) {
      if (!fl[j]) continue;
      UnitIn u;
      load(tag, j, u);
      update_unit(u, rha[j], rhb[j], KEEP_R ? ra[KEEP_R ? j : 0] : sixths(fl[j] & 15u),
                  KEEP_R ? rb[KEEP_R ? j : 0] : sixths((fl[j] >> 4) & 15u));
      if (RAGGED) {
        const unsigned len = (fl[j] >> kLenShift) & 3u;
        if (len) {
          u.a = copy_tail(u.a, len);
          u.b = copy_tail(u.b, len);
        }
        if (fl[j] & kCopyB) u.b = u.a;
      }
      st4<O>(own + j * kT * 16, u.a);
      st4<O + kHalf>(own + j * kT * 16, u.b);
      if (KEEP_C) {
        ca[KEEP_C ? j : 0] = u.a;
        cb[KEEP_C ? j : 0] = u.b;
      }
    }
    cluster_sync(nr);
  };
  using B0 = std::integral_constant<int, 0>;
  using B1 = std::integral_constant<int, 1>;
  bool odd = false;  // the iterate is in buffer 1
  auto residual_of = [&](auto tag) {
#pragma unroll
    for (int j = 0; j < U; ++j) {
      double acc = 0.0;
      if (fl[j]) {
        UnitIn u;
        load(tag, j, u);
        acc = resid_unit(u, rha[j], rhb[j], fl[j]);
      }
      acc = warp_sum(acc);
      const int s0 = j * kT + warp * 32;
      if (lane == 0 && s0 < nloc) S.part[(first + s0) / 32] = acc;
    }
  };
  solve_loop(
      S, a, v, s_red,
      [&](int k) {
        if (odd) {
          sweep(B1{});
          --k;
          odd = false;
        }
        for (; k >= 2; k -= 2) {
          sweep(B0{});
          sweep(B1{});
        }
        if (k) {
          sweep(B0{});
          odd = true;
        }
      },
      [&]() {
        if (odd) residual_of(B1{});
        else residual_of(B0{});
      });
  for (int s = tid; s < nloc; s += kT) {
    const UnitPos p = unit_pos(d, nq, __ldcg(S.list + first + s));
    const unsigned at0 = smem + s * 16;
    store_cells(S.pa, p.cell, p.len, odd ? ld4<kBufBytes, false>(at0) : ld4<0, false>(at0));
    if (p.two)
      store_cells(S.pa, p.cell + plane, p.len, odd ? ld4<kBufBytes + kHalf, false>(at0) : ld4<kHalf, false>(at0));
  }
  cluster_sync(nr);  // no CTA leaves while another reads its buffers
}

template <bool RAGGED>
__device__ __forceinline__ void solve_units(const ClusterScene& S, const SolveArgs& a, Solve& v, double* s_red,
                                            unsigned smem) {
  const int nj = (v.per + kT - 1) / kT;  // the same in every CTA
  if (nj == 1) solve_shared<1, RAGGED>(S, a, v, s_red, smem);
  else if (nj == 2) solve_shared<2, RAGGED>(S, a, v, s_red, smem);
  else if (nj == 3) solve_shared<3, RAGGED>(S, a, v, s_red, smem);
  else solve_shared<4, RAGGED>(S, a, v, s_red, smem);
}

// The fluid does not fit.  Called out of line, with the running values by
// address: they then live on the stack between a solve's checks and the sweeps'
// registers hold their units with hardly a spill.  For the same reason another
// kernel sets the graph's condition: a call of the device runtime in this one
// costs registers (with both 192 bytes spilled and 12% longer sweeps).
__device__ __noinline__ void outgrown(const SolveArgs& a, Solve& v) {
  if (v.me == 0 && threadIdx.x == 0) *a.spilled = 1;
  v.n = -1;
}

// Starts from pa; the result is in pa.  False where the fluid does not fit the
// cluster, which leaves pa and the solve state alone.
__device__ __forceinline__ bool cluster_solve(const ClusterScene& S, const SolveArgs& a) {
  extern __shared__ __align__(16) unsigned char cl_smem[];
  __shared__ double s_red[kT];
  __shared__ int s_warp[kT / 32];
  __shared__ int s_count;
  const Dims& d = S.d;
  Solve v;
  v.me = cluster_rank();
  v.nr = cluster_size();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nq = (d.sz + 3) / 4, total = (d.sx + 1) / 2 * d.sy * nq;
  const bool vec = d.sz % 4 == 0;

  // number the fluid units: CTA `me` scans units [lo, hi)
  const int chunk = ((total + (int)v.nr - 1) / (int)v.nr + kT - 1) / kT * kT;
  const int lo = (int)v.me * chunk, hi = min(lo + chunk, total);
  unsigned bits = 0;
  for (int k = 0, u = lo + tid; u < hi; ++k, u += kT)
    if (unit_fluid(d, S.type, unit_pos(d, nq, u), vec)) bits |= 1u << k;
  if (tid == 0) s_count = 0;
  __syncthreads();
  {
    int c = __popc(bits);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if (lane == 0) atomicAdd(&s_count, c);
  }
  cluster_sync(v.nr);
  int base = 0;
  v.n = 0;
  for (unsigned r = 0; r < v.nr; ++r) {
    const unsigned at = static_cast<unsigned>(__cvta_generic_to_shared(&s_count));
    const int c = v.nr == 1 ? s_count : __float_as_int(ld1<0, true>(mapa(at, r)));
    if (r < v.me) base += c;
    v.n += c;
  }
  for (int k = 0, u0 = lo; u0 < hi; ++k, u0 += kT) {
    const bool f = (bits >> k) & 1u;
    const unsigned m = __ballot_sync(0xffffffffu, f);
    __syncthreads();
    if (lane == 0) s_warp[warp] = __popc(m);
    __syncthreads();
    int before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < kT / 32; ++w) {
      const int c = s_warp[w];
      if (w < warp) before += c;
      all += c;
    }
    const int u = u0 + tid;
    const int idx = base + before + __popc(m & ((1u << lane) - 1u));
    if (u < hi) S.umap[u] = f ? idx : -1;
    if (f) S.list[idx] = u;
    base += all;
  }
  cluster_sync(v.nr);

  v.per = max(32, ((v.n + (int)v.nr - 1) / (int)v.nr + 31) / 32 * 32);
  v.b2 = S.ss->b2;
  v.it0 = S.ss->iterations;
  v.done = v.checks = 0;
  v.r2 = v.rel = -1.0;
  const unsigned smem = static_cast<unsigned>(__cvta_generic_to_shared(cl_smem));
  if (v.per > kCap) outgrown(a, v);  // the same in every CTA
  else if (d.sx % 2 || !vec) solve_units<true>(S, a, v, s_red, smem);
  else solve_units<false>(S, a, v, s_red, smem);
  if (v.n < 0) return false;
  if (v.me == 0 && tid == 0 && a.r2_only) {
    *a.r2_only = v.r2;
  } else if (v.me == 0 && tid == 0) {
    SolveState* ss = S.ss;
    ss->iterations = v.it0 + v.done;
    ss->bodies += v.checks;
    ss->total_sweeps += v.done;
    ss->total_bodies += v.checks;
    ss->r2 = v.r2;
    ss->rel_residual = v.rel;
    const bool finite = isfinite(v.rel);
    if (!finite) ss->nonfinite = ss->nonfinite_seen = 1;
    ss->converged = finite && v.rel <= a.tol ? 1 : 0;
  }
  return true;
}

__global__ void __launch_bounds__(kT, 1) k_cluster_solve(const __grid_constant__ ClusterScene S, SolveArgs a) {
  cluster_solve(S, a);
}

// One cluster per scene of a batch: the clusters of the launch take the scenes
// order[0], order[1], ... (largest first) that are live, and clear the mark of
// those they solve.
__global__ void __launch_bounds__(kT, 1) kb_cluster_solve(BatchIndex bi, const int* __restrict__ order,
                                                        const int2* __restrict__ scratch, int* live, float* pa,
                                                        const float* rhs, const int8_t* type, int* umap, int* list,
                                                        double* part, SolveState* ss, SolveArgs a) {
  const int s = order[blockIdx.x / cluster_size()];
  if (!__ldcg(live + s)) return;  // the same in all CTAs of the cluster: none clears it before all have met
  const SceneDesc& D = bi.scenes[s];
  const int2 at = scratch[s];  // the scene's first unit and first residual partial
  const int c = D.c_off;
  const ClusterScene S{D.d, pa + c, rhs + c, type + c, umap + at.x, list + at.x, part + at.y, ss + s};
  if (cluster_solve(S, a) && cluster_rank() == 0 && threadIdx.x == 0) live[s] = 0;
}

// The condition from the mark of the cluster solves before, which it clears.
__global__ void k_spill_condition(int* spilled, cudaGraphConditionalHandle handle) {
  cudaGraphSetConditional(handle, *spilled ? 1 : 0);
  *spilled = 0;
}

// Self-check of update_quad's quotients against the IEEE divide over all 2^32
// bit patterns (zeros compare equal, NaN equal to NaN).
__global__ void k_cluster_div_check(unsigned long long* bad) {
  unsigned long long local = 0;
  const unsigned stride = gridDim.x * blockDim.x;
  const Quad none = pack4(make_float4(-0.f, -0.f, -0.f, -0.f));
  for (unsigned long long i = blockIdx.x * blockDim.x + threadIdx.x; i <= 0xffffffffull; i += stride) {
    const float x = __uint_as_float((unsigned)i);
    const float4 q = unpack4(update_quad(pack4(make_float4(x, 1.f, 0.f, -x)), none, none, none, none, -0.f, -0.f, none,
                                         sixths(15u)));
    const float a[2] = {q.x, q.w}, e[2] = {__fdiv_rn(x, 6.f), __fdiv_rn(-x, 6.f)};
    for (int k = 0; k < 2; ++k)
      if (!(isnan(a[k]) && isnan(e[k])) && !(a[k] == 0.f && e[k] == 0.f) &&
          __float_as_uint(a[k]) != __float_as_uint(e[k]))
        ++local;
  }
  if (local) atomicAdd(bad, local);
}

// Launch configuration of `clusters` clusters of `width` CTAs.
struct ClusterLaunch {
  cudaLaunchConfig_t lc = {};
  cudaLaunchAttribute at[1];
  ClusterLaunch(cudaStream_t st, int clusters, int width) {
    lc.gridDim = dim3(clusters * width);
    lc.blockDim = dim3(kT);
    lc.dynamicSmemBytes = kSmem;
    lc.stream = st;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = width;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    lc.attrs = at;
    lc.numAttrs = 1;
  }
};

template <class K>
cudaError_t allow_cluster(K kernel) {
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
  return e != cudaSuccess ? e : cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
}
cudaError_t allow_solve() {
  static PerDevice once;
  return once([] { return allow_cluster(k_cluster_solve); });
}
cudaError_t allow_batch_solve() {
  static PerDevice once;
  return once([] { return allow_cluster(kb_cluster_solve); });
}

}  // namespace

long long cluster_solve_units(const Dims& d) { return (long long)((d.sx + 1) / 2) * d.sy * ((d.sz + 3) / 4); }

// One CTA sweeps about 200 fluid units in 0.39 us and 700 in 0.75 us; 16 CTAs
// take 0.55 us for either, most of it the cluster's barrier.  A grid of 1024
// units rarely holds more than 300 fluid ones.
int cluster_solve_width(const Dims& d) { return cluster_solve_units(d) <= kSmallUnits ? 1 : 16; }

bool cluster_solve_holds(const Dims& d, int width) { return cluster_solve_units(d) <= (long long)width * kCap; }

bool cluster_solve_takes(const Dims& d, int width) {
  return width >= 1 && width <= 16 && (width & (width - 1)) == 0 &&
         cluster_solve_units(d) <= (long long)width * kT * kScanBits;
}

bool cluster_solve_fits(const Dims& d, long long particles) {
  const int w = cluster_solve_width(d);
  if (!cluster_solve_takes(d, w)) return false;
  // 8 particles to a fluid cell, 8 cells to a unit.  The row list catches up
  // with the cluster where a thread has three units (64^3 three quarters full:
  // 2.4 us a sweep against 2.2 us), and a fluid that has spread needs room.
  return particles / 64 <= (long long)w * kCap * 7 / 10;
}

bool cluster_solve_runs(int width) {
  ClusterLaunch l(nullptr, 1, width);
  int alone = 0, batch = 0;
  cudaError_t e = allow_solve();
  if (e == cudaSuccess) e = allow_batch_solve();
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&alone, k_cluster_solve, &l.lc);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&batch, kb_cluster_solve, &l.lc);
  if (e != cudaSuccess) cudaGetLastError();
  return e == cudaSuccess && alone > 0 && batch > 0;
}

cudaError_t launch_cluster_solve(cudaStream_t st, const Dims& d, int width, float* pa, const float* rhs,
                                 const int8_t* type, int* umap, int* list, double* part, SolveState* ss,
                                 int fixed_sweeps, int check, int max_iters, double tol, double* r2_only,
                                 int* spilled) {
  if (!spilled && !cluster_solve_holds(d, width)) return cudaErrorInvalidValue;
  if (const cudaError_t e = allow_solve()) return e;
  ClusterLaunch l(st, 1, width);
  const ClusterScene S{d, pa, rhs, type, umap, list, part, ss};
  return cudaLaunchKernelEx(&l.lc, k_cluster_solve, S,
                            SolveArgs{fixed_sweeps, check, max_iters, tol, r2_only, spilled});
}

cudaError_t launch_spill_condition(cudaStream_t st, int* spilled, unsigned long long handle) {
  k_spill_condition<<<1, 1, 0, st>>>(spilled, (cudaGraphConditionalHandle)handle);
  return cudaGetLastError();
}

cudaError_t launch_cluster_div_check(cudaStream_t st, unsigned long long* bad) {
  k_cluster_div_check<<<148 * 8, 256, 0, st>>>(bad);
  return cudaGetLastError();
}

// A batch fills the machine by its number of scenes, so a scene takes the
// narrowest cluster that holds twice its initial fluid (up to kU units to a
// thread cost a sweep 0.37 us each against 0.4 us for the cluster's barrier).
// Where the fluid has spread further the scene's solve goes to a cluster of 16
// CTAs, and to the sweeps where even that does not hold it: the solve that the
// scene has alone.
int batch_cluster_width(const Dims& d, long long particles) {
  if (!cluster_solve_fits(d, particles)) return 0;
  const long long units = std::min(cluster_solve_units(d), std::max(1LL, 2 * particles / 64));
  for (int w = 1; w <= 16; w *= 2)
    if ((units <= (long long)w * kCap || w == 16) && cluster_solve_takes(d, w)) return w;
  return 0;
}

cudaError_t launch_batch_cluster_solve(cudaStream_t st, const BatchIndex& bi, int scenes, int width, const int* order,
                                       const int2* scratch, int* live, float* pa, const float* rhs,
                                       const int8_t* type, int* umap, int* list, double* part, SolveState* ss,
                                       int fixed_sweeps, int check, int max_iters, double tol,
                                       int* spilled) {
  if (scenes <= 0) return cudaSuccess;
  if (const cudaError_t e = allow_batch_solve()) return e;
  ClusterLaunch l(st, scenes, width);
  return cudaLaunchKernelEx(&l.lc, kb_cluster_solve, bi, order, scratch, live, pa, rhs, type, umap, list, part, ss,
                            SolveArgs{fixed_sweeps, check, max_iters, tol, nullptr, spilled});
}

}  // namespace aqb
