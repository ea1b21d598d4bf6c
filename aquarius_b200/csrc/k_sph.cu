// Kernels of the particle-only solvers: position-based fluids and PCISPH.
//
// Reference: Fluid_3D_PBF (Fluid/Fluid_3D_PBF.cu:6-267) and Fluid_3D_PCISPH
// (Fluid/Fluid_3D_PCISPH.cu:13-202), with poly6 / spikey_grad /
// cubic_spline_kernel (Fluid/WeightKernels.cuh:13-58, 196-206) and the
// spatial hash of performSpatialHashing2 (Fluid/Fluid_3D_common.cuh:27-56).
//
// Particles live as float4 arrays (16-byte loads in the neighbour loops):
//   PBF:    P = (position, restDensity), L = (lastPosition, -),
//           V = (velocity, density), Q = (position, lambda) written by the
//           lambda pass and read by the delta pass, which writes P.
//   PCISPH: P = (position, restDensity), V = (velocity, density),
//           Q = (predictedPosition, -), W = (predictedVelocity, pressure),
//           F = (pressureForces, -), R = (predictedPosition, p / rho^2)
//           written by the density pass and read by the force pass.
// No pass reads a float4 another thread of the same pass writes.
//
// Every float operation is an explicitly rounded intrinsic in the order the
// reference writes it (no contraction), and neighbours are walked in the
// reference's order (27 cells x-major, particles in stable sorted order), so
// results equal the CPU oracle's bit for bit.
#include "aq_kernels.cuh"

namespace aqb {
namespace {

inline int blocks(int n, int t) { return (n + t - 1) / t; }

__device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float dvd(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ float clampw(float v, float lo, float hi) { return fminf(hi, fmaxf(lo, v)); }

__device__ __forceinline__ float dot3(float x, float y, float z) { return add(add(mul(x, x), mul(y, y)), mul(z, z)); }

// Neighbour pairs with r2 > p.skip_r2 lie outside both kernels' support:
// poly6 is 0 (r2 > h2) and spikey_grad is the zero vector (sqrt(r2) > h).
// Adding their zero terms changes no sum (at most the sign of a zero that is
// then squared or added to a nonzero value), so the passes skip them; about
// 85% of the 27-cell candidates are such pairs.
__device__ __forceinline__ bool outside(float r2, const SphParams& p) { return r2 > p.skip_r2; }

__device__ __forceinline__ float dvd(float a, const Divisor& d) {
  return d.ok && mag_key(a) >= kLeastKey && fabsf(a) <= 0x1p60f ? dvd_fast(a, d) : dvd(a, d.b);
}
__device__ __forceinline__ float3 dvd(const float3& a, const Divisor& d) {
  const unsigned least = min(min(mag_key(a.x), mag_key(a.y)), mag_key(a.z));
  const float most = fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fabsf(a.z));
  if (d.ok && least >= kLeastKey && most <= 0x1p60f)
    return make_float3(dvd_fast(a.x, d), dvd_fast(a.y, d), dvd_fast(a.z, d));
  return make_float3(dvd(a.x, d.b), dvd(a.y, d.b), dvd(a.z, d.b));
}

// poly6 (Fluid/WeightKernels.cuh:13-26)
__device__ __forceinline__ float poly6(float r2, const SphParams& p) {
  if (r2 <= p.kr2) {
    const float t = sub(p.kr2, r2);
    return dvd(mul(mul(mul(t, t), t), 315.f), divisor(p.poly6_den, p.poly6_rcp));
  }
  return 0.f;
}

// spikey_grad (Fluid/WeightKernels.cuh:43-58); r2 = v . v
__device__ __forceinline__ float3 spikey(float vx, float vy, float vz, float r2, const SphParams& p) {
  const float r = __fsqrt_rn(r2);
  float3 u = make_float3(vx, vy, vz);
  if (r != 0.f) u = dvd(u, divisor(r, __frcp_rn(r)));
  if (0.f <= r && r <= p.kr) {
    const float hr = sub(p.kr, r);
    return dvd(make_float3(mul(mul(mul(-u.x, hr), hr), 45.f), mul(mul(mul(-u.y, hr), hr), 45.f),
                           mul(mul(mul(-u.z, hr), hr), 45.f)),
               divisor(p.spikey_den, p.spikey_rcp));
  }
  return make_float3(0.f, 0.f, 0.f);
}

__device__ __forceinline__ int3 cell_of(const SphParams& p, float x, float y, float z) {
  return make_int3((int)dvd(x, p.kr), (int)dvd(y, p.kr), (int)dvd(z, p.kr));
}

// The neighbour walk: the 27 cells around c, dx, dy, dz from -1 to 1, outside
// ones skipped (Fluid/Fluid_3D_PBF.cu:37-58), particles in sorted order.  The
// up to three cells of a (dx, dy) are consecutive in the cell order, so their
// particles are one run.
//
// Four lanes work on a particle.  They scan four candidates of a run at a time
// and append the inside ones (about 15%) to the particle's list in order (a
// ballot), then evaluate four of its terms at a time, and lane k adds component
// k (and k + 4) of the terms in list order: the reference's sums, term for
// term.  Evaluated in the scan, one thread a particle, the costly terms ran
// with 13.9 of 32 lanes on the average; one thread a particle with lists of
// its own leaves the machine short of warps at the reference's default of
// 60k particles (PBF step 1290 us against 826 us).
//
// The density pass keeps the lists for the pass that follows it on the same
// positions (PBF's delta, PCISPH's force), which then scans nothing.
constexpr int kThreads = 128, kPart = kThreads / 4;  // particles per CTA
constexpr int kList = 64;                            // listed at a time
template <int NC>
struct WalkShared {
  int list[kPart][kList];
  float4 term[kPart][NC];
};

// Adds the terms of up to four list entries: this lane's is t (zeros past the
// end, which change no sum).
template <int NC>
__device__ __forceinline__ void add_terms(WalkShared<NC>& sm, const float (&t)[NC], float (&sum)[2]) {
  const int l = threadIdx.x & 3, g = threadIdx.x >> 2;
#pragma unroll
  for (int k = 0; k < NC; ++k) reinterpret_cast<float*>(&sm.term[g][k])[l] = t[k];
  __syncwarp();
  if (l < NC) {
    const float4 v = sm.term[g][l];
    sum[0] = add(add(add(add(sum[0], v.x), v.y), v.z), v.w);
  }
  if (l + 4 < NC) {
    const float4 v = sm.term[g][l + 4];
    sum[1] = add(add(add(add(sum[1], v.x), v.y), v.z), v.w);
  }
  __syncwarp();
}

// All lanes of the warp call this together; lanes of a missing particle
// (!valid) walk nothing.  sum[0], sum[1]: components k and k + 4 in lane k.
// keep (may be null): where the particle's first kSphList neighbours go;
// returns how many there are.
template <int NC, typename Inside, typename Term>
__device__ __forceinline__ int walk(const SphParams& p, int3 c, bool valid, const int* __restrict__ off,
                                    int* __restrict__ keep, WalkShared<NC>& sm, float (&sum)[2], Inside&& inside,
                                    Term&& term) {
  const int l = threadIdx.x & 3, g = threadIdx.x >> 2, shift = threadIdx.x & 28;
  int cnt = 0, total = 0;
  sum[0] = sum[1] = 0.f;
  auto flush = [&]() {
    __syncwarp();
    const int most = __reduce_max_sync(0xffffffffu, cnt);
    for (int b = 0; b < most; b += 4) {
      float t[NC];
#pragma unroll
      for (int k = 0; k < NC; ++k) t[k] = 0.f;
      if (b + l < cnt) {
        const int j = sm.list[g][b + l];
        if (keep && total + b + l < kSphList) keep[total + b + l] = j;
        term(j, t);
      }
      add_terms<NC>(sm, t, sum);
    }
    total += cnt;
    cnt = 0;
  };
  const int z0 = max(c.z - 1, 0), z1 = min(c.z + 1, p.gz - 1) + 1;
  for (int dx = -1; dx <= 1; ++dx)
    for (int dy = -1; dy <= 1; ++dy) {
      const int x = c.x + dx, y = c.y + dy;
      int j = 0, j1 = 0;
      if (valid && z1 > z0 && x >= 0 && x < p.gx && y >= 0 && y < p.gy) {
        const int row = (x * p.gy + y) * p.gz;
        j = __ldg(off + row + z0) + l;
        j1 = __ldg(off + row + z1);
      }
      while (__any_sync(0xffffffffu, j < j1)) {
        const bool in = j < j1 && inside(j);
        const unsigned m = (__ballot_sync(0xffffffffu, in) >> shift) & 15u;
        if (in) sm.list[g][cnt + __popc(m & ((1u << l) - 1u))] = j;
        cnt += __popc(m);
        j += 4;
        if (__any_sync(0xffffffffu, cnt > kList - 4)) flush();
      }
    }
  flush();
  return total;
}

// The same sums from the lists a walk on the same positions kept; a warp with
// a particle of more than kSphList neighbours (or without lists) walks.
template <int NC, typename Inside, typename Term>
__device__ __forceinline__ void walk_kept(const SphParams& p, int3 c, int i, bool valid, const int* __restrict__ off,
                                          const int* __restrict__ count, const int* __restrict__ lists,
                                          WalkShared<NC>& sm, float (&sum)[2], Inside&& inside, Term&& term) {
  const int cnt = valid && count ? __ldg(count + i) : 0;
  const int most = __reduce_max_sync(0xffffffffu, cnt);
  if (!count || most > kSphList) {
    walk<NC>(p, c, valid, off, nullptr, sm, sum, inside, term);
    return;
  }
  const int l = threadIdx.x & 3;
  const int* __restrict__ row = lists + (size_t)i * kSphList;
  sum[0] = sum[1] = 0.f;
  int j = l < cnt ? __ldg(row + l) : 0;
  for (int b = 0; b < most; b += 4) {
    const int next = b + 4 + l < cnt ? __ldg(row + b + 4 + l) : 0;
    float t[NC];
#pragma unroll
    for (int k = 0; k < NC; ++k) t[k] = 0.f;
    if (b + l < cnt) term(j, t);
    add_terms<NC>(sm, t, sum);
    j = next;
  }
}

// --------------------------------------------------------------- sorting

// calcHashImpl (Fluid/Fluid_3D_kernels.cuh:8-27) on the kernel-radius grid,
// and a warp-aggregated slot in the cell's count.  Positions are kept inside
// the container, so the clamps only guard against other input.
__global__ void __launch_bounds__(256) k_sph_keys(SphParams p, const float4* __restrict__ pos, int* __restrict__ key,
                                                 int* __restrict__ slot, int* __restrict__ count, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = i < n;
  int k = -1;
  if (valid) {
    const float4 q = pos[i];
    int3 c = cell_of(p, q.x, q.y, q.z);
    c.x = min(max(c.x, 0), p.gx - 1);
    c.y = min(max(c.y, 0), p.gy - 1);
    c.z = min(max(c.z, 0), p.gz - 1);
    k = (c.x * p.gy + c.y) * p.gz + c.z;
    key[i] = k;
  }
  const unsigned peers = __match_any_sync(0xffffffffu, k);
  if (valid) {
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(peers) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(count + k, __popc(peers));
    base = __shfl_sync(peers, base, leader);
    slot[i] = base + __popc(peers & ((1u << lane) - 1u));
  }
}

// Stable placement (rank among the cell's particles by previous index, as
// thrust's stable sort orders them) and the gather of every particle array.
__global__ void __launch_bounds__(256) k_sph_gather(const int* __restrict__ key, const int* __restrict__ off,
                                                   const int* __restrict__ perm_u, SphArrays src, SphArrays dst, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int k = key[i];
  const int b = __ldg(off + k), e = __ldg(off + k + 1);
  int r = 0;
  for (int j = b; j < e; ++j) r += __ldg(perm_u + j) < i;
  const int d = b + r;
#pragma unroll
  for (int a = 0; a < kSphArrays; ++a)
    if (src.a[a]) dst.a[a][d] = src.a[a][i];
}

// ------------------------------------------------------------------- PBF

// applyForcesImpl + predictPositionImpl (Fluid_3D_PBF.cu:6-26)
__global__ void __launch_bounds__(256) k_pbf_predict(SphParams p, float4* __restrict__ P, const float4* __restrict__ L,
                                                    float4* __restrict__ V, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float4 v = V[i], q = P[i];
  const float4 l = L[i];
  v.x = add(v.x, mul(p.dt, p.g.x));
  v.y = add(v.y, mul(p.dt, p.g.y));
  v.z = add(v.z, mul(p.dt, p.g.z));
  q.x = clampw(add(l.x, mul(p.dt, v.x)), p.md, sub(p.size, p.md));
  q.y = clampw(add(l.y, mul(p.dt, v.y)), p.md, sub(p.size, p.md));
  q.z = clampw(add(l.z, mul(p.dt, v.z)), p.md, sub(p.size, p.md));
  V[i] = v;
  P[i] = q;
}

// computeDensityAndLambdaImpl (Fluid_3D_PBF.cu:28-110): reads P, writes
// Q = (position, lambda), the density into V.w and, on the rest-density
// pass, P.w.  A term: poly6, spikey_grad and its square.
__device__ __forceinline__ void lambda_term(const SphParams& p, const float4& me, const float4& o, float (&t)[5]) {
  const float dx = sub(me.x, o.x), dy = sub(me.y, o.y), dz = sub(me.z, o.z);
  const float r2 = dot3(dx, dy, dz);
  const float3 w = spikey(dx, dy, dz, r2, p);
  t[0] = w.x;
  t[1] = w.y;
  t[2] = w.z;
  t[3] = poly6(r2, p);
  t[4] = dot3(w.x, w.y, w.z);
}
__global__ void __launch_bounds__(kThreads) k_pbf_lambda(SphParams p, const int* __restrict__ off,
                                                        float4* __restrict__ P, float4* __restrict__ V,
                                                        float4* __restrict__ Q, int* __restrict__ count,
                                                        int* __restrict__ lists, int set_rest, int n) {
  __shared__ WalkShared<5> sm;
  const int i = (blockIdx.x * kThreads + threadIdx.x) >> 2;
  const float4 me = i < n ? P[i] : make_float4(0.f, 0.f, 0.f, 0.f);
  float s[2];
  const int found = walk<5>(
      p, cell_of(p, me.x, me.y, me.z), i < n, off, lists ? lists + (size_t)i * kSphList : nullptr, sm, s,
      [&](int j) {
        const float4 o = P[j];
        return !outside(dot3(sub(me.x, o.x), sub(me.y, o.y), sub(me.z, o.z)), p);
      },
      [&](int j, float (&t)[5]) { lambda_term(p, me, P[j], t); });
  const int first = threadIdx.x & 28;
  const float gx = s[0], gy = __shfl_sync(0xffffffffu, s[0], first + 1), gz = __shfl_sync(0xffffffffu, s[0], first + 2);
  const float density = __shfl_sync(0xffffffffu, s[0], first + 3), sdot = s[1];
  if ((threadIdx.x & 3) || i >= n) return;
  if (count) count[i] = found;
  const float rho0 = set_rest ? density : me.w;
  const float ci = sub(dvd(density, rho0), 1.f);
  const float q = dvd(add(sdot, dot3(gx, gy, gz)), mul(rho0, rho0));
  const float den = __double2float_rn(__dadd_rn(1e-3, (double)q));
  float lambda = dvd(-ci, den);
  if (ci < 0.f) lambda = __double2float_rn(__dmul_rn((double)lambda, 1e-2));
  V[i].w = density;
  if (set_rest) P[i].w = density;
  Q[i] = make_float4(me.x, me.y, me.z, lambda);
}

// computeDeltaPositionImpl + applyDeltaPositionImpl (Fluid_3D_PBF.cu:114-206):
// reads Q, writes the moved position into P (its w, the rest density, kept).
__global__ void __launch_bounds__(kThreads) k_pbf_delta(SphParams p, const int* __restrict__ off,
                                                       const float4* __restrict__ Q, float4* __restrict__ P,
                                                       const int* __restrict__ count, const int* __restrict__ lists,
                                                       int n) {
  __shared__ WalkShared<3> sm;
  const int i = (blockIdx.x * kThreads + threadIdx.x) >> 2;
  const float4 me = i < n ? Q[i] : make_float4(0.f, 0.f, 0.f, 0.f);
  const float rho0 = i < n ? P[i].w : 1.f;
  const Divisor by_rho0 = divisor(rho0, __frcp_rn(rho0)), by_corr = divisor(p.s_corr_den, p.s_corr_rcp);
  float s[2];
  walk_kept<3>(
      p, cell_of(p, me.x, me.y, me.z), i, i < n, off, count, lists, sm, s,
      [&](int j) {
        const float4 o = __ldg(Q + j);
        return !outside(dot3(sub(me.x, o.x), sub(me.y, o.y), sub(me.z, o.z)), p);
      },
      [&](int j, float (&t)[3]) {
        const float4 o = __ldg(Q + j);
        const float dx = sub(me.x, o.x), dy = sub(me.y, o.y), dz = sub(me.z, o.z);
        const float r2 = dot3(dx, dy, dz);
        const float3 w = spikey(dx, dy, dz, r2, p);
        const float c = dvd(poly6(r2, p), by_corr);
        const float c2 = mul(c, c);
        const float sc = mul(mul(c2, c2), -p.s_corr_k);
        const float f = add(add(me.w, o.w), sc);
        const float3 q = dvd(make_float3(mul(w.x, f), mul(w.y, f), mul(w.z, f)), by_rho0);
        t[0] = q.x;
        t[1] = q.y;
        t[2] = q.z;
      });
  const int first = threadIdx.x & 28;
  const float ay = __shfl_sync(0xffffffffu, s[0], first + 1), az = __shfl_sync(0xffffffffu, s[0], first + 2);
  if ((threadIdx.x & 3) || i >= n) return;
  const float hi = sub(p.size, p.md);
  P[i] = make_float4(clampw(add(me.x, s[0]), p.md, hi), clampw(add(me.y, ay), p.md, hi),
                     clampw(add(me.z, az), p.md, hi), rho0);
}

// updatePositionAndVelocityImpl (Fluid_3D_PBF.cu:209-267)
__device__ __forceinline__ float pbf_wall(float v, bool low, bool high, float leave) {
  if (low) v = v == 0.f ? leave : mul(v, -0.5f);
  if (high) v = v == 0.f ? -leave : mul(v, -0.5f);
  return v;
}

__global__ void __launch_bounds__(256) k_pbf_update(SphParams p, const float4* __restrict__ P, float4* __restrict__ L,
                                                   float4* __restrict__ V, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 q = P[i];
  const float4 l = L[i];
  float4 v = V[i];
  const float hi = sub(p.size, p.md);
  v.x = pbf_wall(dvd(sub(q.x, l.x), p.dt), q.x == p.md, q.x >= hi, p.leave);
  v.y = pbf_wall(dvd(sub(q.y, l.y), p.dt), q.y <= p.md, q.y >= hi, p.leave);
  v.z = pbf_wall(dvd(sub(q.z, l.z), p.dt), q.z <= p.md, q.z >= hi, p.leave);
  V[i] = v;
  L[i] = make_float4(q.x, q.y, q.z, l.w);
}

// ---------------------------------------------------------------- PCISPH

// predictVelocityAndPositionImpl (Fluid_3D_PCISPH.cu:32-86): the predicted
// position / velocity (into Q, W) or, at the end of a substep, the actual
// ones (into P, V); the acceleration is the gravity.
__device__ __forceinline__ void pci_wall(float& q, float& v, float md, float hi) {
  if (q < md) { q = md; v = mul(v, -0.0f); }
  if (q > hi) { q = hi; v = mul(v, -0.0f); }
}

__global__ void __launch_bounds__(256) k_pci_predict(SphParams p, float4* __restrict__ P, float4* __restrict__ V,
                                                    float4* __restrict__ Q, float4* __restrict__ W,
                                                    const float4* __restrict__ F, int actual, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 q = P[i], v = V[i], f = F[i];
  float vx = add(v.x, mul(add(p.g.x, f.x), p.dt)), vy = add(v.y, mul(add(p.g.y, f.y), p.dt)),
        vz = add(v.z, mul(add(p.g.z, f.z), p.dt));
  float px = add(q.x, mul(vx, p.dt)), py = add(q.y, mul(vy, p.dt)), pz = add(q.z, mul(vz, p.dt));
  const float hi = sub(p.size, p.md);
  pci_wall(px, vx, p.md, hi);
  pci_wall(py, vy, p.md, hi);
  pci_wall(pz, vz, p.md, hi);
  if (actual) {
    P[i] = make_float4(px, py, pz, q.w);
    V[i] = make_float4(vx, vy, vz, v.w);
  } else {
    Q[i] = make_float4(px, py, pz, 0.f);
    W[i] = make_float4(vx, vy, vz, W[i].w);
  }
}

// predictDensityAndPressureImpl (Fluid_3D_PCISPH.cu:88-159): cells from the
// position, distances from the predicted positions; pressure += 50 * (density
// - rest density), the coefficient the kernel ends with.  Writes the density
// into V.w, the pressure into W.w, R = (predicted position, p / rho^2) and, on
// the rest-density pass, P.w.
__global__ void __launch_bounds__(kThreads) k_pci_density(SphParams p, const int* __restrict__ off,
                                                         float4* __restrict__ P, float4* __restrict__ V,
                                                         const float4* __restrict__ Q, float4* __restrict__ W,
                                                         float4* __restrict__ R, int* __restrict__ count,
                                                         int* __restrict__ lists, int set_rest, int n) {
  __shared__ WalkShared<1> sm;
  const int i = (blockIdx.x * kThreads + threadIdx.x) >> 2;
  const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
  const float4 me = i < n ? P[i] : none, pq = i < n ? Q[i] : none;
  float s[2];
  const int found = walk<1>(
      p, cell_of(p, me.x, me.y, me.z), i < n, off, lists ? lists + (size_t)i * kSphList : nullptr, sm, s,
      [&](int j) {
        const float4 o = __ldg(Q + j);
        return !outside(dot3(sub(pq.x, o.x), sub(pq.y, o.y), sub(pq.z, o.z)), p);
      },
      [&](int j, float (&t)[1]) {
        const float4 o = __ldg(Q + j);
        t[0] = poly6(dot3(sub(pq.x, o.x), sub(pq.y, o.y), sub(pq.z, o.z)), p);
      });
  if ((threadIdx.x & 3) || i >= n) return;
  if (count) count[i] = found;
  const float density = s[0];
  const float err = sub(density, me.w);
  const float pressure = add(W[i].w, mul(50.0f, err));
  V[i].w = density;
  W[i].w = pressure;
  if (set_rest) P[i].w = density;
  R[i] = make_float4(pq.x, pq.y, pq.z, dvd(pressure, mul(density, density)));
}

// computePressureForceImpl (Fluid_3D_PCISPH.cu:161-202); the reference
// subtracts each term, and adding its negative rounds the same.
__global__ void __launch_bounds__(kThreads) k_pci_force(SphParams p, const int* __restrict__ off,
                                                       const float4* __restrict__ P, const float4* __restrict__ R,
                                                       float4* __restrict__ F, const int* __restrict__ count,
                                                       const int* __restrict__ lists, int n) {
  __shared__ WalkShared<3> sm;
  const int i = (blockIdx.x * kThreads + threadIdx.x) >> 2;
  const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
  const float4 me = i < n ? P[i] : none, r = i < n ? R[i] : none;
  float s[2];
  walk_kept<3>(
      p, cell_of(p, me.x, me.y, me.z), i, i < n, off, count, lists, sm, s,
      [&](int j) {
        const float4 o = __ldg(R + j);
        return !outside(dot3(sub(r.x, o.x), sub(r.y, o.y), sub(r.z, o.z)), p);
      },
      [&](int j, float (&t)[3]) {
        const float4 o = __ldg(R + j);
        const float dx = sub(r.x, o.x), dy = sub(r.y, o.y), dz = sub(r.z, o.z);
        const float3 w = spikey(dx, dy, dz, dot3(dx, dy, dz), p);
        const float q = add(o.w, r.w);
        t[0] = -mul(w.x, q);
        t[1] = -mul(w.y, q);
        t[2] = -mul(w.z, q);
      });
  const int first = threadIdx.x & 28;
  const float fy = __shfl_sync(0xffffffffu, s[0], first + 1), fz = __shfl_sync(0xffffffffu, s[0], first + 2);
  if ((threadIdx.x & 3) || i >= n) return;
  F[i] = make_float4(s[0], fy, fz, 0.f);
}

// initPressureImpl (Fluid_3D_PCISPH.cu:22-30): pressure and pressure force 0.
__global__ void __launch_bounds__(256) k_pci_init(float4* __restrict__ W, float4* __restrict__ F, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  W[i].w = 0.f;
  F[i] = make_float4(0.f, 0.f, 0.f, 0.f);
}

__global__ void __launch_bounds__(256) k_sph_planes(const float4* __restrict__ a, float* __restrict__ planes, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 v = a[i];
  const size_t m = (size_t)n;
  planes[i] = v.x;
  planes[m + i] = v.y;
  planes[2 * m + i] = v.z;
  planes[3 * m + i] = v.w;
}

}  // namespace

cudaError_t launch_sph_planes(cudaStream_t st, const float4* a, float* planes, int n) {
  if (n <= 0) return cudaSuccess;
  k_sph_planes<<<blocks(n, 256), 256, 0, st>>>(a, planes, n);
  return cudaGetLastError();
}

cudaError_t launch_sph_keys(cudaStream_t st, const SphParams& p, const float4* pos, int* key, int* slot, int* count,
                            int n) {
  if (n <= 0) return cudaSuccess;
  k_sph_keys<<<blocks(n, 256), 256, 0, st>>>(p, pos, key, slot, count, n);
  return cudaGetLastError();
}

cudaError_t launch_sph_gather(cudaStream_t st, const int* key, const int* off, const int* perm_u, const SphArrays& src,
                              const SphArrays& dst, int n) {
  if (n <= 0) return cudaSuccess;
  k_sph_gather<<<blocks(n, 256), 256, 0, st>>>(key, off, perm_u, src, dst, n);
  return cudaGetLastError();
}

cudaError_t launch_pbf_predict(cudaStream_t st, const SphParams& p, float4* P, const float4* L, float4* V, int n) {
  if (n <= 0) return cudaSuccess;
  k_pbf_predict<<<blocks(n, 256), 256, 0, st>>>(p, P, L, V, n);
  return cudaGetLastError();
}

cudaError_t launch_pbf_lambda(cudaStream_t st, const SphParams& p, const int* off, float4* P, float4* V, float4* Q,
                              int* count, int* lists, bool set_rest, int n) {
  if (n <= 0) return cudaSuccess;
  k_pbf_lambda<<<blocks(n, kPart), kThreads, 0, st>>>(p, off, P, V, Q, count, lists, set_rest ? 1 : 0, n);
  return cudaGetLastError();
}

cudaError_t launch_pbf_delta(cudaStream_t st, const SphParams& p, const int* off, const float4* Q, float4* P,
                             const int* count, const int* lists, int n) {
  if (n <= 0) return cudaSuccess;
  k_pbf_delta<<<blocks(n, kPart), kThreads, 0, st>>>(p, off, Q, P, count, lists, n);
  return cudaGetLastError();
}

cudaError_t launch_pbf_update(cudaStream_t st, const SphParams& p, const float4* P, float4* L, float4* V, int n) {
  if (n <= 0) return cudaSuccess;
  k_pbf_update<<<blocks(n, 256), 256, 0, st>>>(p, P, L, V, n);
  return cudaGetLastError();
}

cudaError_t launch_pci_init(cudaStream_t st, float4* W, float4* F, int n) {
  if (n <= 0) return cudaSuccess;
  k_pci_init<<<blocks(n, 256), 256, 0, st>>>(W, F, n);
  return cudaGetLastError();
}

cudaError_t launch_pci_predict(cudaStream_t st, const SphParams& p, float4* P, float4* V, float4* Q, float4* W,
                               const float4* F, bool actual, int n) {
  if (n <= 0) return cudaSuccess;
  k_pci_predict<<<blocks(n, 256), 256, 0, st>>>(p, P, V, Q, W, F, actual ? 1 : 0, n);
  return cudaGetLastError();
}

cudaError_t launch_pci_density(cudaStream_t st, const SphParams& p, const int* off, float4* P, float4* V,
                               const float4* Q, float4* W, float4* R, int* count, int* lists, bool set_rest, int n) {
  if (n <= 0) return cudaSuccess;
  k_pci_density<<<blocks(n, kPart), kThreads, 0, st>>>(p, off, P, V, Q, W, R, count, lists, set_rest ? 1 : 0, n);
  return cudaGetLastError();
}

cudaError_t launch_pci_force(cudaStream_t st, const SphParams& p, const int* off, const float4* P, const float4* R,
                             float4* F, const int* count, const int* lists, int n) {
  if (n <= 0) return cudaSuccess;
  k_pci_force<<<blocks(n, kPart), kThreads, 0, st>>>(p, off, P, R, F, count, lists, n);
  return cudaGetLastError();
}

}  // namespace aqb
