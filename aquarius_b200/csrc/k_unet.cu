// Kernels of the learned pressure warm start: a small 3D U-Net in BF16 with
// FP32 accumulation.  No counterpart in the reference.
//
// Activations are channels-last over the cell layout: element (x,y,z,c) of a
// grid s = (sx,sy,sz) with C channels is at ((x*sy + y)*sz + z)*C + c.
// Convolutions are 3x3x3, stride 1, zero padding 1, as implicit GEMMs on the
// tensor cores (mma.sync m16n8k16, bf16 x bf16 -> f32):
//   forward   out[v][co] = act(b[co] + sum_t sum_ci in[v + o_t][ci] w[t][co][ci])
//             M = voxels, N = Cout, K = 27 taps x Cin; operands staged in shared
//             memory by cp.async (zero fill outside the grid), fragments by ldmatrix.
//   data grad the forward kernel on dY with the flipped, transposed weights
//             w'[t][ci][co] = w[26-t][co][ci].
//   weight grad dw[t][co][ci] = sum_v dY[v][co] x[v + o_t][ci]: M = Cout, N = Cin,
//             K = voxels, per (tap, voxel chunk) partial sums reduced in a fixed
//             order (deterministic).
// Tap t = (dx+1)*9 + (dy+1)*3 + (dz+1).
#include <cuda_bf16.h>

#include <algorithm>

#include "aq_kernels.cuh"

namespace aqb {
namespace {

using bf16 = __nv_bfloat16;

// Forward convolution variant: 2 = tcgen05 UMMA where its operands fit in
// shared memory, else halo-tiled mma.sync (default); 1 = halo-tiled
// mma.sync; 0 = im2col streaming mma.sync.
int g_conv_impl = 2;

constexpr int kTileM = 128;  // voxels per forward CTA (4 warps x 32)
constexpr int kRowK = 24;    // smem row of one 16-wide k chunk: 16 + 8 pad bf16 (48 B, conflict-free ldmatrix)

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool pred) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  const int n = pred ? 16 : 0;  // n = 0: no bytes read, 16 zero bytes written
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(n));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

__device__ __forceinline__ void ldsm_x4(unsigned (&r)[4], const void* p) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(s));
}
__device__ __forceinline__ void ldsm_x2(unsigned (&r)[2], const void* p) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];\n" : "=r"(r[0]), "=r"(r[1]) : "r"(s));
}
__device__ __forceinline__ void ldsm_x4_t(unsigned (&r)[4], const void* p) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(s));
}
__device__ __forceinline__ void ldsm_x2_t(unsigned (&r)[2], const void* p) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];\n" : "=r"(r[0]), "=r"(r[1]) : "r"(s));
}

// d += a * b, m16n8k16, bf16 inputs, f32 accumulators
__device__ __forceinline__ void mma_bf16(float (&d)[4], const unsigned (&a)[4], const unsigned (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ void tap_offset(int tap, int& dx, int& dy, int& dz) {
  dx = tap / 9 - 1;
  dy = (tap / 3) % 3 - 1;
  dz = tap % 3 - 1;
}

// ------------------------------------------------------------------ forward
// 128 threads; CTA = 128 consecutive voxels x all COUT channels; warp w owns
// voxels [32w, 32w+32) as two m16 tiles.  K steps: 27 taps x CIN/16 chunks,
// double-buffered in shared memory.
template <int CIN, int COUT, bool RELU, bool BIAS>
__global__ void __launch_bounds__(128) k_conv3_fwd(const bf16* __restrict__ in, const bf16* __restrict__ w,
                                                  const float* __restrict__ bias, bf16* __restrict__ out, int sx,
                                                  int sy, int sz) {
  static_assert(CIN % 16 == 0 && COUT % 8 == 0, "channel counts");
  constexpr int KC = CIN / 16;
  constexpr int STEPS = 27 * KC;
  constexpr int NT = COUT / 8;
  __shared__ __align__(16) bf16 sA[2][kTileM * kRowK];
  __shared__ __align__(16) bf16 sB[2][COUT * kRowK];
  const int V = sx * sy * sz;
  const int m0 = blockIdx.x * kTileM;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int v = m0 + tid;  // the A row this thread stages
  const bool vin = v < V;
  int vx = 0, vy = 0, vz = 0;
  if (vin) {
    vz = v % sz;
    const int t = v / sz;
    vy = t % sy;
    vx = t / sy;
  }
  auto stage = [&](int step, int buf) {
    const int tap = step / KC, kc = step % KC;
    int dx, dy, dz;
    tap_offset(tap, dx, dy, dz);
    const int nx = vx + dx, ny = vy + dy, nz = vz + dz;
    const bool ok = vin && nx >= 0 && nx < sx && ny >= 0 && ny < sy && nz >= 0 && nz < sz;
    const bf16* src = ok ? in + ((size_t)((nx * sy + ny) * sz + nz) * CIN + kc * 16) : in;
    bf16* dst = &sA[buf][tid * kRowK];
    cp_async16(dst, src, ok);
    cp_async16(dst + 8, ok ? src + 8 : in, ok);
    for (int i = tid; i < COUT * 2; i += 128) {
      const int n = i >> 1, h = i & 1;
      cp_async16(&sB[buf][n * kRowK + h * 8], w + ((size_t)(tap * COUT + n) * CIN + kc * 16 + h * 8), true);
    }
  };
  float acc[2][NT][4];
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < NT; ++b)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[a][b][c] = 0.f;
  stage(0, 0);
  cp_async_commit();
  for (int step = 0; step < STEPS; ++step) {
    const int buf = step & 1;
    if (step + 1 < STEPS) stage(step + 1, buf ^ 1);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
    unsigned bfr[NT][2];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) ldsm_x2(bfr[nt], &sB[buf][(nt * 8 + (lane & 7)) * kRowK + ((lane >> 3) & 1) * 8]);
#pragma unroll
    for (int mt = 0; mt < 2; ++mt) {
      unsigned afr[4];
      ldsm_x4(afr, &sA[buf][(warp * 32 + mt * 16 + (lane & 15)) * kRowK + (lane >> 4) * 8]);
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) mma_bf16(acc[mt][nt], afr, bfr[nt]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      const int co = nt * 8 + (lane & 3) * 2;
      const float b0 = BIAS ? bias[co] : 0.f, b1 = BIAS ? bias[co + 1] : 0.f;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = m0 + warp * 32 + mt * 16 + (lane >> 2) + h * 8;
        if (r < V) {
          float a = acc[mt][nt][2 * h] + b0, c = acc[mt][nt][2 * h + 1] + b1;
          if (RELU) {
            a = fmaxf(a, 0.f);
            c = fmaxf(c, 0.f);
          }
          *reinterpret_cast<__nv_bfloat162*>(out + (size_t)r * COUT + co) = __floats2bfloat162_rn(a, c);
        }
      }
    }
}

// Halo-tiled forward: a CTA computes a 4 (x) x 4 (y) x 16 (z) block of
// output voxels.  The input block with its one-voxel halo (6 x 6 x 18
// voxels x CIN channels) is staged in shared memory once (cp.async, zero
// fill outside the grid); every tap then gathers its A fragments straight
// from that block with ldmatrix (each lane addresses its own voxel row), so
// the input is read ~2.5x instead of 27x.  Weights stream per tap, double
// buffered.  8 warps; m tile j = 16 z voxels at (x, y) = (j / 4, j % 4),
// warp w owns tiles 2w and 2w+1.  Rows are padded by 16 B (odd count of 16 B
// chunks: ldmatrix without bank conflicts).
constexpr int kTX = 4, kTY = 4, kTZ = 16;
constexpr int kHX = kTX + 2, kHY = kTY + 2, kHZ = kTZ + 2, kHalo = kHX * kHY * kHZ;

template <int CIN, int COUT>
constexpr size_t fwd_tile_smem() {
  return (size_t)kHalo * (CIN + 8) * sizeof(bf16) + (size_t)2 * COUT * (CIN + 8) * sizeof(bf16);
}

template <int CIN, int COUT, bool RELU, bool BIAS>
__global__ void __launch_bounds__(256) k_conv3_fwd_tile(const bf16* __restrict__ in, const bf16* __restrict__ w,
                                                       const float* __restrict__ bias, bf16* __restrict__ out,
                                                       int sx, int sy, int sz) {
  static_assert(CIN % 16 == 0 && COUT % 8 == 0, "channel counts");
  constexpr int RS = CIN + 8;  // row stride (bf16)
  constexpr int KS = CIN / 16, NT = COUT / 8, CH = CIN / 8;
  extern __shared__ __align__(16) unsigned char ft_smem[];
  bf16* sH = reinterpret_cast<bf16*>(ft_smem);
  bf16* sW = sH + kHalo * RS;  // [2][COUT][RS]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int z0 = blockIdx.x * kTZ, y0 = blockIdx.y * kTY, x0 = blockIdx.z * kTX;
  // stage the halo block
  for (int i = tid; i < kHalo * CH; i += 256) {
    const int c = i % CH, h = i / CH;
    const int hz = h % kHZ, t = h / kHZ, hy = t % kHY, hx = t / kHY;
    const int gx = x0 + hx - 1, gy = y0 + hy - 1, gz = z0 + hz - 1;
    const bool ok = gx >= 0 && gx < sx && gy >= 0 && gy < sy && gz >= 0 && gz < sz;
    cp_async16(sH + h * RS + c * 8, ok ? in + ((size_t)((gx * sy + gy) * sz + gz) * CIN + c * 8) : in, ok);
  }
  auto stage_w = [&](int tap, int buf) {
    bf16* dst = sW + buf * COUT * RS;
    for (int i = tid; i < COUT * CH; i += 256) {
      const int c = i % CH, n = i / CH;
      cp_async16(dst + n * RS + c * 8, w + ((size_t)(tap * COUT + n) * CIN + c * 8), true);
    }
  };
  stage_w(0, 0);
  cp_async_commit();
  float acc[2][NT][4];
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < NT; ++b)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[a][b][c] = 0.f;
  for (int tap = 0; tap < 27; ++tap) {
    const int buf = tap & 1;
    if (tap + 1 < 27) stage_w(tap + 1, buf ^ 1);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
    int dx, dy, dz;
    tap_offset(tap, dx, dy, dz);
    const bf16* wb = sW + buf * COUT * RS;
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
      unsigned bfr[NT][2];
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) ldsm_x2(bfr[nt], wb + (nt * 8 + (lane & 7)) * RS + ks * 16 + ((lane >> 3) & 1) * 8);
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) {
        const int j = warp * 2 + mt;
        const int ox = j >> 2, oy = j & 3;
        const int h = ((ox + dx + 1) * kHY + (oy + dy + 1)) * kHZ + (lane & 15) + dz + 1;
        unsigned afr[4];
        ldsm_x4(afr, sH + h * RS + ks * 16 + (lane >> 4) * 8);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) mma_bf16(acc[mt][nt], afr, bfr[nt]);
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int mt = 0; mt < 2; ++mt) {
    const int j = warp * 2 + mt;
    const int gx = x0 + (j >> 2), gy = y0 + (j & 3);
    if (gx >= sx || gy >= sy) continue;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      const int co = nt * 8 + (lane & 3) * 2;
      const float b0 = BIAS ? bias[co] : 0.f, b1 = BIAS ? bias[co + 1] : 0.f;
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        const int gz = z0 + (lane >> 2) + hh * 8;
        if (gz < sz) {
          float a = acc[mt][nt][2 * hh] + b0, c = acc[mt][nt][2 * hh + 1] + b1;
          if (RELU) {
            a = fmaxf(a, 0.f);
            c = fmaxf(c, 0.f);
          }
          *reinterpret_cast<__nv_bfloat162*>(out + (size_t)((gx * sy + gy) * sz + gz) * COUT + co) =
              __floats2bfloat162_rn(a, c);
        }
      }
    }
  }
}

// ------------------------------------------------- forward on tcgen05 (TMEM)
// UMMA implicit GEMM: D[voxels x COUT] (f32, TMEM) += A[voxels x 16 channels]
// x B[16 channels x COUT] per tap and k step, bf16 operands in shared memory
// read through matrix descriptors (canonical K-major layout, no swizzle:
// 8-row x 16-byte core matrices), tcgen05.mma.cta_group::1.kind::f16 issued by
// one thread, completion through tcgen05.commit on an mbarrier whose wait is
// bounded (a timeout is recorded in g_umma_timeout; the kernel then frees its
// TMEM without storing), results read back with tcgen05.ld.
__device__ int g_umma_timeout;
// Test hook of the bounded wait: when set, the issuing thread neither issues
// the MMAs nor commits (nothing is left in flight), so every thread's wait
// runs out; g_umma_wait_ns bounds the wait (default one second).
__device__ int g_umma_test_skip;
__device__ unsigned long long g_umma_wait_ns = 1000000000ull;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor: start, leading (K) and stride (M/N) byte
// offsets of the core matrices, the fixed version bits 46-47 = 1, no swizzle.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) |
         (1ull << 46);
}

// Instruction descriptor, kind::f16: D f32, A and B bf16, both K-major, N, M.
__host__ __device__ constexpr uint32_t umma_idesc(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(acc));
}

__device__ __forceinline__ void umma_commit(uint64_t* mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(smem_u32(mbar))
               : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* mbar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n.reg .pred P1;\nmbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\nselp.b32 %0, 1, 0, P1;\n}\n"
      : "=r"(done)
      : "r"(smem_u32(mbar)), "r"(parity)
      : "memory");
  return done != 0;
}

__device__ __forceinline__ unsigned long long umma_now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Bounded wait on an mbarrier phase; false (and the timeout recorded) if it
// does not complete within g_umma_wait_ns or 2^22 polls, whichever is first.
__device__ __forceinline__ bool mbar_wait(uint64_t* mbar, uint32_t parity) {
  const unsigned long long t0 = umma_now_ns(), limit = g_umma_wait_ns;
  for (int i = 0; i < (1 << 22); ++i) {
    if (mbar_try_wait(mbar, parity)) return true;
    if ((i & 255) == 255 && umma_now_ns() - t0 > limit) break;
  }
  atomicExch(&g_umma_timeout, 1);
  return false;
}

// 16 consecutive f32 columns of this thread's TMEM lane (32x32b shape).
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// 16 columns of this thread's TMEM lane set to 0 (tcgen05.wait::st follows).
__device__ __forceinline__ void tmem_zero16(uint32_t taddr) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};\n" ::"r"(taddr),
      "r"(0u)
      : "memory");
}

__host__ __device__ constexpr int tmem_cols(int n) {
  return n <= 32 ? 32 : n <= 64 ? 64 : n <= 128 ? 128 : n <= 256 ? 256 : 512;
}

// The tcgen05 kernel: a CTA owns a column of 16 (y) x 8 (z) voxels, an M = 128
// tile per x plane (row m = 8 y + z), and marches over `planes` of them.  A
// halo plane (18 x 10 voxels) is stored per 8-channel chunk as z columns of 10
// rows of 16 B: the A operand of any (dy, dz) is then a descriptor into the
// plane itself - rows of a core matrix are 8 consecutive z (16 B apart), the
// 16 core matrices along M are the y columns (SBO = 160 B), the two along K the
// chunks (LBO) - so no per-tap copy.  Halo plane h feeds the output planes
// h - 2, h - 1 and h, whose accumulators are neighbours in TMEM: one MMA with
// N = 3 COUT takes the three dx of a (dy, dz), as reading A (128 rows for every
// MMA, 32 cycles) bounds the narrow layers.  An accumulator still takes its taps
// in the order dx, dy, dz, the same bits as one MMA a tap.  MMAs are ordered
// among themselves only where they share accumulator and shape, so the
// accumulators are cleared first (every MMA of a halo plane then has that
// plane's window of columns and its N), and a plane's MMAs are issued when the
// plane before, whose window overlaps, has completed.  Four planes are in
// shared memory: two being loaded, one whose MMAs run, one that waits; finished
// output planes are written meanwhile.  The weights are loaded once a CTA.
// 128^3 in us, against a CTA that loaded a 2-plane halo and all weights, issued
// an MMA a tap and stored: 48 -> 16 channels 427 -> 219 (400 with the wide MMAs
// alone), 16 -> 16 148 -> 96, 64^3 32 -> 32 82 -> 41; the network's inference
// 1.23 -> 0.78 ms.
constexpr int kUY = 16, kUZ = 8;
constexpr int kUHY = kUY + 2, kUHZ = kUZ + 2;
constexpr int kUChunk = kUHY * kUHZ * 16;  // bytes of one 8-channel chunk of a halo plane
constexpr int kUSlots = 4;                 // halo planes in shared memory

template <int CIN, int COUT>
__host__ __device__ constexpr size_t fwd_umma_smem() {
  return (size_t)kUSlots * (CIN / 8) * kUChunk + (size_t)27 * COUT * CIN * 2 + 1024;
}

// CTAs an SM holds (shared memory, and 4 by registers) and the output planes
// that its share of the 512 TMEM columns holds.
template <int CIN, int COUT>
__host__ __device__ constexpr int umma_ctas() {
  const size_t s = fwd_umma_smem<CIN, COUT>() + 1024;
  return s * 4 <= 227 * 1024 && COUT <= 16 ? 4 : s * 2 <= 227 * 1024 ? 2 : 1;
}
template <int CIN, int COUT>
__host__ __device__ constexpr int umma_planes() {
  return 512 / umma_ctas<CIN, COUT>() / COUT;
}

// The pairs the tcgen05 kernel takes: cout a multiple of 16 (UMMA N), the
// halo and all weights resident.
template <int CIN, int COUT>
__host__ __device__ constexpr bool umma_fits() {
  return COUT % 16 == 0 && COUT <= 80 && fwd_umma_smem<CIN, COUT>() <= 200 * 1024;
}

// SKIP > 0: the input's last SKIP channels are read from `skip`, the others from
// `in` at half the resolution (the concatenation that k_upcat writes, without
// writing it: 128^3, 32 + 16 channels, 236 us against 67 + 219).
template <int CIN, int COUT, bool RELU, bool BIAS, int SKIP = 0>
__global__ void __launch_bounds__(256) k_conv3_fwd_umma(const bf16* __restrict__ in, const bf16* __restrict__ skip,
                                                       const bf16* __restrict__ w, const float* __restrict__ bias,
                                                       bf16* __restrict__ out, int sx, int sy, int sz, int planes) {
  static_assert(umma_fits<CIN, COUT>(), "UMMA shapes: M = 128, N = COUT .. 3 COUT, operands resident");
  constexpr int CH = CIN / 8, KS = CIN / 16;
  constexpr int SLOT = CH * kUChunk;
  constexpr int TAPB = COUT * CIN * 2;  // one tap's weights
  constexpr int COLS = tmem_cols(umma_planes<CIN, COUT>() * COUT);
  extern __shared__ __align__(1024) unsigned char um_smem[];
  unsigned char* sH = um_smem;                  // [kUSlots][CH][kUHY][kUHZ][16 B]
  unsigned char* sB = um_smem + kUSlots * SLOT;  // [9 (dy, dz)][canonical 3 COUT x CIN]
  __shared__ __align__(8) uint64_t s_mbar[kUSlots];
  __shared__ uint32_t s_tmem;
  const int tid = threadIdx.x, warp = tid >> 5;
  const int z0 = blockIdx.x * kUZ, y0 = blockIdx.y * kUY, x0 = blockIdx.z * planes;
  const int n = min(planes, sx - x0);  // output planes; halo planes 0 .. n + 1
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&s_tmem)),
                 "r"(COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  if (tid == 0) {
    for (int i = 0; i < kUSlots; ++i)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(&s_mbar[i])), "r"(1));
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  // halo plane h, zero outside the grid, as one copy group (an empty one past the last)
  auto load = [&](int h) {
    if (h < n + 2) {
      const int gx = x0 + h - 1;
      unsigned char* const slot = sH + (h % kUSlots) * SLOT;
      for (int i = tid; i < kUHY * kUHZ * CH; i += 256) {
        const int c = i % CH, t = i / CH, gy = y0 + t / kUHZ - 1, gz = z0 + t % kUHZ - 1;
        const bool ok = gx >= 0 && gx < sx && gy >= 0 && gy < sy && gz >= 0 && gz < sz;
        const bf16* src = in;
        if (ok) {
          constexpr int CU = CIN - SKIP;
          const size_t v = (size_t)(gx * sy + gy) * sz + gz;
          if (SKIP == 0) src = in + v * CIN + c * 8;
          else if (c * 8 < CU) src = in + ((size_t)((gx >> 1) * (sy >> 1) + (gy >> 1)) * (sz >> 1) + (gz >> 1)) * CU + c * 8;
          else src = skip + v * SKIP + (c * 8 - CU);
        }
        cp_async16(slot + c * kUChunk + t * 16, src, ok);
      }
    }
    cp_async_commit();
  };
  // all weights: of (dy, dz) the rows of dx = +1, 0, -1, in the canonical
  // K-major layout (with plane 0's copy group)
  for (int i = tid; i < 27 * COUT * CH; i += 256) {
    const int c = i % CH, r = (i / CH) % COUT, t = i / (CH * COUT);
    const int row = (2 - t / 9) * COUT + r;
    cp_async16(sB + (t % 9) * (3 * TAPB) + (c >> 1) * (3 * COUT * 32) + (row >> 3) * 256 + (c & 1) * 128 + (row & 7) * 16,
               w + ((size_t)(t * COUT + r) * CIN + c * 8), true);
  }
  load(0);
  load(1);
  const uint32_t h0 = smem_u32(sH), b0 = smem_u32(sB);
  // warp w reads TMEM lanes 32 (w % 4) .., channels 16 (w / 4) and on in steps
  // of 32 (of every other plane where COUT is 16): row m -> (y, z)
  const int m = (warp & 3) * 32 + (tid & 31);
  const int gy = y0 + (m >> 3), gz = z0 + (m & 7);
  // the accumulators start at zero, so that every MMA adds
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem = s_tmem;
  for (int c0 = (warp >> 2) * 16; c0 < n * COUT; c0 += 32)
    tmem_zero16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0);
  asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
  auto store_plane = [&](int q) {
    const bool store = gy < sy && gz < sz;
    const uint32_t trow = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(q * COUT);
    bf16* dst = out + (size_t)(((x0 + q) * sy + gy) * sz + gz) * COUT;
    if (COUT == 16 && (q & 1) != (warp >> 2)) return;
#pragma unroll
    for (int cb = 0; cb < COUT; cb += 32) {
      const int c0 = COUT == 16 ? 0 : cb + (warp >> 2) * 16;
      if (c0 < COUT) {
        float v[16];
        tmem_ld16(trow + (uint32_t)c0, v);
        if (store) {
          __align__(16) __nv_bfloat162 pk[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            float a = v[2 * q] + (BIAS ? bias[c0 + 2 * q] : 0.f), b = v[2 * q + 1] + (BIAS ? bias[c0 + 2 * q + 1] : 0.f);
            if (RELU) {
              a = fmaxf(a, 0.f);
              b = fmaxf(b, 0.f);
            }
            pk[q] = __floats2bfloat162_rn(a, b);
          }
          uint4* d4 = reinterpret_cast<uint4*>(dst + c0);
          d4[0] = reinterpret_cast<const uint4*>(pk)[0];
          d4[1] = reinterpret_cast<const uint4*>(pk)[1];
        }
      }
    }
  };
  // wait until the products of halo plane h are done (the last wait of a slot's
  // barrier before its next use, so the parity tells them apart).  The warp's
  // lanes decide together: what follows reads TMEM, which takes whole warps.
  auto wait_plane = [&](int h) {
    const bool ok = __all_sync(0xffffffffu, mbar_wait(&s_mbar[h % kUSlots], (uint32_t)((h / kUSlots) & 1)));
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    return ok;
  };
  bool ok = true;
  for (int h = 0; h < n + 2; ++h) {
    // the slot of plane h - 2 is free once its products are done, which also
    // completes output plane h - 4
    if (h >= 2) ok = wait_plane(h - 2);
    load(h + 2);
    if (ok && h >= 4) store_plane(h - 4);
    cp_async_wait<2>();
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    ok = __syncthreads_and(ok);
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    if (!ok) break;  // a wait ran out (flagged); the same for every thread
    // the products of plane h - 1 first: the accumulators' window moves on
    const bool go = warp == 0 && (h == 0 || wait_plane(h - 1));
    if (tid == 0 && go && !g_umma_test_skip) {
      // halo plane h feeds the output planes lo .. hi, whose accumulators are neighbours
      const int lo = max(h - 2, 0), hi = min(h, n - 1);
      const uint32_t idesc = umma_idesc(128, (hi - lo + 1) * COUT);
      const uint32_t d_lo = tmem + (uint32_t)(lo * COUT), b_lo = b0 + (uint32_t)((lo - h + 2) * (COUT * 32));
      const uint32_t ah = h0 + (uint32_t)((h % kUSlots) * SLOT);
#pragma unroll 1
      for (int g = 0; g < 9; ++g) {
        const uint32_t a0 = ah + (uint32_t)(((g / 3) * kUHZ + g % 3) * 16);
        const uint32_t bg = b_lo + (uint32_t)(g * (3 * TAPB));
#pragma unroll
        for (int ks = 0; ks < KS; ++ks)
          umma_f16(d_lo, umma_desc(a0 + (uint32_t)(2 * ks * kUChunk), kUChunk, kUHZ * 16),
                   umma_desc(bg + (uint32_t)(ks * (3 * COUT * 32)), 128, 256), idesc, 1u);
      }
      umma_commit(&s_mbar[h % kUSlots]);
    }
  }
  cp_async_wait<0>();
  if (ok) ok = wait_plane(n);
  if (ok && n >= 2) store_plane(n - 2);
  if (ok) ok = wait_plane(n + 1);
  if (ok) store_plane(n - 1);
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(COLS));
  }
}

// ------------------------------------------------------------- weight grad
// grid (chunks, 27): one tap, `cv` voxels per CTA in tiles of 128.  A = dY^T
// (COUT x voxels), B = x shifted by the tap (voxels x CIN); both staged with
// voxels as rows and read transposed by ldmatrix.trans.  Warp w owns the
// n tiles nt = w, w+4, ...
template <int CIN, int COUT>
__global__ void __launch_bounds__(128) k_conv3_wgrad(const bf16* __restrict__ x, const bf16* __restrict__ dy,
                                                    float* __restrict__ part, int sx, int sy, int sz, int cv) {
  static_assert(CIN % 16 == 0 && COUT % 16 == 0, "channel counts");
  constexpr int RX = CIN + 8, RD = COUT + 8;  // padded smem rows (odd count of 16 B chunks)
  constexpr int MT = COUT / 16, NTT = CIN / 8, NTW = (NTT + 3) / 4;
  extern __shared__ __align__(16) unsigned char wg_smem[];
  bf16(*sX)[kTileM * RX] = reinterpret_cast<bf16(*)[kTileM * RX]>(wg_smem);
  bf16(*sD)[kTileM * RD] = reinterpret_cast<bf16(*)[kTileM * RD]>(wg_smem + 2 * kTileM * RX * sizeof(bf16));
  const int V = sx * sy * sz;
  const int tap = blockIdx.y;
  int dx, dy_, dz;
  tap_offset(tap, dx, dy_, dz);
  const int v0 = blockIdx.x * cv, v1 = min(V, v0 + cv);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tiles = (v1 - v0 + kTileM - 1) / kTileM;
  auto stage = [&](int tile, int buf) {
    const int base = v0 + tile * kTileM;
    // x rows: CIN/8 chunks each
    for (int i = tid; i < kTileM * (CIN / 8); i += 128) {
      const int r = i / (CIN / 8), c = i % (CIN / 8);
      const int v = base + r;
      bool ok = v < v1;
      const bf16* src = x;
      if (ok) {
        const int vz = v % sz, t = v / sz, vy = t % sy, vx = t / sy;
        const int nx = vx + dx, ny = vy + dy_, nz = vz + dz;
        ok = nx >= 0 && nx < sx && ny >= 0 && ny < sy && nz >= 0 && nz < sz;
        if (ok) src = x + ((size_t)((nx * sy + ny) * sz + nz) * CIN + c * 8);
      }
      cp_async16(&sX[buf][r * RX + c * 8], src, ok);
    }
    for (int i = tid; i < kTileM * (COUT / 8); i += 128) {
      const int r = i / (COUT / 8), c = i % (COUT / 8);
      const int v = base + r;
      const bool ok = v < v1;
      cp_async16(&sD[buf][r * RD + c * 8], ok ? dy + ((size_t)v * COUT + c * 8) : dy, ok);
    }
  };
  float acc[MT][NTW][4];
#pragma unroll
  for (int a = 0; a < MT; ++a)
#pragma unroll
    for (int b = 0; b < NTW; ++b)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[a][b][c] = 0.f;
  if (tiles > 0) stage(0, 0);
  cp_async_commit();
  for (int tile = 0; tile < tiles; ++tile) {
    const int buf = tile & 1;
    if (tile + 1 < tiles) stage(tile + 1, buf ^ 1);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
#pragma unroll
    for (int k0 = 0; k0 < kTileM; k0 += 16) {
      unsigned afr[MT][4];
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
        ldsm_x4_t(afr[mt], &sD[buf][(k0 + (lane & 7) + (lane >> 4) * 8) * RD + mt * 16 + ((lane >> 3) & 1) * 8]);
#pragma unroll
      for (int j = 0; j < NTW; ++j) {
        const int nt = warp + 4 * j;
        if (nt < NTT) {
          unsigned bfr[2];
          ldsm_x2_t(bfr, &sX[buf][(k0 + (lane & 15)) * RX + nt * 8]);
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) mma_bf16(acc[mt][j], afr[mt], bfr);
        }
      }
    }
    __syncthreads();
  }
  float* dst = part + ((size_t)blockIdx.x * 27 + tap) * COUT * CIN;
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int j = 0; j < NTW; ++j) {
      const int nt = warp + 4 * j;
      if (nt < NTT) {
        const int ci = nt * 8 + (lane & 3) * 2;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int co = mt * 16 + (lane >> 2) + h * 8;
          dst[co * CIN + ci] = acc[mt][j][2 * h];
          dst[co * CIN + ci + 1] = acc[mt][j][2 * h + 1];
        }
      }
    }
}

// dst[i] = sum over k of part[k*n + i], k ascending (the order of a serial
// sum).  A warp has 32 columns; the block's warps fetch kSumRows rows of them
// at a time into shared memory while the first warp adds up the ones before,
// so the chain of dependent adds waits for shared memory, not for a load from
// L2 each (mean over the launches of a 64^3 training step: 29.7 us as one
// thread a column, 9.0 us now).
constexpr int kSumRows = 128;
__global__ void __launch_bounds__(256) k_sum_parts(const float* __restrict__ part, int nparts, int n,
                                                   float* __restrict__ dst) {
  __shared__ float sm[2][kSumRows][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i = blockIdx.x * 32 + lane;
  auto fetch = [&](int k0, float (*to)[32]) {
    float v[kSumRows / 8];
#pragma unroll
    for (int r = 0; r < kSumRows / 8; ++r) {
      const int k = k0 + r * 8 + warp;
      v[r] = i < n && k < nparts ? __ldg(part + (size_t)k * n + i) : 0.f;
    }
#pragma unroll
    for (int r = 0; r < kSumRows / 8; ++r) to[r * 8 + warp][lane] = v[r];
  };
  fetch(0, sm[0]);
  __syncthreads();
  float s = 0.f;
  for (int k0 = 0, b = 0; k0 < nparts; k0 += kSumRows, b ^= 1) {
    if (k0 + kSumRows < nparts) fetch(k0 + kSumRows, sm[b ^ 1]);
    if (warp == 0) {
      const int m = min(kSumRows, nparts - k0);
#pragma unroll 16
      for (int k = 0; k < m; ++k) s += sm[b][k][lane];
    }
    __syncthreads();
  }
  if (warp == 0 && i < n) dst[i] = s;
}

// w'[t][ci][co] = w[26-t][co][ci]
__global__ void k_flip_transpose(const bf16* __restrict__ w, bf16* __restrict__ wt, int cin, int cout) {
  const int n = 27 * cin * cout;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int co = i % cout, t = i / cout, ci = t % cin, tap = t / cin;
    wt[i] = w[((size_t)(26 - tap) * cout + co) * cin + ci];
  }
}

// Output planes of a CTA, at most as many as TMEM holds: the number whose waves
// of resident CTAs take the fewest plane steps (a chunk of n planes loads
// n + 2 and starts and ends in about one more).  A 64^3 layer of 32 columns in
// chunks of 8 fills one wave of 296; in chunks of 6, as many as give every
// resident CTA one, a second wave of 56 CTAs followed (16 -> 32 channels 41 us
// against 29, 32 -> 32 55 against 41).
int umma_chunk_planes(int sx, int sy, int sz, int most, int ctas) {
  const long long columns = (long long)((sz + kUZ - 1) / kUZ) * ((sy + kUY - 1) / kUY), resident = 148LL * ctas;
  int best = 2;
  long long least = 0;
  for (int p = 2; p <= most; ++p) {
    const long long waves = (columns * ((sx + p - 1) / p) + resident - 1) / resident, cost = waves * (p + 3);
    if (p == 2 || cost < least) {
      best = p;
      least = cost;
    }
  }
  return best;
}

template <int CIN, int COUT, bool RELU, bool BIAS, int SKIP>
cudaError_t umma_launch(cudaStream_t st, const bf16* in, const bf16* skip, const bf16* w, const float* b, bf16* out,
                        int sx, int sy, int sz) {
  constexpr size_t smem = fwd_umma_smem<CIN, COUT>();
  static PerDevice once;
  const cudaError_t attr = once([] {
    return cudaFuncSetAttribute(k_conv3_fwd_umma<CIN, COUT, RELU, BIAS, SKIP>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  });
  if (attr != cudaSuccess) return attr;
  const int planes = umma_chunk_planes(sx, sy, sz, umma_planes<CIN, COUT>(), umma_ctas<CIN, COUT>());
  const dim3 grid((sz + kUZ - 1) / kUZ, (sy + kUY - 1) / kUY, (sx + planes - 1) / planes);
  k_conv3_fwd_umma<CIN, COUT, RELU, BIAS, SKIP><<<grid, 256, smem, st>>>(in, skip, w, b, out, sx, sy, sz, planes);
  return cudaGetLastError();
}

template <int CIN, int COUT, bool RELU, bool BIAS>
cudaError_t fwd_launch(cudaStream_t st, const bf16* in, const bf16* w, const float* b, bf16* out, int sx, int sy,
                       int sz) {
  if constexpr (umma_fits<CIN, COUT>()) {
    if (g_conv_impl == 2) return umma_launch<CIN, COUT, RELU, BIAS, 0>(st, in, nullptr, w, b, out, sx, sy, sz);
  }
  if (g_conv_impl >= 1) {
    constexpr size_t smem = fwd_tile_smem<CIN, COUT>();
    static PerDevice once;
    const cudaError_t attr = once([] {
      return cudaFuncSetAttribute(k_conv3_fwd_tile<CIN, COUT, RELU, BIAS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)smem);
    });
    if (attr != cudaSuccess) return attr;
    const dim3 grid((sz + kTZ - 1) / kTZ, (sy + kTY - 1) / kTY, (sx + kTX - 1) / kTX);
    k_conv3_fwd_tile<CIN, COUT, RELU, BIAS><<<grid, 256, smem, st>>>(in, w, b, out, sx, sy, sz);
    return cudaGetLastError();
  }
  const int V = sx * sy * sz;
  k_conv3_fwd<CIN, COUT, RELU, BIAS><<<(V + kTileM - 1) / kTileM, 128, 0, st>>>(in, w, b, out, sx, sy, sz);
  return cudaGetLastError();
}

template <int CIN, int COUT, bool RELU>
cudaError_t fwd_bias(cudaStream_t st, bool has_bias, const bf16* in, const bf16* w, const float* b, bf16* out, int sx,
                     int sy, int sz) {
  return has_bias ? fwd_launch<CIN, COUT, RELU, true>(st, in, w, b, out, sx, sy, sz)
                  : fwd_launch<CIN, COUT, RELU, false>(st, in, w, b, out, sx, sy, sz);
}

template <int CIN, int COUT>
cudaError_t fwd_relu(cudaStream_t st, bool relu, bool has_bias, const bf16* in, const bf16* w, const float* b,
                     bf16* out, int sx, int sy, int sz) {
  return relu ? fwd_bias<CIN, COUT, true>(st, has_bias, in, w, b, out, sx, sy, sz)
              : fwd_bias<CIN, COUT, false>(st, has_bias, in, w, b, out, sx, sy, sz);
}

// ------------------------------------------------------------ U-Net glue
// Grid-stride elementwise kernels over channels-last tensors.  Fine grid
// (sx,sy,sz), coarse grid (sx/2,sy/2,sz/2); every size is even.

__device__ __forceinline__ int coarse_of(int v, int sx, int sy, int sz) {
  const int z = v % sz, t = v / sz, y = t % sy, x = t / sy;
  return (((x >> 1) * (sy >> 1) + (y >> 1)) * (sz >> 1)) + (z >> 1);
}

// max |a[i]| over i < n: per-block maxima, then one block (order-independent)
__global__ void k_absmax_part(const float* __restrict__ a, int n, float* __restrict__ part) {
  __shared__ float sm[256];
  float m = 0.f;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) m = fmaxf(m, fabsf(a[i]));
  sm[threadIdx.x] = m;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) sm[threadIdx.x] = fmaxf(sm[threadIdx.x], sm[threadIdx.x + o]);
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = sm[0];
}
__global__ void k_absmax_final(const float* __restrict__ part, int n, float* __restrict__ out) {
  __shared__ float sm[256];
  float m = 0.f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) m = fmaxf(m, part[i]);
  sm[threadIdx.x] = m;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) sm[threadIdx.x] = fmaxf(sm[threadIdx.x], sm[threadIdx.x + o]);
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = sm[0];
}

// Network input, 16 channels: [rhs / max|rhs|, 1 on fluid cells (0 air), 0 x 14].
__global__ void k_unet_input(const float* __restrict__ rhs, const int8_t* __restrict__ type,
                             const float* __restrict__ scale, bf16* __restrict__ out, int V) {
  const float s = *scale;
  const float inv = s > 0.f ? 1.f / s : 0.f;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
    __align__(16) bf16 row[16];
    row[0] = __float2bfloat16(rhs[v] * inv);
    row[1] = __float2bfloat16(type[v] == kFluid ? 1.f : 0.f);
#pragma unroll
    for (int c = 2; c < 16; ++c) row[c] = __float2bfloat16(0.f);
    uint4* dst = reinterpret_cast<uint4*>(out + (size_t)v * 16);
    dst[0] = reinterpret_cast<const uint4*>(row)[0];
    dst[1] = reinterpret_cast<const uint4*>(row)[1];
  }
}

// Eight consecutive channels of a voxel (every channel count is a multiple of
// 8): the elementwise kernels below move 16 bytes a thread.  With 2 bytes a
// thread and a division by the channel count for each they were bound by
// their instructions (upsample-concat at 128^3: 375 us for 276 MB; at 64^3,
// mean of both, 31.4 us, 7.5 us now).
struct __align__(16) Oct {
  __nv_bfloat162 h[4];
};
__device__ __forceinline__ Oct ld_oct(const bf16* p) {
  Oct o;
  *reinterpret_cast<uint4*>(&o) = __ldg(reinterpret_cast<const uint4*>(p));
  return o;
}
__device__ __forceinline__ void st_oct(bf16* p, const Oct& o) {
  *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(&o);
}
// 0 where the layer's output y is not positive (ReLU backward).
__device__ __forceinline__ void relu_mask(Oct& o, const Oct& y) {
  const bf16 zero = __float2bfloat16(0.f);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float2 v = __bfloat1622float2(y.h[k]);
    if (!(v.x > 0.f)) o.h[k].x = zero;
    if (!(v.y > 0.f)) o.h[k].y = zero;
  }
}
// Sum of the eight children (x, y, z ascending) of coarse voxel V.
__device__ __forceinline__ void sum_children(const bf16* __restrict__ fine, int V, int cy, int cz, int sy, int sz, int C,
                                             int c, float (&acc)[8]) {
  const int z = V % cz, t = V / cz, y = t % cy, x = t / cy;
  Oct o[8];
#pragma unroll
  for (int k = 0; k < 8; ++k)
    o[k] = ld_oct(fine + ((size_t)(((2 * x + (k >> 2)) * sy + 2 * y + ((k >> 1) & 1)) * sz + 2 * z + (k & 1))) * C + c);
#pragma unroll
  for (int e = 0; e < 8; ++e) acc[e] = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 v = __bfloat1622float2(o[k].h[e]);
      acc[2 * e] += v.x;
      acc[2 * e + 1] += v.y;
    }
}

// 2x2x2 average pooling: out (coarse) from in (fine), C channels.
__global__ void k_pool2(const bf16* __restrict__ in, bf16* __restrict__ out, int sx, int sy, int sz, int C) {
  const int cx = sx >> 1, cy = sy >> 1, cz = sz >> 1, C8 = C >> 3;
  const int n = cx * cy * cz * C8;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int V = i / C8, c = (i - V * C8) * 8;
    float acc[8];
    sum_children(in, V, cy, cz, sy, sz, C, c, acc);
    Oct o;
#pragma unroll
    for (int e = 0; e < 4; ++e) o.h[e] = __floats2bfloat162_rn(acc[2 * e] * 0.125f, acc[2 * e + 1] * 0.125f);
    st_oct(out + (size_t)i * 8, o);
  }
}

// din (fine) = relu'(y) (din + dout(coarse parent) / 8)
__global__ void k_pool2_bwd(const bf16* __restrict__ dout, bf16* __restrict__ din, const bf16* __restrict__ y, int sx,
                            int sy, int sz, int C) {
  const int C8 = C >> 3, n = sx * sy * sz * C8;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int v = i / C8, c = (i - v * C8) * 8;
    const Oct d = ld_oct(dout + (size_t)coarse_of(v, sx, sy, sz) * C + c);
    Oct g;
    *reinterpret_cast<uint4*>(&g) = *reinterpret_cast<const uint4*>(din + (size_t)i * 8);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 a = __bfloat1622float2(d.h[e]), b = __bfloat1622float2(g.h[e]);
      g.h[e] = __floats2bfloat162_rn(__fadd_rn(__fmul_rn(a.x, 0.125f), b.x), __fadd_rn(__fmul_rn(a.y, 0.125f), b.y));
    }
    relu_mask(g, ld_oct(y + (size_t)i * 8));
    st_oct(din + (size_t)i * 8, g);
  }
}

// out (fine, Cu + Cs channels) = [coarse(parent) (Cu), skip (Cs)]
__global__ void k_upcat(const bf16* __restrict__ coarse, const bf16* __restrict__ skip, bf16* __restrict__ out,
                        int sx, int sy, int sz, int Cu, int Cs) {
  const int C8 = (Cu + Cs) >> 3;
  const int n = sx * sy * sz * C8;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int v = i / C8, c = (i - v * C8) * 8;
    st_oct(out + (size_t)i * 8,
           ld_oct(c < Cu ? coarse + (size_t)coarse_of(v, sx, sy, sz) * Cu + c : skip + (size_t)v * Cs + (c - Cu)));
  }
}

// dskip = dout[:, Cu:]; dcoarse[P] = relu'(y) sum over the 8 children of dout[:, :Cu]
__global__ void k_upcat_bwd(const bf16* __restrict__ dout, bf16* __restrict__ dcoarse, const bf16* __restrict__ y,
                            bf16* __restrict__ dskip, int sx, int sy, int sz, int Cu, int Cs) {
  const int cx = sx >> 1, cy = sy >> 1, cz = sz >> 1;
  const int C = Cu + Cs, u8 = Cu >> 3, s8 = Cs >> 3;
  const int nc = cx * cy * cz * u8, n = nc + sx * sy * sz * s8;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    if (i < nc) {
      const int V = i / u8, c = (i - V * u8) * 8;
      float acc[8];
      sum_children(dout, V, cy, cz, sy, sz, C, c, acc);
      Oct o;
#pragma unroll
      for (int e = 0; e < 4; ++e) o.h[e] = __floats2bfloat162_rn(acc[2 * e], acc[2 * e + 1]);
      relu_mask(o, ld_oct(y + (size_t)i * 8));
      st_oct(dcoarse + (size_t)i * 8, o);
    } else {
      const int q = i - nc, v = q / s8, c = (q - v * s8) * 8;
      st_oct(dskip + (size_t)q * 8, ld_oct(dout + (size_t)v * C + Cu + c));
    }
  }
}

// dy = y > 0 ? dy : 0 (ReLU backward, y the layer's output), n8 octets
__global__ void k_relu_bwd(bf16* __restrict__ dy, const bf16* __restrict__ y, int n8) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n8; i += gridDim.x * blockDim.x) {
    Oct o;
    *reinterpret_cast<uint4*>(&o) = *reinterpret_cast<const uint4*>(dy + (size_t)i * 8);
    relu_mask(o, ld_oct(y + (size_t)i * 8));
    st_oct(dy + (size_t)i * 8, o);
  }
}

// Channel sums of dy (V x C) over `rows` consecutive voxels each, voxels in
// order: thread c of 64 / C parts a block; 16 loads are in flight before their
// (serial) adds (mean over a 64^3 training step: 31.3 us as one load at a
// time, 12.9 us now).
__global__ void k_chan_sum_part(const bf16* __restrict__ dy, int V, int C, int rows, int nparts,
                                float* __restrict__ part) {
  const int per = max(1, (int)blockDim.x / C);
  const int g = threadIdx.x / C, c = threadIdx.x - g * C;
  const int p = blockIdx.x * per + g;
  if (g >= per || p >= nparts) return;
  const int v0 = p * rows, v1 = min(V, v0 + rows);
  float s = 0.f;
  int v = v0;
  for (; v + 16 <= v1; v += 16) {
    bf16 t[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) t[k] = dy[(size_t)(v + k) * C + c];
#pragma unroll
    for (int k = 0; k < 16; ++k) s += __bfloat162float(t[k]);
  }
  for (; v < v1; ++v) s += __bfloat162float(dy[(size_t)v * C + c]);
  part[(size_t)p * C + c] = s;
}

// Output head: out[v] = b + sum_c w[c] h[v][c] (16 channels), f32
__global__ void k_head_fwd(const bf16* __restrict__ h, const float* __restrict__ w, const float* __restrict__ b,
                           float* __restrict__ out, int V) {
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
    float s = *b;
    const Oct o[2] = {ld_oct(h + (size_t)v * 16), ld_oct(h + (size_t)v * 16 + 8)};
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const float2 f = __bfloat1622float2(o[c >> 2].h[c & 3]);
      s += w[2 * c] * f.x;
      s += w[2 * c + 1] * f.y;
    }
    out[v] = s;
  }
}

// Adam (bias-corrected) on every tensor of the network in one launch (31
// launches of under 30k elements each otherwise); refreshes the bf16 copies
// of the convolution weights, as they are and flipped and transposed.
__global__ void k_adam(const __grid_constant__ AdamTensors T, float lr, float b1, float b2, float eps, float c1,
                       float c2) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < T.first[T.count]; i += gridDim.x * blockDim.x) {
    int k = 0;
    while (i >= T.first[k + 1]) ++k;
    const AdamTensor& t = T.t[k];
    const int j = i - T.first[k];
    const float gi = t.g[j];
    const float mi = b1 * t.m[j] + (1.f - b1) * gi;
    const float vi = b2 * t.v[j] + (1.f - b2) * gi * gi;
    t.m[j] = mi;
    t.v[j] = vi;
    const float wi = t.w[j] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    t.w[j] = wi;
    if (t.wb) {
      const bf16 h = __float2bfloat16(wi);
      t.wb[j] = h;
      const int ci = j % t.cin, r = j / t.cin, co = r % t.cout, tap = r / t.cout;
      t.wt[((26 - tap) * t.cin + ci) * t.cout + co] = h;
    }
  }
}

__global__ void k_scale_copy(const float* __restrict__ a, float k, float* __restrict__ b, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) b[i] = a[i] * k;
}

__global__ void k_f32_to_bf16(const float* __restrict__ a, bf16* __restrict__ b, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) b[i] = __float2bfloat16(a[i]);
}

// Warm start: p = out * scale * out_scale on fluid cells, 0 elsewhere.
__global__ void k_unet_to_pressure(const float* __restrict__ out, const float* __restrict__ scale, float out_scale,
                                   const int8_t* __restrict__ type, float* __restrict__ p, int V) {
  const float s = *scale * out_scale;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x)
    p[v] = type[v] == kFluid ? out[v] * s : 0.f;
}

// Dataset sample: rhs / scale, type, target p / scale.
__global__ void k_unet_sample(const float* __restrict__ rhs, const int8_t* __restrict__ type,
                              const double* __restrict__ p, const float* __restrict__ scale, float* __restrict__ rhs_s,
                              int8_t* __restrict__ type_s, float* __restrict__ target, int V) {
  const float s = *scale;
  const float inv = s > 0.f ? 1.f / s : 0.f;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
    rhs_s[v] = rhs[v] * inv;
    type_s[v] = type[v];
    target[v] = type[v] == kFluid ? (float)p[v] * inv : 0.f;
  }
}

// ---------------------------------------------------------- training loss
// L = ||e||^2 / ||t||^2 + alpha ||A e||^2 / ||A t||^2 over fluid cells, e = o - t,
// with A the pressure operator the Jacobi sweeps solve ((A x)_i = 6 x_i - sum
// of the six neighbours, a neighbour outside the grid taking x_i, air 0).
// The second term is the prediction's relative residual: it penalises the
// rough error that Jacobi sweeps do not remove.

__device__ __forceinline__ void block_sum2(float a, float b, float* part) {
  __shared__ float sa[256], sb[256];
  sa[threadIdx.x] = a;
  sb[threadIdx.x] = b;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      sa[threadIdx.x] += sa[threadIdx.x + o];
      sb[threadIdx.x] += sb[threadIdx.x + o];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[blockIdx.x * 2] = sa[0];
    part[blockIdx.x * 2 + 1] = sb[0];
  }
}

// e = o - t on fluid cells (0 elsewhere); partial sums of e^2 and t^2.
__global__ void __launch_bounds__(256) k_loss_err(const float* __restrict__ o, const float* __restrict__ t,
                                                  const int8_t* __restrict__ type, float* __restrict__ e, int V,
                                                  float* __restrict__ part) {
  float se = 0.f, st = 0.f;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
    const bool fl = type[v] == kFluid;
    const float ev = fl ? o[v] - t[v] : 0.f;
    e[v] = ev;
    se += ev * ev;
    st += fl ? t[v] * t[v] : 0.f;
  }
  block_sum2(se, st, part);
}

// y = A x on fluid cells (0 elsewhere); partial sums of y^2 (and 0).
__global__ void __launch_bounds__(256) k_apply_A(const float* __restrict__ x, const int8_t* __restrict__ type,
                                                 float* __restrict__ y, int sx, int sy, int sz,
                                                 float* __restrict__ part) {
  float sq = 0.f;
  const int V = sx * sy * sz;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
    float r = 0.f;
    if (type[v] == kFluid) {
      const int z = v % sz, tt = v / sz, yy = tt % sy, xx = tt / sy;
      const float c = x[v];
      float s = xx + 1 < sx ? x[v + sy * sz] : c;
      s += xx > 0 ? x[v - sy * sz] : c;
      s += yy + 1 < sy ? x[v + sz] : c;
      s += yy > 0 ? x[v - sz] : c;
      s += z + 1 < sz ? x[v + 1] : c;
      s += z > 0 ? x[v - 1] : c;
      r = 6.f * c - s;
    }
    y[v] = r;
    sq += r * r;
  }
  block_sum2(sq, 0.f, part);
}

// y = J x on fluid cells (0 elsewhere): one homogeneous Jacobi sweep, the
// mean of the six neighbours (a neighbour outside the grid taking x_i).
// J is symmetric, so it is its own adjoint in the gradient.
// Four cells along z to a thread, launched with programmatic dependent launch:
// a training step runs 60 of these in a row, each bound by its launch and one
// round of loads (64^3: 6.7 us as one cell a thread, 4.0 us now, and the
// launches overlap).
__global__ void __launch_bounds__(256) k_apply_J(const float* __restrict__ x, const int8_t* __restrict__ type,
                                                 float* __restrict__ y, int sx, int sy, int sz) {
  const int nq = sz >> 2, plane = sy * sz;
  const int i = blockIdx.x * 256 + threadIdx.x;
  const bool in = i < sx * sy * nq;
  const int row = i / nq, zq = i - row * nq, xx = row / sy, yy = row - xx * sy;
  const int v = row * sz + 4 * zq;
  char4 t = make_char4(0, 0, 0, 0);
  if (in) t = *reinterpret_cast<const char4*>(type + v);  // written before the previous launch
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");
  if (!in) return;
  auto at = [&](int o) { return *reinterpret_cast<const float4*>(x + o); };
  const float4 c = at(v);
  const float4 xp = xx + 1 < sx ? at(v + plane) : c, xm = xx > 0 ? at(v - plane) : c;
  const float4 yp = yy + 1 < sy ? at(v + sz) : c, ym = yy > 0 ? at(v - sz) : c;
  const float zh = zq + 1 < nq ? x[v + 4] : c.w, zl = zq > 0 ? x[v - 1] : c.x;
  auto mean = [&](int8_t ty, float a, float b, float d, float e, float f, float g) {
    float s = a;
    s += b;
    s += d;
    s += e;
    s += f;
    s += g;
    return ty == kFluid ? s * (1.f / 6.f) : 0.f;
  };
  *reinterpret_cast<float4*>(y + v) =
      make_float4(mean(t.x, xp.x, xm.x, yp.x, ym.x, c.y, zl), mean(t.y, xp.y, xm.y, yp.y, ym.y, c.z, c.x),
                  mean(t.z, xp.z, xm.z, yp.z, ym.z, c.w, c.y), mean(t.w, xp.w, xm.w, yp.w, ym.w, zh, c.z));
}

// g = 2 e / ||t||^2 + 2 alpha q / ||A t||^2 on fluid cells (q = A A e);
// sums = [||e||^2, ||t||^2, ||Ae||^2, ||At||^2]; loss written to *loss.
__global__ void k_loss_grad(const float* __restrict__ e, const float* __restrict__ q, const int8_t* __restrict__ type,
                            const float* __restrict__ sums, float alpha, float* __restrict__ g, int V,
                            float* __restrict__ loss) {
  const float st = fmaxf(sums[1], 1e-30f), sat = fmaxf(sums[3], 1e-30f);
  const float a = 2.f / st, c = 2.f * alpha / sat;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x)
    g[v] = type[v] == kFluid ? a * e[v] + c * q[v] : 0.f;
  if (blockIdx.x == 0 && threadIdx.x == 0) *loss = sums[0] / st + alpha * sums[2] / sat;
}

// Head backward from the output gradient g: dh[v][c] = relu'(h) g_v w[c]; per-block
// partial sums of g_v h[v][c] (16) and g_v.
__global__ void __launch_bounds__(256) k_head_bwd(const float* __restrict__ g, const bf16* __restrict__ h,
                                                  const float* __restrict__ w, bf16* __restrict__ dh, int V,
                                                  float* __restrict__ part) {
  __shared__ float sm[17][256];
  float acc[17];
#pragma unroll
  for (int k = 0; k < 17; ++k) acc[k] = 0.f;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
    const float gv = g[v];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const Oct o = ld_oct(h + (size_t)v * 16 + 8 * q);
      Oct d;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int c = 8 * q + 2 * e;
        const float2 f = __bfloat1622float2(o.h[e]);
        acc[c] += gv * f.x;
        acc[c + 1] += gv * f.y;
        d.h[e] = __floats2bfloat162_rn(gv * w[c], gv * w[c + 1]);
      }
      relu_mask(d, o);
      st_oct(dh + (size_t)v * 16 + 8 * q, d);
    }
    acc[16] += gv;
  }
#pragma unroll
  for (int k = 0; k < 17; ++k) sm[k][threadIdx.x] = acc[k];
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o)
#pragma unroll
      for (int k = 0; k < 17; ++k) sm[k][threadIdx.x] += sm[k][threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x < 17) part[(size_t)blockIdx.x * 17 + threadIdx.x] = sm[threadIdx.x][0];
}

inline int ew_grid(long long n) {
  const long long b = (n + 255) / 256;
  return (int)std::min<long long>(std::max<long long>(b, 1), 148 * 16);
}

}  // namespace

void set_conv_impl(int impl) { g_conv_impl = impl; }

int conv_umma_timeouts() {
  int v = 0;
  cudaMemcpyFromSymbol(&v, g_umma_timeout, sizeof(int));
  return v;
}

cudaError_t conv_umma_test_hook(int skip, unsigned long long wait_ns) {
  const int zero = 0;
  const unsigned long long ns = wait_ns ? wait_ns : 1000000000ull;
  cudaError_t e = cudaMemcpyToSymbol(g_umma_test_skip, &skip, sizeof(int));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_umma_wait_ns, &ns, sizeof(ns));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_umma_timeout, &zero, sizeof(int));
  return e;
}

int unet_wgrad_chunk(int voxels) {
  // about 2 CTAs per SM per tap at 128^3, at least one 128-voxel tile
  const int target = std::max(1, voxels / 512);
  return std::max(kTileM, (target + kTileM - 1) / kTileM * kTileM);
}

// Channel pairs the kernels are instantiated for (the U-Net's layers and
// their data-gradient transposes).
#define AQ_CONV_LAYERS(X) X(16, 16) X(16, 32) X(32, 32) X(32, 64) X(64, 64) X(96, 32) X(48, 16)
#define AQ_CONV_PAIRS(X) AQ_CONV_LAYERS(X) X(32, 16) X(64, 32) X(32, 96) X(16, 48)

template <int CIN, int COUT>
constexpr size_t wgrad_smem() {
  return (size_t)2 * kTileM * ((CIN + 8) + (COUT + 8)) * sizeof(bf16);
}

cudaError_t launch_conv3_fwd(cudaStream_t st, int cin, int cout, bool relu, const void* in, const void* w,
                             const float* bias, void* out, int sx, int sy, int sz) {
  const bf16* i = (const bf16*)in;
  const bf16* ww = (const bf16*)w;
  bf16* o = (bf16*)out;
#define X(A, B) \
  if (cin == A && cout == B) return fwd_relu<A, B>(st, relu, bias != nullptr, i, ww, bias, o, sx, sy, sz);
  AQ_CONV_PAIRS(X)
#undef X
  return cudaErrorInvalidValue;
}

// The tcgen05 convolution reads the concatenation's parts itself.
cudaError_t launch_upcat_conv3_fwd(cudaStream_t st, const void* coarse, const void* skip, void* cat, const void* w,
                                   const float* bias, void* out, int sx, int sy, int sz) {
  if (g_conv_impl == 2)
    return umma_launch<48, 16, true, true, 16>(st, (const bf16*)coarse, (const bf16*)skip, (const bf16*)w, bias,
                                               (bf16*)out, sx, sy, sz);
  const cudaError_t e = launch_upcat(st, coarse, skip, cat, sx, sy, sz, 32, 16);
  return e != cudaSuccess ? e : launch_conv3_fwd(st, 48, 16, true, cat, w, bias, out, sx, sy, sz);
}

cudaError_t launch_conv3_wgrad(cudaStream_t st, int cin, int cout, const void* x, const void* dy, float* part,
                               float* dw, int sx, int sy, int sz) {
  const int V = sx * sy * sz;
  const int cv = unet_wgrad_chunk(V);
  const int chunks = (V + cv - 1) / cv;
  const dim3 grid(chunks, 27);
  bool done = false;
#define X(A, B)                                                                                   \
  if (!done && cin == A && cout == B) {                                                           \
    static PerDevice once;                                                                        \
    const cudaError_t attr = once([] {                                                            \
      return cudaFuncSetAttribute(k_conv3_wgrad<A, B>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                  (int)wgrad_smem<A, B>());                                       \
    });                                                                                           \
    if (attr != cudaSuccess) return attr;                                                         \
    k_conv3_wgrad<A, B><<<grid, 128, wgrad_smem<A, B>(), st>>>((const bf16*)x, (const bf16*)dy, part, sx, sy, \
                                                             sz, cv);                             \
    done = true;                                                                                  \
  }
  AQ_CONV_LAYERS(X)
#undef X
  if (!done) return cudaErrorInvalidValue;
  const int n = 27 * cin * cout;
  k_sum_parts<<<(n + 31) / 32, 256, 0, st>>>(part, chunks, n, dw);
  return cudaGetLastError();
}

size_t conv3_wgrad_part_floats(int cin, int cout, int voxels) {
  const int cv = unet_wgrad_chunk(voxels);
  return (size_t)((voxels + cv - 1) / cv) * 27 * cin * cout;
}

cudaError_t launch_flip_transpose(cudaStream_t st, const void* w, void* wt, int cin, int cout) {
  const int n = 27 * cin * cout;
  k_flip_transpose<<<(n + 255) / 256, 256, 0, st>>>((const bf16*)w, (bf16*)wt, cin, cout);
  return cudaGetLastError();
}

}  // namespace aqb

namespace aqb {

cudaError_t launch_absmax(cudaStream_t st, const float* a, int n, float* part /*>= 1024*/, float* out) {
  const int g = std::min(1024, std::max(1, (n + 255) / 256));
  k_absmax_part<<<g, 256, 0, st>>>(a, n, part);
  k_absmax_final<<<1, 256, 0, st>>>(part, g, out);
  return cudaGetLastError();
}
cudaError_t launch_unet_input(cudaStream_t st, const float* rhs, const int8_t* type, const float* scale, void* out,
                              int V) {
  k_unet_input<<<ew_grid(V), 256, 0, st>>>(rhs, type, scale, (bf16*)out, V);
  return cudaGetLastError();
}
cudaError_t launch_pool2(cudaStream_t st, const void* in, void* out, int sx, int sy, int sz, int C) {
  k_pool2<<<ew_grid((long long)sx * sy * sz * C / 64), 256, 0, st>>>((const bf16*)in, (bf16*)out, sx, sy, sz, C);
  return cudaGetLastError();
}
cudaError_t launch_pool2_bwd(cudaStream_t st, const void* dout, void* din, const void* y, int sx, int sy, int sz,
                             int C) {
  k_pool2_bwd<<<ew_grid((long long)sx * sy * sz * C / 8), 256, 0, st>>>((const bf16*)dout, (bf16*)din, (const bf16*)y,
                                                                        sx, sy, sz, C);
  return cudaGetLastError();
}
cudaError_t launch_upcat(cudaStream_t st, const void* coarse, const void* skip, void* out, int sx, int sy, int sz,
                         int Cu, int Cs) {
  k_upcat<<<ew_grid((long long)sx * sy * sz * (Cu + Cs) / 8), 256, 0, st>>>((const bf16*)coarse, (const bf16*)skip,
                                                                        (bf16*)out, sx, sy, sz, Cu, Cs);
  return cudaGetLastError();
}
cudaError_t launch_upcat_bwd(cudaStream_t st, const void* dout, void* dcoarse, const void* y, void* dskip, int sx,
                             int sy, int sz, int Cu, int Cs) {
  const long long V = (long long)sx * sy * sz;
  k_upcat_bwd<<<ew_grid((V / 8 * Cu + V * Cs) / 8), 256, 0, st>>>((const bf16*)dout, (bf16*)dcoarse, (const bf16*)y,
                                                                  (bf16*)dskip, sx, sy, sz, Cu, Cs);
  return cudaGetLastError();
}
cudaError_t launch_relu_bwd(cudaStream_t st, void* dy, const void* y, int n) {
  k_relu_bwd<<<ew_grid(n / 8), 256, 0, st>>>((bf16*)dy, (const bf16*)y, n / 8);
  return cudaGetLastError();
}
int chan_sum_parts(int V) { return std::min(1024, std::max(1, (V + 255) / 256)); }
cudaError_t launch_chan_sum(cudaStream_t st, const void* dy, int V, int C, float* part, float* out) {
  const int np = chan_sum_parts(V);
  const int rows = (V + np - 1) / np;
  const int threads = std::max(64, (C + 31) / 32 * 32), per = threads / C;
  k_chan_sum_part<<<(np + per - 1) / per, threads, 0, st>>>((const bf16*)dy, V, C, rows, np, part);
  k_sum_parts<<<(C + 31) / 32, 256, 0, st>>>(part, np, C, out);
  return cudaGetLastError();
}
cudaError_t launch_head_fwd(cudaStream_t st, const void* h, const float* w, const float* b, float* out, int V) {
  k_head_fwd<<<ew_grid(V), 256, 0, st>>>((const bf16*)h, w, b, out, V);
  return cudaGetLastError();
}
cudaError_t launch_adam(cudaStream_t st, const AdamTensors& T, float lr, float b1, float b2, float eps, int t) {
  const float c1 = 1.f - powf(b1, (float)t), c2 = 1.f - powf(b2, (float)t);
  k_adam<<<ew_grid(T.first[T.count]), 256, 0, st>>>(T, lr, b1, b2, eps, c1, c2);
  return cudaGetLastError();
}
cudaError_t launch_f32_to_bf16(cudaStream_t st, const float* a, void* b, int n) {
  k_f32_to_bf16<<<ew_grid(n), 256, 0, st>>>(a, (bf16*)b, n);
  return cudaGetLastError();
}
cudaError_t launch_unet_to_pressure(cudaStream_t st, const float* out, const float* scale, float out_scale,
                                    const int8_t* type, float* p, int V) {
  k_unet_to_pressure<<<ew_grid(V), 256, 0, st>>>(out, scale, out_scale, type, p, V);
  return cudaGetLastError();
}
cudaError_t launch_unet_scale_copy(cudaStream_t st, const float* a, float k, float* b, int n) {
  k_scale_copy<<<ew_grid(n), 256, 0, st>>>(a, k, b, n);
  return cudaGetLastError();
}
cudaError_t launch_unet_sample(cudaStream_t st, const float* rhs, const int8_t* type, const double* p,
                               const float* scale, float* rhs_s, int8_t* type_s, float* target, int V) {
  k_unet_sample<<<ew_grid(V), 256, 0, st>>>(rhs, type, p, scale, rhs_s, type_s, target, V);
  return cudaGetLastError();
}

}  // namespace aqb

namespace aqb {

int loss_parts() { return 296; }

// L = ||e||^2/||t||^2 + alpha ||A J^k e||^2 / ||A J^k t||^2: the second term is
// (residual after k Jacobi sweeps from the prediction / the same from zero)^2.
// Scratch: e, p0..p3, g (V floats each), part (loss_parts() * 8), sums (6).
cudaError_t launch_unet_loss_bwd(cudaStream_t st, const float* out, const float* target, const int8_t* type,
                                 const void* h, const float* w, float alpha, int k, void* dh, int sx, int sy, int sz,
                                 float* e, float* p0, float* p1, float* p2, float* p3, float* g, float* part,
                                 float* sums, float* head_part, float* head_sums /* 18: dw 16, db, loss */) {
  const int V = sx * sy * sz;
  const int P = loss_parts();
  cudaError_t smooth_err = cudaSuccess;
  // J^k x into p0/p1; returns the buffer holding the result
  auto smooth = [&](const float* x, float* a, float* b) -> const float* {
    const float* src = x;
    float* bufs[2] = {a, b};
    for (int i = 0; i < k; ++i) {
      cudaLaunchConfig_t lc = {};
      lc.gridDim = dim3((V / 4 + 255) / 256);
      lc.blockDim = dim3(256);
      lc.stream = st;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      at[0].val.programmaticStreamSerializationAllowed = 1;
      lc.attrs = at;
      lc.numAttrs = 1;
      if (cudaError_t e = cudaLaunchKernelEx(&lc, k_apply_J, src, type, bufs[i % 2], sx, sy, sz)) smooth_err = e;
      src = bufs[i % 2];
    }
    return src;
  };
  k_loss_err<<<P, 256, 0, st>>>(out, target, type, e, V, part);
  const float* je = smooth(e, p0, p1);
  k_apply_A<<<P, 256, 0, st>>>(je, type, p2, sx, sy, sz, part + 2 * P);  // r = A J^k e
  const float* jt = smooth(target, p0, p1);
  k_apply_A<<<P, 256, 0, st>>>(jt, type, p3, sx, sy, sz, part + 4 * P);  // A J^k t (sum only)
  k_apply_A<<<P, 256, 0, st>>>(p2, type, p3, sx, sy, sz, part + 6 * P);  // q = A r
  const float* v = smooth(p3, p0, p1);                                    // J^k q
  if (smooth_err != cudaSuccess) return smooth_err;
  k_sum_parts<<<1, 256, 0, st>>>(part, P, 2, sums);
  k_sum_parts<<<1, 256, 0, st>>>(part + 2 * P, P, 2, sums + 2);
  k_sum_parts<<<1, 256, 0, st>>>(part + 4 * P, P, 2, sums + 4);
  cudaError_t err = cudaMemcpyAsync(sums + 3, sums + 4, sizeof(float), cudaMemcpyDeviceToDevice, st);
  if (err != cudaSuccess) return err;
  k_loss_grad<<<ew_grid(V), 256, 0, st>>>(e, v, type, sums, alpha, g, V, head_sums + 17);
  k_head_bwd<<<P, 256, 0, st>>>(g, (const bf16*)h, w, (bf16*)dh, V, head_part);
  k_sum_parts<<<1, 256, 0, st>>>(head_part, P, 17, head_sums);
  return cudaGetLastError();
}

}  // namespace aqb
