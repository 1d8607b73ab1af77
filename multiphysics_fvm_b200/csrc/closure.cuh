// Learned flux-correction closure: device code (sm_100a).
//
// A 3-layer periodic 3x3x3 CNN (16 -> 32 -> 32 -> 16 channels, ReLU between)
// maps normalised primitive variables of a coarse navier_stokes state to face
// flux corrections dF (channel a*5+q: variable q on the +x_a face of the
// cell).  The reference has no learned part; this file holds
//
//   * conv3_kernel: forward conv and data-gradient conv as one BF16 implicit
//     GEMM on the 5th-generation tensor cores (tcgen05.mma, FP32 accumulators
//     in tensor memory), M = 128 positions (an 8 x 16 x-y tile), N = output
//     channels, K = 27 taps x input channels, marching along z;
//   * wgrad_kernel: weight gradient as tcgen05 GEMMs contracting over
//     positions (MN-major operands; three y-taps share one M = 128 MMA);
//   * Adam with bias correction that also writes the packed BF16 operands;
//   * features, the a-priori loss and its gradient, the box filter, and the
//     per-stage correction (clipped, positivity-gated) used by the solver.
//
// Activations are channels-last ([z][y][x][c], x fastest among positions),
// periodic in all three directions.  Tap t = (dz+1)*9 + (dy+1)*3 + (dx+1),
// weights W[t][co][ci].
#pragma once
#include <cuda_bf16.h>
#include <type_traits>
#include "fvm_common.cuh"

namespace fvm {
namespace closure {

constexpr int C_IN0 = 16;   // input features (5 used, zero padded)
constexpr int C_HID = 32;   // hidden channels
constexpr int C_OUT = 16;   // face corrections (15 used)
constexpr int N_VAR = 5;
constexpr uint64_t WAIT_NS = 2000000000ull;  // 2 s bound on every wait

// ------------------------------------------------------ tcgen05 helpers ----
__device__ __forceinline__ void tmem_alloc(uint32_t* dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// D[tmem] (+)= A[smem] * B[smem]^T, BF16 inputs, FP32 accumulate.  Its operands
// are uniform registers: issued by `if (lane == 0)` with operands in vector
// registers, one instruction cost about 165 cycles of the issuing thread (weight
// gradient, 24 per plane), more than the MMA; in warp-uniform code
// under elect_one, about 66.
__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// One lane of the warp, known to the compiler as a single thread.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}
// Arrive on `bar` once every MMA issued so far by this thread has completed.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// 32 lanes x N columns of 32-bit accumulators, one row per thread.
template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t* v);
template <>
__device__ __forceinline__ void tmem_ld<16>(uint32_t taddr, uint32_t* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
}
template <>
__device__ __forceinline__ void tmem_ld<32>(uint32_t taddr, uint32_t* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
        "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]),
        "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]),
        "=r"(v[30]), "=r"(v[31])
      : "r"(taddr));
}

// Shared-memory matrix descriptor, no swizzle (canonical "interleave"
// layout of 8 rows x 16 bytes core matrices).  K-major: LBO = stride between
// the two 8-element K halves, SBO = stride between 8-row groups.  MN-major:
// LBO = stride between 8-row K groups, SBO = stride between 8-element MN
// chunks.  Bits 46-47 hold the descriptor version (1).
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
// Instruction descriptor: BF16 x BF16 -> FP32, dense, M x N, operand majors
// (0 = K-major, 1 = MN-major).
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N, int a_mn, int b_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) |
         ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// One contiguous global -> shared bulk copy completing on `bar`.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ uint4 ldg16(const void* p) { return __ldg(reinterpret_cast<const uint4*>(p)); }
__device__ __forceinline__ void sts16(uint8_t* p, uint4 v) { *reinterpret_cast<uint4*>(p) = v; }

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Bounded wait of one role of a warp-specialised kernel: gives up after WAIT_NS
// or as soon as another role has (`*abort`).
__device__ __forceinline__ bool role_wait(uint64_t* bar, unsigned parity, volatile int* abort) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = global_ns();
  while (!mbar_try_wait(bar, parity))
    if (*abort || global_ns() - t0 > WAIT_NS) return false;
  return true;
}

// Packed B operand (K-major): element (tap t, row n, reduction index k) of a
// layer with K-extent kin and N-extent nout.  One MMA of K = 16 covers an x-y
// tap for up to three output planes: its rows are three blocks of nout, the
// taps dz = +1, 0, -1 (outputs one plane below, at and one above the input
// plane).
__host__ __device__ inline long long pack_index(int t, int n, int k, int kin, int nout) {
  const int ks = kin / 16, u = t % 9, b = 2 - t / 9;
  return (((((long long)u * ks + k / 16) * 2 + (k % 16) / 8) * 3 + b) * nout + n) * 8 + (k % 8);
}

// The runs of planes of one CTA: the n3 planes of all x-y tiles in a row, cut
// into gridDim.x equal runs; a run that crosses a tile boundary is two pieces.
struct PlaneRun {
  long long pos, end;
  int n3;
  __device__ __forceinline__ PlaneRun(int tiles, int n3_) : n3(n3_) {
    const long long total = (long long)tiles * n3_;
    pos = total * blockIdx.x / gridDim.x;
    end = total * (blockIdx.x + 1) / gridDim.x;
  }
  __device__ __forceinline__ bool next(int& tile, int& z0, int& len) {
    if (pos >= end) return false;
    tile = (int)(pos / n3);
    z0 = (int)(pos - (long long)tile * n3);
    len = (int)min((long long)(n3 - z0), end - pos);
    pos += len;
    return true;
  }
};

// ------------------------------------------------------ forward / dgrad ----
enum Epi : int {
  EPI_RELU_BF16 = 0,  // y = max(acc + b, 0), BF16
  EPI_LIN_F32 = 1,    // y = acc + b, FP32
  EPI_MASK_BF16 = 2   // y = acc where mask > 0 else 0, BF16 (ReLU backward)
};

struct ConvArgs {
  const __nv_bfloat16* x;     // input [pos][CIN]
  const void* wpack;          // packed weights (pack_index layout), 27*CIN*COUT bf16
  const float* bias;          // COUT (EPI_RELU_BF16 / EPI_LIN_F32)
  void* y;                    // output [pos][COUT]
  const __nv_bfloat16* mask;  // EPI_MASK_BF16: [pos][COUT]
  int n1, n2, n3;
  unsigned* status;
};

template <int CIN, int COUT>
struct ConvCfg {
  static constexpr int NCH = CIN / 8;      // 16-byte channel chunks
  static constexpr int KS = CIN / 16;      // K = 16 steps per tap
  static constexpr int XE = 10, YE = 18;   // staged x, y extent (tile + halo)
  static constexpr int CHB = XE * 16;      // chunk stride inside a row
  static constexpr int ROWB = NCH * CHB;   // row stride (= SBO of A)
  static constexpr int PLANEB = YE * ROWB;
  static constexpr int NACC = 8;           // accumulators (output planes) in tensor memory
  static constexpr int NLOAD = 128, NT = 288;  // loader threads; 4 epilogue warps + MMA warp + 4 loader warps
  static constexpr int WB = 27 * CIN * COUT * 2;
  // plane ring and copies in flight behind the newest (rings of 5 to 8 slots,
  // where they fit, ran 1-7 % slower)
  static constexpr int NSLOT = 4, LAG = 2;
  static constexpr int OFF_W = 0;
  static constexpr int OFF_RING = WB;
  static constexpr int OFF_BIAS = OFF_RING + NSLOT * PLANEB;
  static constexpr int OFF_BAR = OFF_BIAS + COUT * 4;
  // weights, full[NSLOT], empty[NSLOT], accumulator full / empty [NACC], drain
  static constexpr int NBAR = 2 + 2 * NSLOT + 2 * NACC;
  static constexpr int USED = OFF_BAR + NBAR * 8 + 16;
  // two CTAs per SM: each holds half of the 512 tensor-memory columns at most,
  // so an allocation never waits for another CTA
  static constexpr int BYTES = USED > 77 * 1024 ? USED : 77 * 1024;
  static constexpr int ELEMS = YE * XE * NCH;
  static constexpr int PER = (ELEMS + NLOAD - 1) / NLOAD;
  static constexpr int TCOLS = NACC * COUT;
  static_assert(WB % 128 == 0 && PLANEB % 16 == 0 && OFF_BAR % 8 == 0, "alignment");
  static_assert(TCOLS <= 256 && 2 * (BYTES + 1024) <= 227 * 1024 + 1024, "two CTAs per SM");
};

// Warp-specialised.  Loader warps bring input planes z0-1 .. z0+len of an 8 x 16
// tile into a ring with cp.async; one thread issues the MMAs; four warps drain
// finished accumulators.  An input plane feeds three output planes, so each of
// its 9 x-y taps is one MMA with N = 3 COUT into the adjacent accumulators of
// planes q-1, q, q+1 (a ring of NACC in tensor memory; where the window wraps,
// two MMAs): A, the 4 KB operand that bounds small-N MMAs (shared memory feeds
// the tensor cores 128 B per cycle), is read once for three output planes.
// One MMA per tap, plane and output plane (N = COUT, 27 taps) with the plane
// copies, MMAs and epilogue serialised by block barriers took 204 us for the
// 32 -> 32 layer at 128^3 and 212 us for 32 -> 16; this takes 118 and 100 us.
// The order of the sum over taps is unchanged, the results are bitwise equal.
template <int CIN, int COUT, int EPI>
__global__ void __launch_bounds__(ConvCfg<CIN, COUT>::NT, 2) conv3_kernel(const ConvArgs a) {
  using C = ConvCfg<CIN, COUT>;
  extern __shared__ __align__(128) uint8_t smem[];
  uint64_t* wbar = reinterpret_cast<uint64_t*>(smem + C::OFF_BAR);
  uint64_t* full = wbar + 1;
  uint64_t* empty = full + C::NSLOT;
  uint64_t* accf = empty + C::NSLOT;
  uint64_t* acce = accf + C::NACC;
  uint64_t* drain = acce + C::NACC;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(drain + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tslot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n1 = a.n1, n2 = a.n2, n3 = a.n3;
  const int tx = n1 / 8, tiles = tx * (n2 / 16);
  const uint32_t sbase = smem_u32(smem);

  if (tid == 0) {
    mbar_init(wbar, 1);
    mbar_init(drain, 1);
    for (int s = 0; s < C::NSLOT; ++s) {
      mbar_init(&full[s], C::NLOAD);
      mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < C::NACC; ++s) {
      mbar_init(&accf[s], 1);
      mbar_init(&acce[s], 4);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 4) {
    tmem_alloc(tslot, C::TCOLS);
    tmem_relinquish();
  }
  if constexpr (EPI != EPI_MASK_BF16) {
    if (tid < COUT) reinterpret_cast<float*>(smem + C::OFF_BIAS)[tid] = __ldg(a.bias + tid);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = __shfl_sync(0xffffffffu, *tslot, 0);
  auto give_up = [&]() {
    *abort_flag = 1;
    atomicOr(a.status, ST_TMA_TIMEOUT);
  };

  PlaneRun run(tiles, n3);
  int tile, z0, len;
  if (warp >= 5) {
    // ------------------------------------------------------- loaders ----
    const int lt = tid - 160;
    const size_t zstride = (size_t)n2 * n1 * CIN;
    int g = 0;  // input planes so far: ring slot g % NSLOT
    bool ok = true;
    while (ok && run.next(tile, z0, len)) {
      const int x0 = (tile % tx) * 8, y0 = (tile / tx) * 16;
      // the (periodic) x-y offsets of this thread's 16-byte elements
      int goff[C::PER];
      uint32_t soff[C::PER];
#pragma unroll
      for (int u = 0; u < C::PER; ++u) {
        const int e = lt + u * C::NLOAD;
        const int r = e / (C::XE * C::NCH), rem = e - r * (C::XE * C::NCH);
        const int xe = rem / C::NCH, c = rem - xe * C::NCH;
        int y = y0 - 1 + r, x = x0 - 1 + xe;
        y = y < 0 ? y + n2 : (y >= n2 ? y - n2 : y);
        x = x < 0 ? x + n1 : (x >= n1 ? x - n1 : x);
        goff[u] = (y * n1 + x) * CIN + c * 8;
        soff[u] = ((r * C::NCH + c) * C::XE + xe) * 16;
      }
      for (int q = -1; q <= len; ++q, ++g) {
        const int slot = g % C::NSLOT;
        if (g >= C::NSLOT && !role_wait(&empty[slot], ((g / C::NSLOT) - 1) & 1, abort_flag)) {
          give_up();
          ok = false;
          break;
        }
        int z = z0 + q;
        z = z < 0 ? z + n3 : (z >= n3 ? z - n3 : z);
        const __nv_bfloat16* zb = a.x + (size_t)z * zstride;
        const uint32_t base = sbase + C::OFF_RING + slot * C::PLANEB;
#pragma unroll
        for (int u = 0; u < C::PER; ++u)
          if (lt + u * C::NLOAD < C::ELEMS) cp_async16(base + soff[u], zb + goff[u]);
        cp_async_commit();
        if (g >= C::LAG) {  // plane g - LAG has landed: publish it to the tensor cores
          cp_async_wait<C::LAG>();
          fence_proxy_async();
          mbar_arrive(&full[(g - C::LAG) % C::NSLOT]);
        }
      }
    }
    cp_async_wait<0>();
    fence_proxy_async();
    for (int k = max(g - C::LAG, 0); ok && k < g; ++k) mbar_arrive(&full[k % C::NSLOT]);
  } else if (warp == 4) {
    // ---------------------------------------------------- MMA issuer ----
    // The whole warp runs the loop, so that descriptors stay in uniform
    // registers; one elected lane issues (see umma_bf16).
    if (elect_one()) {
      mbar_arrive_expect_tx(wbar, C::WB);
      bulk_g2s(smem + C::OFF_W, a.wpack, C::WB, wbar);
    }
    __syncwarp();
    bool ok = __all_sync(0xffffffffu, role_wait(wbar, 0, abort_flag));
    if (!ok) {
      give_up();
      mbar_wait_bounded(wbar, 0, WAIT_NS);  // the copy must land before the block ends
    }
    const uint64_t bbase = sdesc(sbase + C::OFF_W, 3 * COUT * 16, 128);
    int g = 0, o0 = 0;  // input planes and output planes so far
    while (ok && run.next(tile, z0, len)) {
      for (int q = -1; q <= len; ++q, ++g) {
        const int slot = g % C::NSLOT;
        // blocks b = 0, 1, 2: output planes q-1, q, q+1 of this piece
        const int blo = q < 1 ? 1 - q : 0, bhi = q + 1 < len ? 2 : len - q;
        const int n = o0 + q + 1;  // the accumulator that block 2 opens
        ok = __all_sync(0xffffffffu, role_wait(&full[slot], (g / C::NSLOT) & 1, abort_flag) &&
                                         (bhi < 2 || n < C::NACC ||
                                          role_wait(&acce[n % C::NACC], ((n / C::NACC) - 1) & 1, abort_flag)));
        if (!ok) {
          give_up();
          break;
        }
        tc_fence_after();
        const uint64_t abase = sdesc(sbase + C::OFF_RING + slot * C::PLANEB, C::CHB, C::ROWB);
        const int s0 = (o0 + q - 1 + blo) & (C::NACC - 1), cnt = bhi - blo + 1;
        const int na = min(cnt, C::NACC - s0), nb = cnt - na;
        const uint32_t da = tbase + (uint32_t)(s0 * COUT);
        const uint32_t ida = idesc_bf16(128, na * COUT, 0, 0), idb = idesc_bf16(128, nb * COUT, 0, 0);
        const uint64_t ba = bbase + (uint64_t)(blo * COUT), bb = ba + (uint64_t)(na * COUT);
        if (elect_one()) {
          // the first K step of a plane opens block 2's accumulator by itself
          const int old = bhi == 2 ? cnt - 1 : cnt, oa = min(old, na), ob = old - oa;
          if (oa) umma_bf16(da, abase, ba, idesc_bf16(128, oa * COUT, 0, 0), 1u);
          if (ob) umma_bf16(tbase, abase, ba + (uint64_t)(oa * COUT), idesc_bf16(128, ob * COUT, 0, 0), 1u);
          if (bhi == 2)
            umma_bf16(tbase + (uint32_t)((n & (C::NACC - 1)) * COUT), abase, bbase + (uint64_t)(2 * COUT),
                      idesc_bf16(128, COUT, 0, 0), 0u);
          // a tap shift only moves the 14-bit start-address field of the
          // descriptors (addresses stay below 256 KB: no carry out of it)
          auto taps = [&](auto wrap) {
#pragma unroll
            for (int k = 1; k < 9 * C::KS; ++k) {
              const int u = k / C::KS, s = k % C::KS;
              const uint64_t ad = abase + (uint64_t)((u / 3 * C::ROWB + 2 * s * C::CHB + (u % 3) * 16) >> 4);
              const uint64_t bo = (uint64_t)((k * 6 * COUT * 16) >> 4);
              umma_bf16(da, ad, ba + bo, ida, 1u);
              if constexpr (decltype(wrap)::value) umma_bf16(tbase, ad, bb + bo, idb, 1u);
            }
          };
          if (nb) taps(std::true_type{});
          else taps(std::false_type{});
          umma_commit(&empty[slot]);
          if (q >= 1) umma_commit(&accf[(o0 + q - 1) % C::NACC]);
        }
        __syncwarp();
      }
      o0 += len;
    }
    // every MMA has completed before tensor memory is freed
    if (elect_one()) umma_commit(drain);
    __syncwarp();
    mbar_wait_bounded(drain, 0, WAIT_NS);
    __syncwarp();
  } else {
    // ------------------------------------------------------ epilogue ----
    const int m = warp * 32 + lane, xl = m & 7, yl = m >> 3;
    const float* bias = reinterpret_cast<const float*>(smem + C::OFF_BIAS);
    int o = 0;  // output planes so far
    bool ok = true;
    while (ok && run.next(tile, z0, len)) {
      const int x0 = (tile % tx) * 8, y0 = (tile / tx) * 16;
      for (int s = 0; s < len; ++s, ++o) {
        const size_t pos = ((size_t)(z0 + s) * n2 + (y0 + yl)) * n1 + (x0 + xl);
        // the mask of this plane, loaded ahead of the wait and of every store
        uint4 mks[EPI == EPI_MASK_BF16 ? COUT / 8 : 1];
        if constexpr (EPI == EPI_MASK_BF16) {
#pragma unroll
          for (int q = 0; q < COUT / 8; ++q) mks[q] = ldg16(a.mask + pos * COUT + 8 * q);
        }
        const int slot = o % C::NACC;
        // (the lanes of a warp give up together: tensor-memory loads are warp-wide)
        if (!__all_sync(0xffffffffu, role_wait(&accf[slot], (o / C::NACC) & 1, abort_flag))) {
          give_up();
          ok = false;
          break;
        }
        tc_fence_after();
        uint32_t v[COUT];
        tmem_ld<COUT>(tbase + ((uint32_t)(warp * 32) << 16) + (uint32_t)(slot * COUT), v);
        tmem_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acce[slot]);
        if constexpr (EPI == EPI_LIN_F32) {
          float4* out = reinterpret_cast<float4*>(static_cast<float*>(a.y) + pos * COUT);
#pragma unroll
          for (int q = 0; q < COUT / 4; ++q)
            out[q] = make_float4(__uint_as_float(v[4 * q]) + bias[4 * q], __uint_as_float(v[4 * q + 1]) + bias[4 * q + 1],
                                 __uint_as_float(v[4 * q + 2]) + bias[4 * q + 2],
                                 __uint_as_float(v[4 * q + 3]) + bias[4 * q + 3]);
        } else {
          uint4* out = reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(a.y) + pos * COUT);
#pragma unroll
          for (int q = 0; q < COUT / 8; ++q) {
            float f[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(v[8 * q + e]);
            if constexpr (EPI == EPI_RELU_BF16) {
#pragma unroll
              for (int e = 0; e < 8; ++e) f[e] = fmaxf(f[e] + bias[8 * q + e], 0.f);
            } else {
              const uint4 mk = mks[q];
              const uint32_t mw[4] = {mk.x, mk.y, mk.z, mk.w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                if (!(bf16_lo(mw[e]) > 0.f)) f[2 * e] = 0.f;
                if (!(bf16_hi(mw[e]) > 0.f)) f[2 * e + 1] = 0.f;
              }
            }
            out[q] = make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]),
                                pack_bf16x2(f[6], f[7]));
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 4) {
    tc_fence_after();
    tmem_dealloc(tbase, C::TCOLS);
  }
}

// ------------------------------------------------------------- wgrad ----
// dW[t][co][ci] = sum_p G[p][co] X[p + off_t][ci].  An MMA contracts 16
// consecutive x positions of one row: A = X shifted by (dz, dx) (MN-major, M =
// 128: rows (j, ci), j = dy + 1; rows of j >= 3 are unused), B = the rows of the
// G planes z_x - 1, z_x, z_x + 1 (MN-major, N = 3 COUT: taps dz = +1, 0, -1),
// accumulator D[dx][(j, ci)][(dz, co)].
struct WgradArgs {
  const __nv_bfloat16* x;  // [pos][CIN]
  const __nv_bfloat16* g;  // [pos][COUT]
  float* partial;          // [chunk][27][COUT][CIN]
  int n1, n2, n3, zc;      // chunks of zc planes of one 16 x 8 tile
  unsigned* status;
};

template <int CIN, int COUT>
struct WgCfg {
  static constexpr int NCH = CIN / 8, NCHG = COUT / 8;
  static constexpr int NSH = 128 / CIN;
  static constexpr int TY = 8, TX = 16;
  static constexpr int XE = TX + 2, YE = TY + 2;
  static constexpr int CHB = XE * 16;
  static constexpr int ROWB = NCH * CHB;
  static constexpr int PLANEB = YE * ROWB;
  static constexpr int PADB = (NSH - 3) * ROWB;  // rows read by the unused shifts past the last slot
  static constexpr int NSLOT = 4, LAG = 2;       // X plane ring
  static constexpr int NG = 16;                  // G plane ring, interleaved by row: [y][slot][chunk][x]
  static constexpr int GCHB = TX * 16;
  static constexpr int GSLOTB = NCHG * GCHB;
  static constexpr int GROWB = NG * GSLOTB;
  static constexpr int NLOAD = 256, NT = 416;    // 8 loader warps, MMA warp, 4 epilogue warps
  static constexpr int OFF_X = 0;
  static constexpr int OFF_G = NSLOT * PLANEB + PADB;
  static constexpr int OFF_BAR = OFF_G + TY * GROWB;
  static constexpr int NBAR = 2 * NSLOT + 3;     // full, empty, accumulators done, accumulators free, drain
  static constexpr int USED = OFF_BAR + NBAR * 8 + 16;
  static constexpr int TCOLS = 9 * COUT <= 256 ? 256 : 512;
  // as many CTAs per SM as its tensor memory holds, never more
  static constexpr int CTAS = 512 / TCOLS;
  static constexpr int FLOOR = (CTAS == 1 ? 120 : 78) * 1024;
  static constexpr int BYTES = USED > FLOOR ? USED : FLOOR;
  static constexpr int XELEMS = YE * XE * NCH, XPER = (XELEMS + NLOAD - 1) / NLOAD;
  static constexpr int GELEMS = TY * TX * NCHG, GPER = (GELEMS + NLOAD - 1) / NLOAD;
  static_assert(NSH >= 3, "three y taps per MMA");
  static_assert(CTAS * (BYTES + 1024) <= 227 * 1024 + 1024, "CTAs per SM");
};

// Same roles as conv3_kernel: A is read once for the three taps dz, so the
// 8 rows x 3 dx MMAs of a plane have N = 3 COUT (nine MMAs of N = COUT per row,
// with plane copies and MMAs serialised, took 359 us for 32 x 32 and 348 us for
// 32 x 16 at 128^3; this takes 157 and 107 us).  A CTA takes every gridDim.x-th chunk; a
// chunk's sums are kept apart and in plane order, so the gradients do not depend
// on the grid of the launch.
template <int CIN, int COUT>
__global__ void __launch_bounds__(WgCfg<CIN, COUT>::NT, WgCfg<CIN, COUT>::CTAS) wgrad_kernel(const WgradArgs a) {
  using C = WgCfg<CIN, COUT>;
  extern __shared__ __align__(128) uint8_t smem[];
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + C::OFF_BAR);
  uint64_t* empty = full + C::NSLOT;
  uint64_t* done = empty + C::NSLOT;
  uint64_t* accfree = done + 1;
  uint64_t* drain = accfree + 1;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(drain + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tslot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n1 = a.n1, n2 = a.n2, n3 = a.n3, len = a.zc;
  const int tx = n1 / C::TX, tiles = tx * (n2 / C::TY), nchunk = tiles * (n3 / a.zc);
  const uint32_t sbase = smem_u32(smem);

  if (tid == 0) {
    mbar_init(done, 1);
    mbar_init(accfree, 4);
    mbar_init(drain, 1);
    for (int s = 0; s < C::NSLOT; ++s) {
      mbar_init(&full[s], C::NLOAD);
      mbar_init(&empty[s], 1);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 8) {
    tmem_alloc(tslot, C::TCOLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = __shfl_sync(0xffffffffu, *tslot, 0);
  auto give_up = [&]() {
    *abort_flag = 1;
    atomicOr(a.status, ST_TMA_TIMEOUT);
  };

  // step g of a chunk: X plane q = -1 .. len and, while q + 1 < len, G plane q + 1
  if (warp < 8) {
    uint32_t xs[C::XPER], gs[C::GPER];
    int xr[C::XPER], xx[C::XPER], xc[C::XPER], gr[C::GPER];
#pragma unroll
    for (int u = 0; u < C::XPER; ++u) {
      const int e = tid + u * C::NLOAD;
      const int r = e / (C::XE * C::NCH), rem = e - r * (C::XE * C::NCH);
      const int xe = rem / C::NCH, c = rem - xe * C::NCH;
      xr[u] = r - 1;
      xx[u] = xe - 1;
      xc[u] = c * 8;
      xs[u] = C::OFF_X + ((r * C::NCH + c) * C::XE + xe) * 16;
    }
#pragma unroll
    for (int u = 0; u < C::GPER; ++u) {
      const int e = tid + u * C::NLOAD;
      const int r = e / (C::TX * C::NCHG), rem = e - r * (C::TX * C::NCHG);
      const int xe = rem / C::NCHG, c = rem - xe * C::NCHG;
      gr[u] = (r * n1 + xe) * COUT + c * 8;
      gs[u] = C::OFF_G + r * C::GROWB + c * C::GCHB + xe * 16;
    }
    int g = 0, go = 0;  // steps and G planes so far
    bool ok = true;
    for (int ch = blockIdx.x; ok && ch < nchunk; ch += gridDim.x) {
      const int tile = ch % tiles, z0 = (ch / tiles) * len;
      const int x0 = (tile % tx) * C::TX, y0 = (tile / tx) * C::TY;
      int xg[C::XPER];
#pragma unroll
      for (int u = 0; u < C::XPER; ++u) {
        int y = y0 + xr[u], x = x0 + xx[u];
        y = y < 0 ? y + n2 : (y >= n2 ? y - n2 : y);
        x = x < 0 ? x + n1 : (x >= n1 ? x - n1 : x);
        xg[u] = (y * n1 + x) * CIN + xc[u];
      }
      for (int q = -1; q <= len; ++q, ++g) {
        const int slot = g % C::NSLOT;
        // X slot: its last step's MMAs are done; the G slot of this step was
        // last read at least six steps ago
        if (g >= C::NSLOT && !role_wait(&empty[slot], ((g / C::NSLOT) - 1) & 1, abort_flag)) {
          give_up();
          ok = false;
          break;
        }
        int z = z0 + q;
        z = z < 0 ? z + n3 : (z >= n3 ? z - n3 : z);
        const __nv_bfloat16* zb = a.x + (size_t)z * n2 * n1 * CIN;
#pragma unroll
        for (int u = 0; u < C::XPER; ++u)
          if (tid + u * C::NLOAD < C::XELEMS) cp_async16(sbase + xs[u] + slot * C::PLANEB, zb + xg[u]);
        if (q + 1 < len) {
          const int gslot = go++ % C::NG;
          const __nv_bfloat16* gb = a.g + ((size_t)(z0 + q + 1) * n2 * n1 + (size_t)y0 * n1 + x0) * COUT;
#pragma unroll
          for (int u = 0; u < C::GPER; ++u)
            if (tid + u * C::NLOAD < C::GELEMS) cp_async16(sbase + gs[u] + gslot * C::GSLOTB, gb + gr[u]);
        }
        cp_async_commit();
        if (g >= C::LAG) {
          cp_async_wait<C::LAG>();
          fence_proxy_async();
          mbar_arrive(&full[(g - C::LAG) % C::NSLOT]);
        }
      }
    }
    cp_async_wait<0>();
    fence_proxy_async();
    for (int k = max(g - C::LAG, 0); ok && k < g; ++k) mbar_arrive(&full[k % C::NSLOT]);
  } else if (warp == 8) {
    int g = 0, o0 = 0, it = 0;  // steps, G planes and chunks so far
    bool ok = true;
    for (int ch = blockIdx.x; ok && ch < nchunk; ch += gridDim.x, ++it) {
      // the accumulators of the previous chunk have been read
      if (it > 0) ok = __all_sync(0xffffffffu, role_wait(accfree, (it - 1) & 1, abort_flag));
      for (int q = -1; ok && q <= len; ++q, ++g) {
        const int slot = g % C::NSLOT;
        ok = __all_sync(0xffffffffu, role_wait(&full[slot], (g / C::NSLOT) & 1, abort_flag));
        if (!ok) break;
        tc_fence_after();
        // blocks b = 0, 1, 2: G planes q-1, q, q+1 (taps dz = +1, 0, -1)
        const int blo = q < 1 ? 1 - q : 0, bhi = q + 1 < len ? 2 : len - q;
        const int s0 = (o0 + q - 1 + blo) & (C::NG - 1), cnt = bhi - blo + 1;
        const int na = min(cnt, C::NG - s0), nb = cnt - na;
        const uint64_t abase = sdesc(sbase + C::OFF_X + slot * C::PLANEB, 128, C::CHB);
        const uint64_t gbase = sdesc(sbase + C::OFF_G, 128, C::GCHB);
        const uint64_t ba = gbase + (uint64_t)((s0 * C::GSLOTB) >> 4);
        const uint32_t ida = idesc_bf16(128, na * COUT, 1, 1), idb = idesc_bf16(128, nb * COUT, 1, 1);
        const uint32_t da = tbase + (uint32_t)(blo * COUT), db = da + (uint32_t)(na * COUT);
        // the chunk's first G plane opens block 1 - q of every dx
        const int fresh = 1 - q;
        if (elect_one()) {
          auto rows = [&](auto wrap, int y_first) {
#pragma unroll
            for (int yl = 0; yl < C::TY; ++yl) {
              if (yl < y_first) continue;
              const uint64_t yo = (uint64_t)((yl * C::GROWB) >> 4);
#pragma unroll
              for (int dx = 0; dx < 3; ++dx) {
                const uint64_t ad = abase + (uint64_t)((yl * C::ROWB + dx * 16) >> 4);
                umma_bf16(da + (uint32_t)(dx * 3 * COUT), ad, ba + yo, ida, 1u);
                if constexpr (decltype(wrap)::value) umma_bf16(db + (uint32_t)(dx * 3 * COUT), ad, gbase + yo, idb, 1u);
              }
            }
          };
          if (fresh >= 0) {
            for (int dx = 0; dx < 3; ++dx)
              for (int b = blo; b <= bhi; ++b)
                umma_bf16(tbase + (uint32_t)((dx * 3 + b) * COUT), abase + (uint64_t)dx,
                          gbase + (uint64_t)((((o0 + q - 1 + b) & (C::NG - 1)) * C::GSLOTB) >> 4),
                          idesc_bf16(128, COUT, 1, 1), b == fresh ? 0u : 1u);
          }
          if (nb) rows(std::true_type{}, fresh >= 0 ? 1 : 0);
          else rows(std::false_type{}, fresh >= 0 ? 1 : 0);
          umma_commit(&empty[slot]);
          if (q == len) umma_commit(done);
        }
        __syncwarp();
      }
      o0 += len;
    }
    if (!ok) {
      // drain this CTA's MMAs (bounded) before tensor memory is freed, on a
      // barrier of its own: which phase `done` is in depends on where the wait
      // ran out
      give_up();
      if (elect_one()) umma_commit(drain);
      __syncwarp();
      mbar_wait_bounded(drain, 0, WAIT_NS);
    }
    __syncwarp();
  } else {
    // row m = j*CIN + ci of accumulator (dx, block b): tap (1 - b, j - 1, dx - 1);
    // a warp reads the tensor-memory lanes of its number modulo 4
    const int quad = warp & 3, m = quad * 32 + lane, j = m / CIN, ci = m % CIN;
    int it = 0;
    for (int ch = blockIdx.x; ch < nchunk; ch += gridDim.x, ++it) {
      const bool live = __all_sync(0xffffffffu, role_wait(done, it & 1, abort_flag)) && *abort_flag == 0;
      if (!live) give_up();
      float* part = a.partial + (size_t)ch * 27 * COUT * CIN;
      tc_fence_after();
#pragma unroll 1
      for (int cidx = 0; cidx < 9; ++cidx) {
        uint32_t v[COUT];
        if (__all_sync(0xffffffffu, live)) {
          tmem_ld<COUT>(tbase + ((uint32_t)(quad * 32) << 16) + (uint32_t)(cidx * COUT), v);
          tmem_wait_ld();
        }
        if (j < 3) {
          const int t = (2 - cidx % 3) * 9 + j * 3 + cidx / 3;
#pragma unroll
          for (int co = 0; co < COUT; ++co)
            part[((size_t)t * COUT + co) * CIN + ci] = live ? __uint_as_float(v[co]) : 0.f;
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(accfree);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 8) {
    tc_fence_after();
    tmem_dealloc(tbase, C::TCOLS);
  }
}

// ------------------------------------------------------- small kernels ----
// Per-block channel sums of a [pos][C] BF16 field (bias gradients).
template <int C>
__global__ void __launch_bounds__(256) channel_sum_kernel(const __nv_bfloat16* g, long long npos,
                                                          float* partial) {
  constexpr int NCHK = C / 8;
  __shared__ float red[256][9];
  const int tid = threadIdx.x, c = tid % NCHK;
  float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  const long long stride = (long long)gridDim.x * (256 / NCHK);
  for (long long p = (long long)blockIdx.x * (256 / NCHK) + tid / NCHK; p < npos; p += stride) {
    const uint4 v = ldg16(g + p * C + c * 8);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      acc[2 * e] += bf16_lo(w[e]);
      acc[2 * e + 1] += bf16_hi(w[e]);
    }
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) red[tid][e] = acc[e];
  __syncthreads();
  if (tid < C) {
    const int cc = tid / 8, e = tid % 8;
    float s = 0.f;
    for (int r = cc; r < 256; r += NCHK) s += red[r][e];
    partial[(size_t)blockIdx.x * C + tid] = s;
  }
}

// out[e] = sum_b partial[b*n + e] (float64 accumulation in block order).  64
// elements per block of 256 threads: four threads per element bring RP_ROWS
// partials at a time into shared memory, one of them adds (one thread per element
// loading as it adds took 24 us for 27,648 x 256).
constexpr int RP_ROWS = 64;
__global__ void __launch_bounds__(256) reduce_partials_kernel(const float* partial, int nblk, int n, float* out) {
  __shared__ float tile[RP_ROWS][64];
  const int k = threadIdx.x & 63, grp = threadIdx.x >> 6, e = blockIdx.x * 64 + k;
  double s = 0.0;
  for (int b0 = 0; b0 < nblk; b0 += RP_ROWS) {
#pragma unroll
    for (int r = 0; r < RP_ROWS / 4; ++r) {
      const int row = r * 4 + grp;
      if (e < n && b0 + row < nblk) tile[row][k] = partial[(size_t)(b0 + row) * n + e];
    }
    __syncthreads();
    if (grp == 0 && e < n)
      for (int row = 0; row < RP_ROWS && b0 + row < nblk; ++row) s += tile[row][k];
    __syncthreads();
  }
  if (grp == 0 && e < n) out[e] = (float)s;
}

// Adam (Kingma & Ba 2015, bias-corrected) on one layer's FP32 master weights
// and bias, then the packed BF16 operands: forward (N = cout, K = cin) and,
// when `pack_bwd` is set, data gradient (tap flipped, N = cin, K = cout).
struct AdamLayer {
  float *w, *m, *v, *b, *mb, *vb;
  const float *gw, *gb;
  __nv_bfloat16 *pack_fwd, *pack_bwd;
  int cout, cin;
};
__global__ void adam_pack_kernel(AdamLayer L, int update, float lr, float b1, float b2, float eps, float c1,
                                 float c2) {
  const int nw = 27 * L.cout * L.cin;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < nw + L.cout; e += gridDim.x * blockDim.x) {
    const bool isw = e < nw;
    float* p = isw ? L.w + e : L.b + (e - nw);
    if (update) {
      float* mm = isw ? L.m + e : L.mb + (e - nw);
      float* vv = isw ? L.v + e : L.vb + (e - nw);
      const float g = isw ? L.gw[e] : L.gb[e - nw];
      const float mn = b1 * *mm + (1.f - b1) * g;
      const float vn = b2 * *vv + (1.f - b2) * g * g;
      *mm = mn;
      *vv = vn;
      *p = *p - lr * (mn * c1) / (sqrtf(vn * c2) + eps);
    }
    if (isw) {
      const int t = e / (L.cout * L.cin), co = (e / L.cin) % L.cout, ci = e % L.cin;
      const __nv_bfloat16 h = __float2bfloat16_rn(*p);
      L.pack_fwd[pack_index(t, co, ci, L.cin, L.cout)] = h;
      if (L.pack_bwd) L.pack_bwd[pack_index(26 - t, ci, co, L.cout, L.cin)] = h;
    }
  }
}

// Normalised primitive features (rho, v1, v2, v3, p) of a float32 state in
// the solver layout (interior only) -> [pos][16] BF16, channels 5..15 zero.
struct FeatArgs {
  const float* u;
  Layout lay;
  float gamma;
  float mean[5], inv_scale[5];
  __nv_bfloat16* x;
};
__global__ void features_kernel(const FeatArgs a) {
  const Layout& L = a.lay;
  const long long n = (long long)L.nx * L.ny * L.nz;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(p % L.nx), j = (int)((p / L.nx) % L.ny), k = (int)(p / ((long long)L.nx * L.ny));
    float u[5];
#pragma unroll
    for (int q = 0; q < 5; ++q) u[q] = __ldg(a.u + L.idx(q, k + 1, j + 1, i + 1));
    const float rinv = 1.f / u[0];
    const float v1 = u[1] * rinv, v2 = u[2] * rinv, v3 = u[3] * rinv;
    const float pr = (a.gamma - 1.f) * (u[4] - 0.5f * u[0] * (v1 * v1 + v2 * v2 + v3 * v3));
    const float f[5] = {u[0], v1, v2, v3, pr};
    uint32_t w[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    float h[6];
#pragma unroll
    for (int q = 0; q < 5; ++q) h[q] = (f[q] - a.mean[q]) * a.inv_scale[q];
    h[5] = 0.f;
    w[0] = pack_bf16x2(h[0], h[1]);
    w[1] = pack_bf16x2(h[2], h[3]);
    w[2] = pack_bf16x2(h[4], 0.f);
    uint4* out = reinterpret_cast<uint4*>(a.x + p * C_IN0);
    out[0] = make_uint4(w[0], w[1], w[2], w[3]);
    out[1] = make_uint4(w[4], w[5], w[6], w[7]);
  }
}

// A-priori loss: E = dt * (-sum_a (s F[p] - s F[p - e_a]) / h_a) - D,
// loss = sum_p sum_q w_q E^2 / N (float64 block partials).
struct LossArgs {
  const float* z3;  // [pos][16] network output
  const float* d;   // target defect, dense [q][pos]
  float* e;         // residual E, dense [q][pos]
  __nv_bfloat16* g3;
  float s[5], w[5];
  float coef[3];    // dt / h_a
  float inv_n;
  double* partial;
  int n1, n2, n3;
};
// One x1 row per warp and iteration; a lane's cell reads its own 64-byte
// output and, of each lower neighbour, the float4 that hold that face's five
// channels.  Bound by HBM (z3 and d read, e written); with scalar loads and
// 64-bit divisions per cell it took 121 us at 128^3, this takes 64 us.
__global__ void __launch_bounds__(256) loss_residual_kernel(const LossArgs a) {
  __shared__ double red[256];
  const long long n = (long long)a.n1 * a.n2 * a.n3;
  const int rows = a.n2 * a.n3;
  double acc = 0.0;
  for (int row = blockIdx.x * 8 + (threadIdx.x >> 5); row < rows; row += gridDim.x * 8) {
    const int k = row / a.n2, j = row - k * a.n2;
    const long long p0 = (long long)row * a.n1;
    const long long py = (long long)(k * (long long)a.n2 + (j == 0 ? a.n2 - 1 : j - 1)) * a.n1;
    const long long pz = (long long)((k == 0 ? a.n3 - 1 : k - 1) * (long long)a.n2 + j) * a.n1;
    for (int i = threadIdx.x & 31; i < a.n1; i += 32) {
      const float4* z0 = reinterpret_cast<const float4*>(a.z3 + (p0 + i) * 16);
      const float4* zx = reinterpret_cast<const float4*>(a.z3 + (p0 + (i == 0 ? a.n1 - 1 : i - 1)) * 16);
      const float4* zy = reinterpret_cast<const float4*>(a.z3 + (py + i) * 16);
      const float4* zz = reinterpret_cast<const float4*>(a.z3 + (pz + i) * 16);
      float own[16], low[16];
      auto put = [](float* f, const float4 v) { f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w; };
#pragma unroll
      for (int c = 0; c < 4; ++c) put(own + 4 * c, __ldg(z0 + c));
      float lx[8], ly[8], lz[8];
      put(lx, __ldg(zx));
      put(lx + 4, __ldg(zx + 1));
      put(ly, __ldg(zy + 1));
      put(ly + 4, __ldg(zy + 2));
      put(lz, __ldg(zz + 2));
      put(lz + 4, __ldg(zz + 3));
#pragma unroll
      for (int q = 0; q < 5; ++q) {
        low[q] = lx[q];
        low[5 + q] = ly[1 + q];
        low[10 + q] = lz[2 + q];
      }
#pragma unroll
      for (int q = 0; q < 5; ++q) {
        float r = 0.f;
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) r -= a.coef[ax] * (a.s[q] * own[ax * 5 + q] - a.s[q] * low[ax * 5 + q]);
        const float ev = r - __ldg(a.d + q * n + p0 + i);
        a.e[q * n + p0 + i] = ev;
        acc += (double)a.w[q] * (double)ev * (double)ev;
      }
    }
  }
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int s = 128; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) a.partial[blockIdx.x] = red[0] * (double)a.inv_n;
}
// dL/dZ3[p][a*5+q] = s_q (dt/h_a) (2 w_q / N) (E[q][p + e_a] - E[q][p]), BF16.
__global__ void __launch_bounds__(256) loss_grad_kernel(const LossArgs a) {
  const long long n = (long long)a.n1 * a.n2 * a.n3;
  const int rows = a.n2 * a.n3;
  for (int row = blockIdx.x * 8 + (threadIdx.x >> 5); row < rows; row += gridDim.x * 8) {
    const int k = row / a.n2, j = row - k * a.n2;
    const long long p0 = (long long)row * a.n1;
    const long long py = (long long)(k * (long long)a.n2 + (j + 1 == a.n2 ? 0 : j + 1)) * a.n1;
    const long long pz = (long long)((k + 1 == a.n3 ? 0 : k + 1) * (long long)a.n2 + j) * a.n1;
    for (int i = threadIdx.x & 31; i < a.n1; i += 32) {
      const long long p = p0 + i, pp[3] = {p0 + (i + 1 == a.n1 ? 0 : i + 1), py + i, pz + i};
      float g[16];
#pragma unroll
      for (int ax = 0; ax < 3; ++ax)
#pragma unroll
        for (int q = 0; q < 5; ++q)
          g[ax * 5 + q] = a.s[q] * a.coef[ax] * (2.f * a.w[q] * a.inv_n) *
                          (__ldg(a.e + q * n + pp[ax]) - __ldg(a.e + q * n + p));
      g[15] = 0.f;
      uint4* out = reinterpret_cast<uint4*>(a.g3 + p * 16);
      out[0] = make_uint4(pack_bf16x2(g[0], g[1]), pack_bf16x2(g[2], g[3]), pack_bf16x2(g[4], g[5]),
                          pack_bf16x2(g[6], g[7]));
      out[1] = make_uint4(pack_bf16x2(g[8], g[9]), pack_bf16x2(g[10], g[11]), pack_bf16x2(g[12], g[13]),
                          pack_bf16x2(g[14], g[15]));
    }
  }
}
__global__ void sum_partials_kernel(const double* partial, int n, double* out) {
  __shared__ double red[256];
  double s = 0.0;
  for (int b = threadIdx.x; b < n; b += 256) s += partial[b];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int k = 128; k > 0; k >>= 1) {
    if (threadIdx.x < k) red[threadIdx.x] += red[threadIdx.x + k];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = red[0];
}

// Conservative f^3 box filter of a float32 state (solver layout) -> dense
// coarse [q][k][j][i] (float64 sums).
__global__ void box_filter_kernel(const float* u, Layout lay, int nv, int f, float* out) {
  const int c1 = lay.nx / f, c2 = lay.ny / f, c3 = lay.nz / f;
  const long long nc = (long long)c1 * c2 * c3;
  const double inv = 1.0 / ((double)f * f * f);
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < nc * nv;
       e += (long long)gridDim.x * blockDim.x) {
    const int q = (int)(e / nc);
    const long long p = e % nc;
    const int i = (int)(p % c1), j = (int)((p / c1) % c2), k = (int)(p / ((long long)c1 * c2));
    double s = 0.0;
    for (int dk = 0; dk < f; ++dk)
      for (int dj = 0; dj < f; ++dj)
        for (int di = 0; di < f; ++di)
          s += (double)__ldg(u + lay.idx(q, k * f + dk + 1, j * f + dj + 1, i * f + di + 1));
    out[e] = (float)(s * inv);
  }
}

// Interior copy between a solver-layout state and a dense [q][k][j][i] array,
// bound by HBM: one lane group (2^gsh lanes, gsh <= 5) per x1 row, V elements
// (16 bytes where rows and pointers allow) along it, DC_ROWS rows in flight
// before their stores; blockIdx.y is the variable.  One element per thread with
// 64-bit divisions for its cell took 571 us at 5 x 256^3 (1.2 TB/s), this
// takes 118 us (5.7 TB/s).
constexpr int DC_ROWS = 4;
template <typename V>
__global__ void __launch_bounds__(256) dense_copy_kernel(float* u, Layout lay, float* dense, int to_state, int gsh) {
  const int n = lay.nx / (int)(sizeof(V) / sizeof(float)), rows = lay.ny * lay.nz;
  const int lane = threadIdx.x & ((1 << gsh) - 1);
  const long long ngrp = ((long long)gridDim.x * blockDim.x) >> gsh;
  const long long grp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> gsh;
  for (long long r0 = grp; r0 < rows; r0 += DC_ROWS * ngrp) {
    V* s[DC_ROWS];
    V* d[DC_ROWS];
    bool in[DC_ROWS];
#pragma unroll
    for (int m = 0; m < DC_ROWS; ++m) {
      const long long row = r0 + m * ngrp;
      in[m] = row < rows;
      const int r = in[m] ? (int)row : 0, k = r / lay.ny, j = r - k * lay.ny;
      s[m] = reinterpret_cast<V*>(u + lay.idx(blockIdx.y, k + 1, j + 1, 1));
      d[m] = reinterpret_cast<V*>(dense + ((long long)blockIdx.y * rows + r) * lay.nx);
    }
    for (int x = lane; x < n; x += 1 << gsh) {
      V v[DC_ROWS];
#pragma unroll
      for (int m = 0; m < DC_ROWS; ++m)
        if (in[m]) v[m] = to_state ? d[m][x] : s[m][x];
#pragma unroll
      for (int m = 0; m < DC_ROWS; ++m)
        if (in[m]) (to_state ? s[m] : d[m])[x] = v[m];
    }
  }
}

// Per-stage correction.  For the stage input Uin (the state the stage's
// residual was taken of) and face x_a + 1/2 of cell p:
//   F = clip(s_q Z3[p][a*5+q], +-beta * smax * |Uq(p + e_a) - Uq(p)|),
//   smax = max(|v_a| + c) over the two cells (the first-order upwind
//   dissipation of the face bounds the anti-dissipative correction),
// R_q = -sum_a (F(p) - F(p - e_a)) / h_a and Uout += coef * dt * R unless the
// result has rho <= 0 or p <= 0, in which case the cell keeps the plain
// update (counted in `nswitch`).  Grids are periodic in all three directions.
struct FixArgs {
  const float* uin;
  float* uout;
  Layout lay;
  const float* z3;
  float s[5];
  float beta, gamma, coef;
  float inv_h[3];
  const Clock* clk;   // dt and the active flag of the solver clock, or null
  float dt_host;      // dt when clk is null
  unsigned long long* nswitch;
  float* ratio;       // flux-corrected transport fractions [10][cells] (fct mode)
};
__device__ __forceinline__ void load_cell(const FixArgs& a, int i, int j, int k, float* u) {
#pragma unroll
  for (int q = 0; q < 5; ++q) u[q] = __ldg(a.uin + a.lay.idx(q, k + 1, j + 1, i + 1));
}
__device__ __forceinline__ float wave_speed(const float* u, int ax, float gamma) {
  const float rinv = 1.f / u[0];
  const float v1 = u[1] * rinv, v2 = u[2] * rinv, v3 = u[3] * rinv;
  const float pr = (gamma - 1.f) * (u[4] - 0.5f * u[0] * (v1 * v1 + v2 * v2 + v3 * v3));
  const float c = (pr > 0.f && u[0] > 0.f) ? sqrtf(gamma * pr * rinv) : 0.f;
  const float va = ax == 0 ? v1 : (ax == 1 ? v2 : v3);
  return fabsf(va) + c;
}
// Clipped face corrections of cell c: Fp[ax][q] on its +x_ax face, Fm[ax][q]
// on its -x_ax face (the +face of the neighbour below), and the dense
// indices of the six neighbours (nb[ax][0] = -e_ax, nb[ax][1] = +e_ax).
__device__ __forceinline__ void face_corrections(const FixArgs& a, const int c[3], long long p, float Fp[3][5],
                                                 float Fm[3][5], long long nb[3][2], int nc[3][2][3] = nullptr) {
  const Layout& L = a.lay;
  const int dims[3] = {L.nx, L.ny, L.nz};
  float u0[5];
  load_cell(a, c[0], c[1], c[2], u0);
#pragma unroll
  for (int ax = 0; ax < 3; ++ax) {
    int cp[3] = {c[0], c[1], c[2]}, cm[3] = {c[0], c[1], c[2]};
    cp[ax] = c[ax] + 1 == dims[ax] ? 0 : c[ax] + 1;  // periodic neighbours
    cm[ax] = c[ax] == 0 ? dims[ax] - 1 : c[ax] - 1;
    if (nc) {
#pragma unroll
      for (int d = 0; d < 3; ++d) { nc[ax][0][d] = cm[d]; nc[ax][1][d] = cp[d]; }
    }
    float up[5], um[5];
    load_cell(a, cp[0], cp[1], cp[2], up);
    load_cell(a, cm[0], cm[1], cm[2], um);
    const float s0 = wave_speed(u0, ax, a.gamma);
    const float sp = fmaxf(s0, wave_speed(up, ax, a.gamma));
    const float sm = fmaxf(s0, wave_speed(um, ax, a.gamma));
    nb[ax][0] = ((long long)cm[2] * L.ny + cm[1]) * L.nx + cm[0];
    nb[ax][1] = ((long long)cp[2] * L.ny + cp[1]) * L.nx + cp[0];
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      const float bp = a.beta * sp * fabsf(up[q] - u0[q]);
      const float bm = a.beta * sm * fabsf(u0[q] - um[q]);
      Fp[ax][q] = fminf(fmaxf(a.s[q] * __ldg(a.z3 + p * 16 + ax * 5 + q), -bp), bp);
      Fm[ax][q] = fminf(fmaxf(a.s[q] * __ldg(a.z3 + nb[ax][0] * 16 + ax * 5 + q), -bm), bm);
    }
  }
}

// Write un to the cell unless it breaks positivity (then count the switch-off).
__device__ __forceinline__ void gated_store(const FixArgs& a, const int c[3], const float un[5]) {
  const Layout& L = a.lay;
  const float ke = 0.5f * (un[1] * un[1] + un[2] * un[2] + un[3] * un[3]) / un[0];
  const float pr = (a.gamma - 1.f) * (un[4] - ke);
  if (un[0] > 0.f && pr > 0.f && isfinite(pr)) {
#pragma unroll
    for (int q = 0; q < 5; ++q) a.uout[L.idx(q, c[2] + 1, c[1] + 1, c[0] + 1)] = un[q];
  } else if (a.nswitch) {
    atomicAdd(a.nswitch, 1ull);
  }
}

// Interior cells of the correction kernels: one x1 row per block iteration,
// threads along the row, so (i, j, k) and the dense index p = row * nx + i
// need no 64-bit division.
template <class Body>
__device__ __forceinline__ void for_each_cell(const Layout& L, Body body) {
  const int rows = L.ny * L.nz;
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const int j = row % L.ny, k = row / L.ny;
    const long long p0 = (long long)row * L.nx;
    for (int i = threadIdx.x; i < L.nx; i += blockDim.x) {
      const int c[3] = {i, j, k};
      body(c, p0 + i);
    }
  }
}

__global__ void __launch_bounds__(128) closure_fix_kernel(const FixArgs a) {
  if (a.clk && !a.clk->active) return;
  const float cdt = a.coef * (a.clk ? (float)a.clk->dt : a.dt_host);
  const Layout& L = a.lay;
  for_each_cell(L, [&](const int c[3], long long p) {
    float Fp[3][5], Fm[3][5];
    long long nb[3][2];
    face_corrections(a, c, p, Fp, Fm, nb);
    float un[5];
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      float r = 0.f;
#pragma unroll
      for (int ax = 0; ax < 3; ++ax) r -= (Fp[ax][q] - Fm[ax][q]) * a.inv_h[ax];
      un[q] = a.uout[L.idx(q, c[2] + 1, c[1] + 1, c[0] + 1)] + cdt * r;
    }
    gated_store(a, c, un);
  });
}

// Flux-corrected transport (Zalesak 1979) bound on the corrections: the
// corrected stage result stays inside [min, max] of the plain stage result
// (uout before correction) over the cell and its six face neighbours, so the
// corrections create no new extrema.  Pass 1: per cell and variable the
// fractions R+ (of the summed inflows) and R- (of the summed outflows) that
// fit inside those bounds, ratio[q][p] and ratio[5+q][p].
__global__ void __launch_bounds__(128) fct_ratio_kernel(const FixArgs a) {
  if (a.clk && !a.clk->active) return;
  const float cdt = a.coef * (a.clk ? (float)a.clk->dt : a.dt_host);
  const Layout& L = a.lay;
  const long long n = (long long)L.nx * L.ny * L.nz;
  for_each_cell(L, [&](const int c[3], long long p) {
    float Fp[3][5], Fm[3][5];
    long long nb[3][2];
    int nc[3][2][3];
    face_corrections(a, c, p, Fp, Fm, nb, nc);
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      const float ul = a.uout[L.idx(q, c[2] + 1, c[1] + 1, c[0] + 1)];
      float hi = ul, lo = ul, pin = 0.f, pout = 0.f;
#pragma unroll
      for (int ax = 0; ax < 3; ++ax) {
        // inflow through the +face is -cdt*Fp/h, through the -face +cdt*Fm/h
        const float tp = -cdt * Fp[ax][q] * a.inv_h[ax], tm = cdt * Fm[ax][q] * a.inv_h[ax];
        pin += fmaxf(tp, 0.f) + fmaxf(tm, 0.f);
        pout += fmaxf(-tp, 0.f) + fmaxf(-tm, 0.f);
#pragma unroll
        for (int sd = 0; sd < 2; ++sd) {
          const int* m = nc[ax][sd];
          const float un = a.uout[L.idx(q, m[2] + 1, m[1] + 1, m[0] + 1)];
          hi = fmaxf(hi, un);
          lo = fminf(lo, un);
        }
      }
      a.ratio[(long long)q * n + p] = pin > 0.f ? fminf(1.f, (hi - ul) / pin) : 1.f;
      a.ratio[(long long)(5 + q) * n + p] = pout > 0.f ? fminf(1.f, (ul - lo) / pout) : 1.f;
    }
  });
}

// Pass 2: each face transfer T (from the lower to the upper cell) is scaled
// by C = min(R+ of the receiving cell, R- of the giving cell), the same factor
// seen from both cells, so the limited correction stays conservative.
__global__ void __launch_bounds__(128) fct_apply_kernel(const FixArgs a) {
  if (a.clk && !a.clk->active) return;
  const float cdt = a.coef * (a.clk ? (float)a.clk->dt : a.dt_host);
  const Layout& L = a.lay;
  const long long n = (long long)L.nx * L.ny * L.nz;
  for_each_cell(L, [&](const int c[3], long long p) {
    float Fp[3][5], Fm[3][5];
    long long nb[3][2];
    face_corrections(a, c, p, Fp, Fm, nb);
    float un[5];
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      const float* Rp = a.ratio + (long long)q * n;        // R+
      const float* Rm = a.ratio + (long long)(5 + q) * n;  // R-
      const float rp0 = Rp[p], rm0 = Rm[p];
      float d = 0.f;
#pragma unroll
      for (int ax = 0; ax < 3; ++ax) {
        // +face: transfer T from this cell to the one above
        const float T = cdt * Fp[ax][q] * a.inv_h[ax];
        const long long up = nb[ax][1], dn = nb[ax][0];
        const float Cp = T >= 0.f ? fminf(Rp[up], rm0) : fminf(rp0, Rm[up]);
        // -face: transfer T' from the cell below to this one
        const float Tm = cdt * Fm[ax][q] * a.inv_h[ax];
        const float Cm = Tm >= 0.f ? fminf(rp0, Rm[dn]) : fminf(Rp[dn], rm0);
        d += Cm * Tm - Cp * T;
      }
      un[q] = a.uout[L.idx(q, c[2] + 1, c[1] + 1, c[0] + 1)] + d;
    }
    gated_store(a, c, un);
  });
}

}  // namespace closure
}  // namespace fvm
