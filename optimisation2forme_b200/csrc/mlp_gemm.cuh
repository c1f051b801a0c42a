// BF16 GEMM on the 5th-generation tensor cores (tcgen05) for the warm-start
// network: D[M x N] = sum_k A(m, k) B(n, k), BF16 operands staged in shared
// memory, FP32 accumulators in tensor memory (TMEM), fused epilogues.
//
// One CTA computes a 128 x NT tile (NT = 64 or 16).  The network's layers are
// small (K = 128 or 256), so a launch is latency: all K chunks of a tile are
// requested at once (cp.async, 64 of K each, 96 KB at NT = 64), each chunk's
// tcgen05.mma (M = 128, N = NT, K = 16) are issued by one thread as it arrives,
// and one commit to an mbarrier (bounded wait) ends them.  NT = 64 rather than
// the 256 of a whole layer: a batch of 4,096 then is 128 CTAs instead of 32,
// each with a quarter of the epilogue's exponentials, and two fit an SM.  Every
// 16 columns have four warps of their own (8 threads per column), since with
// four warps for all columns the epilogue took longer than the product.
//
// The weight gradients reduce over the batch (k_weight_grad).  A sum over it is
// one tensor memory accumulator up to 2,048 rows (weight_grad_split), so that
// its bits are a function of the batch alone: two such parts meet by an add
// onto zero, which commutes, and only batches above 4,096 add three and more
// in the order they come in.  The bias gradients are eight sums of consecutive
// rows added in order, by blocks of their own in the same launch.  (Slices of
// 256 rows by atomic adds are faster, 135 us a step at batch 4,096, but no two
// runs agree, and Adam's near-zero second moments turn last bits into steps of
// full size: weights 1.6e-4 apart after 60 steps.)  The rows go through a ring
// of eight chunks, filled by 16 warps and multiplied by a warp of its own; a
// launch takes 33 us at batch 4,096, about 1 us a chunk, on 22 to 28 SMs,
// so the layers' launches run side by side.
//
// Measured on B200 at batch 4,096: a training step 156 us (host draws and
// copies of the next batches beside it; 2,250 with blocks of 256 columns, a
// chunk at a time and launches from the host; 231 with the weight gradients in
// one queue), at batch 256 113 us, a hidden layer's launch about 9 us alone,
// nearly all of it latency; the prediction of 74,528 rows through the API
// 2.24 -> 1.0 ms.
//
// Shared memory holds 8 x 16-byte core matrices without swizzle: K-major
// operands (rows contiguous in K) and MN-major ones (the weight gradients'
// operands as they lie in memory, contiguous in the row index) differ in what
// the 16 bytes of a core matrix run along; both have their core matrices at
// ((k/8)*(rows/8) + r/8)*128 bytes, so the descriptors are the same but for
// the major bits of the instruction.
//
// Descriptor bit layouts come from CUTLASS's cute/arch/mma_sm100_desc.hpp.
#pragma once

#include <cuda_bf16.h>
#include <cstdint>

#include <cute/arch/mma_sm100_desc.hpp>

namespace o2f {
namespace mlp {

using bf16 = __nv_bfloat16;

constexpr int kTileM = 128;
constexpr int kKC = 64;          // K elements per shared-memory chunk
constexpr int kMaxChunks = 4;    // of a layer (K = 256)
constexpr int gemm_threads(int nt) { return 8 * nt; }
constexpr long long kWaitLimit = 1ll << 26;  // mbarrier polls before giving up

enum Epilogue : int {
  kEpiHidden = 0,   // z = acc + bias -> pre (bf16), act = silu(z) (bf16)
  kEpiLinear = 1,   // out32 = acc + bias (fp32)
  kEpiBackAct = 2,  // out = bf16(acc * silu'(zprev))
};

// k_gemm_tc, K-major operands: A(m, k) = A[m*lda + k], B(n, k) = B[n*ldb + k],
// K a multiple of 16, at most kMaxChunks * kKC.  k_weight_grad, MN-major ones:
// A(m, k) = A[k*lda + m], B(n, k) = B[k*ldb + n], M a multiple of 8, N of 64, K
// any number of rows, k_split of them (a multiple of kKC) per blockIdx.z.
// lda, ldb, ldo multiples of 8 elements, A and B 16-byte aligned.
struct GemmArgs {
  int M, N, K;
  int k_split;        // k_weight_grad
  const bf16* A;
  int64_t lda;
  const bf16* B;
  int64_t ldb;
  int epi;
  const float* bias;  // [N] or null
  bf16* out;          // kEpiHidden: activation; kEpiBackAct: gradient
  bf16* pre;          // kEpiHidden: pre-activation
  const bf16* zprev;  // kEpiBackAct: pre-activation of the layer below
  int64_t ldo;        // row stride of out / pre / zprev / out32
  float* out32;       // kEpiLinear; k_weight_grad: += sum over k of A(m, k) B(n, k)
  float* bias_grad;   // k_weight_grad: [M] = sum over k of A(m, k)
  int* err;           // set when a wait exceeds its limit
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ float silu(float z) { return z / (1.f + expf(-z)); }
__device__ __forceinline__ float silu_grad(float z) {
  const float s = 1.f / (1.f + expf(-z));
  return s * (1.f + z * (1.f - s));
}

// Shared-memory matrix descriptor of one K=16 slice of a chunk with `rows`
// rows (no swizzle, either major): leading byte offset = the distance between
// the two 8-element K groups, stride byte offset = the distance between 8-row
// groups.
__device__ __forceinline__ uint64_t kmajor_desc(uint32_t chunk_addr, int rows, int kk) {
  cute::UMMA::SmemDescriptor d;
  d.version_ = 1;
  d.lbo_mode_ = 0;
  d.base_offset_ = 0;
  d.layout_type_ = uint8_t(cute::UMMA::LayoutType::SWIZZLE_NONE);
  const uint32_t group_bytes = (uint32_t)(rows / 8) * 128u;  // one 8-element K group of all rows
  d.start_address_ = (uint16_t)((chunk_addr + (uint32_t)(2 * kk) * group_bytes) >> 4);
  d.leading_byte_offset_ = (uint16_t)(group_bytes >> 4);
  d.stride_byte_offset_ = (uint16_t)(128u >> 4);
  return d.desc_;
}

__device__ __forceinline__ void cp_async16(uint8_t* dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src),
               "r"(valid ? 16 : 0)
               : "memory");
}

// Requests rows [r0, r0 + ROWS) x K chunk [k0, k0 + kKC) of X; out-of-range
// elements are zero.  Eight lanes fill one core matrix (no bank conflicts
// along it); K-major, two lanes read the 32 contiguous bytes of a row.
template <int ROWS, bool kTrans, int kThreads>
__device__ __forceinline__ void fill_chunk(uint8_t* dst, const bf16* __restrict__ X, int64_t ld, int r0, int rmax,
                                           int k0, int kmax) {
  constexpr int kItems = ROWS * kKC / 8;
#pragma unroll
  for (int idx = threadIdx.x; idx < kItems; idx += kThreads) {
    if (kTrans) {
      const int k = idx & 7, rg = (idx >> 3) % (ROWS / 8), kg = (idx >> 3) / (ROWS / 8);
      const int gk = k0 + kg * 8 + k, gr = r0 + rg * 8;
      const bool valid = gk < kmax && gr < rmax;
      cp_async16(dst + (kg * (ROWS / 8) + rg) * 128 + k * 16, valid ? X + (int64_t)gk * ld + gr : X, valid);
    } else {
      const int r = (idx >> 1) % ROWS, kg = (idx >> 1) / ROWS * 2 + (idx & 1);
      const int gr = r0 + r, gk = k0 + kg * 8;
      const bool valid = gr < rmax && gk < kmax;
      cp_async16(dst + (kg * (ROWS / 8) + (r >> 3)) * 128 + (r & 7) * 16, valid ? X + (int64_t)gr * ld + gk : X, valid);
    }
  }
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t phase) {
  for (long long it = 0; it < kWaitLimit; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(phase)
        : "memory");
    if (done) return true;
  }
  return false;
}

__device__ __forceinline__ void red_add4(float* p, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

// TMEM columns for a block, by one warp; their address goes to slot.
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, int cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t tmem, int cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
}
// 16 columns of the warp's 32 TMEM lanes.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// The products of one chunk (k of its kKC elements hold more than zeros) into
// tmem, by one thread; first: tmem holds nothing yet.
template <int NT, bool kTrans>
__device__ __forceinline__ void multiply_chunk(uint32_t aA, uint32_t aB, int k, uint32_t tmem, bool first) {
  constexpr auto kMajor = kTrans ? cute::UMMA::Major::MN : cute::UMMA::Major::K;
  const uint32_t idesc = static_cast<uint32_t>(
      cute::UMMA::make_instr_desc<cute::bfloat16_t, cute::bfloat16_t, float, kTileM, NT, kMajor, kMajor>());
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
  for (int kk = 0; kk < kKC / 16; ++kk) {
    if (kk * 16 >= k) break;
    const uint64_t da = kmajor_desc(aA, kTileM, kk), db = kmajor_desc(aB, NT, kk);
    const uint32_t acc = (first && kk == 0) ? 0u : 1u;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
        "l"(da), "l"(db), "r"(idesc), "r"(acc)
        : "memory");
  }
}
// The barrier's phase completes when all products issued so far are complete.
__device__ __forceinline__ void commit_products(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

template <int NT>
constexpr int gemm_smem_bytes() {
  return kMaxChunks * (kTileM + NT) * kKC * 2 + 16;
}

template <int NT>
__global__ void __launch_bounds__(gemm_threads(NT)) k_gemm_tc(GemmArgs a) {
  constexpr int kThreads = gemm_threads(NT);
  static_assert(NT == 64 || NT == 16, "tile N");
  constexpr int kCols = NT < 32 ? 32 : NT;  // TMEM allocation: power of two >= 32
  constexpr int kChunkA = kTileM * kKC * 2, kChunkB = NT * kKC * 2;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sA = smem;
  uint8_t* sB = smem + kMaxChunks * kChunkA;
  uint64_t* bar = reinterpret_cast<uint64_t*>(sB + kMaxChunks * kChunkB);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.x * kTileM, n0 = blockIdx.y * NT;
  const int chunks = (a.K + kKC - 1) / kKC;

  // every chunk's copies first, one group each
#pragma unroll
  for (int c = 0; c < kMaxChunks; ++c) {
    if (c < chunks) {
      fill_chunk<kTileM, false, kThreads>(sA + c * kChunkA, a.A, a.lda, m0, a.M, c * kKC, a.K);
      fill_chunk<NT, false, kThreads>(sB + c * kChunkB, a.B, a.ldb, n0, a.N, c * kKC, a.K);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tmem_alloc(tmem_slot, kCols);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  const uint32_t aBar = smem_u32(bar);

#pragma unroll
  for (int c = 0; c < kMaxChunks; ++c) {
    if (c >= chunks) break;
    if (c == 0) asm volatile("cp.async.wait_group %0;" ::"n"(kMaxChunks - 1) : "memory");
    if (c == 1) asm volatile("cp.async.wait_group %0;" ::"n"(kMaxChunks - 2) : "memory");
    if (c == 2) asm volatile("cp.async.wait_group %0;" ::"n"(kMaxChunks - 3) : "memory");
    if (c == 3) asm volatile("cp.async.wait_group 0;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // smem writes -> tensor core
    __syncthreads();
    if (threadIdx.x == 0)
      multiply_chunk<NT, false>(smem_u32(sA + c * kChunkA), smem_u32(sB + c * kChunkB), a.K - c * kKC, tmem, c == 0);
  }
  if (threadIdx.x == 0) commit_products(aBar);
  const bool ok = __syncthreads_and(mbar_wait(aBar, 0));
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (!ok) {
    if (threadIdx.x == 0) atomicExch(a.err, 1);
    mbar_wait(aBar, 0);  // the products may still be in flight: one more bounded wait
  } else {
    // Epilogue: warp w owns TMEM lanes (tile rows) 32 (w % 4) .. + 31 of the
    // columns 16 (w / 4) .. + 15.
    const int row = m0 + (warp & 3) * 32 + lane;
    for (int c0 = 16 * (warp >> 2); c0 < NT; c0 += kThreads / 8) {
      uint32_t r[16];
      const uint32_t taddr = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0;
      tmem_ld16(taddr, r);
      if (row >= a.M) continue;
      const int nb = n0 + c0;
      const int64_t o0 = (int64_t)row * a.ldo + nb;
      // The thread's 16 consecutive outputs of its row go out as 16-byte
      // vectors when the slice is whole and aligned (ldo a multiple of 8).
      const bool whole = nb + 16 <= a.N && (a.ldo & 7) == 0;
      if (a.epi == kEpiHidden && whole) {
        alignas(16) bf16 zb[16], yb[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const float z = __uint_as_float(r[j]) + (a.bias ? a.bias[nb + j] : 0.f);
          zb[j] = __float2bfloat16_rn(z);
          yb[j] = __float2bfloat16_rn(silu(z));
        }
        uint4* pz = reinterpret_cast<uint4*>(a.pre + o0);
        uint4* py = reinterpret_cast<uint4*>(a.out + o0);
        pz[0] = reinterpret_cast<const uint4*>(zb)[0];
        pz[1] = reinterpret_cast<const uint4*>(zb)[1];
        py[0] = reinterpret_cast<const uint4*>(yb)[0];
        py[1] = reinterpret_cast<const uint4*>(yb)[1];
        continue;
      }
      if (a.epi == kEpiBackAct && whole) {
        alignas(16) bf16 zp[16], gb[16];
        reinterpret_cast<uint4*>(zp)[0] = reinterpret_cast<const uint4*>(a.zprev + o0)[0];
        reinterpret_cast<uint4*>(zp)[1] = reinterpret_cast<const uint4*>(a.zprev + o0)[1];
#pragma unroll
        for (int j = 0; j < 16; ++j)
          gb[j] = __float2bfloat16_rn(__uint_as_float(r[j]) * silu_grad(__bfloat162float(zp[j])));
        uint4* pg = reinterpret_cast<uint4*>(a.out + o0);
        pg[0] = reinterpret_cast<const uint4*>(gb)[0];
        pg[1] = reinterpret_cast<const uint4*>(gb)[1];
        continue;
      }
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int n = nb + j;
        if (n >= a.N) continue;
        const float acc = __uint_as_float(r[j]);
        const int64_t o = (int64_t)row * a.ldo + n;
        if (a.epi == kEpiHidden) {
          const float z = acc + (a.bias ? a.bias[n] : 0.f);
          a.pre[o] = __float2bfloat16_rn(z);
          a.out[o] = __float2bfloat16_rn(silu(z));
        } else if (a.epi == kEpiLinear) {
          a.out32[o] = acc + (a.bias ? a.bias[n] : 0.f);
        } else {
          a.out[o] = __float2bfloat16_rn(acc * silu_grad(__bfloat162float(a.zprev[o])));
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, kCols);
}

// ---------------------------------------------------------------------------
// Weight gradients: out32[m][n] += sum over the batch of A(m, k) B(n, k).

constexpr int kGradN = 64;                      // columns of a tile
constexpr int kGradLoaders = 512;               // threads that copy operands and write the tile
constexpr int kGradThreads = kGradLoaders + 32; // and a warp that issues the products
constexpr int kGradRing = 8;                    // chunks in shared memory
constexpr int kGradLag = 3;                     // of them on their way
static_assert(kGradLag < kGradRing, "a slot is free only after its products");
constexpr int kGradSmem = kGradRing * ((kTileM + kGradN) * kKC * 2 + 16) + 16;
constexpr int kBiasSlices = 8;
constexpr int kBiasBlocks = 4;  // blocks that compute the bias gradients of a tile's rows
constexpr int kBiasRows = kTileM / kBiasBlocks;
static_assert(kBiasSlices * kBiasRows / 2 <= kGradThreads, "a thread per pair of rows and slice");

// Rows of the batch that one accumulator adds up.
inline int weight_grad_split(int n) {
  const int splits = n > 64 * 2048 ? 64 : (n + 2047) / 2048;
  return ((n + splits - 1) / splits + kKC - 1) / kKC * kKC;
}

// Bias gradients of rows m0 .. m0 + kBiasRows - 1 of A: kBiasSlices sums of
// consecutive k, each by one thread in order, then added up in order.  A
// thread sums two neighbouring rows.  (More rows a block: bound by what one SM
// can read.)
__device__ __forceinline__ void bias_grad_rows(const GemmArgs& a, int m0, float* part) {
  constexpr int kAhead = 64;
  const int slice = threadIdx.x / (kBiasRows / 2), m = threadIdx.x % (kBiasRows / 2) * 2;
  const int per = (a.K + kBiasSlices - 1) / kBiasSlices;
  const int k1 = min(a.K, (slice + 1) * per);
  float s0 = 0.f, s1 = 0.f;
  if (slice < kBiasSlices && m0 + m < a.M) {
    const bf16* p = a.A + m0 + m;
    auto row = [&](int k) { return *reinterpret_cast<const __nv_bfloat162*>(p + (int64_t)k * a.lda); };
    int k = slice * per;
    for (; k + kAhead <= k1; k += kAhead) {
      __nv_bfloat162 v[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) v[u] = row(k + u);
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        s0 += __low2float(v[u]);
        s1 += __high2float(v[u]);
      }
    }
    for (; k < k1; ++k) {
      const __nv_bfloat162 v = row(k);
      s0 += __low2float(v);
      s1 += __high2float(v);
    }
  }
  if (slice < kBiasSlices) {
    part[slice * kBiasRows + m] = s0;
    part[slice * kBiasRows + m + 1] = s1;
  }
  __syncthreads();
  if (threadIdx.x < kBiasRows && m0 + (int)threadIdx.x < a.M) {
    float t = 0.f;
#pragma unroll
    for (int q = 0; q < kBiasSlices; ++q) t += part[q * kBiasRows + threadIdx.x];
    a.bias_grad[m0 + threadIdx.x] = t;
  }
}

__global__ void __launch_bounds__(kGradThreads) k_weight_grad(GemmArgs a) {
  constexpr int kChunkA = kTileM * kKC * 2, kChunkB = kGradN * kKC * 2;
  extern __shared__ __align__(1024) uint8_t smem[];
  const int m0 = blockIdx.x * kTileM;
  if (blockIdx.y * kGradN >= a.N) {  // kBiasBlocks of them
    if (blockIdx.z == 0)
      bias_grad_rows(a, m0 + (blockIdx.y - a.N / kGradN) * kBiasRows, reinterpret_cast<float*>(smem));
    return;
  }
  uint8_t* sA = smem;
  uint8_t* sB = smem + kGradRing * kChunkA;
  uint64_t* full = reinterpret_cast<uint64_t*>(sB + kGradRing * kChunkB);  // a slot's copies have arrived
  uint64_t* done = full + kGradRing;                                       // its products are complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + kGradRing);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = blockIdx.y * kGradN;
  const int kb = blockIdx.z * a.k_split;
  const int ke = min(a.K, kb + a.k_split);
  const int chunks = (ke - kb + kKC - 1) / kKC;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kGradRing; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(full + i)), "r"(kGradLoaders / 32)
                   : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(done + i)) : "memory");
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tmem_alloc(tmem_slot, kGradN);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  // the n-th use of a slot: chunk n * kGradRing + slot
  auto wait_done = [&](int c) { return mbar_wait(smem_u32(done + c % kGradRing), (uint32_t)(c / kGradRing) & 1u); };
  bool ok = true;
  if (threadIdx.x < kGradLoaders) {
    // one lane of a warp waits and arrives for it
    for (int c = 0; c < chunks + kGradLag; ++c) {
      if (c < chunks) {
        if (c >= kGradRing) {
          if (lane == 0) ok = wait_done(c - kGradRing);
          ok = __shfl_sync(0xffffffffu, ok, 0);
          if (!ok) break;
        }
        const int slot = c % kGradRing;
        fill_chunk<kTileM, true, kGradLoaders>(sA + slot * kChunkA, a.A, a.lda, m0, a.M, kb + c * kKC, ke);
        fill_chunk<kGradN, true, kGradLoaders>(sB + slot * kChunkB, a.B, a.ldb, n0, a.N, kb + c * kKC, ke);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      if (c < kGradLag) continue;
      asm volatile("cp.async.wait_group %0;" ::"n"(kGradLag) : "memory");  // chunk c - kGradLag is there
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(full + (c - kGradLag) % kGradRing))
                     : "memory");
    }
    if (ok && lane == 0) ok = wait_done(chunks - 1);
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (threadIdx.x == kGradLoaders) {
    int c = 0;
    for (; c < chunks; ++c) {
      const int slot = c % kGradRing;
      ok = mbar_wait(smem_u32(full + slot), (uint32_t)(c / kGradRing) & 1u);
      if (!ok) break;
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // smem writes -> tensor core
      multiply_chunk<kGradN, true>(smem_u32(sA + slot * kChunkA), smem_u32(sB + slot * kChunkB), ke - kb - c * kKC,
                                   tmem, c == 0);
      commit_products(smem_u32(done + slot));
    }
    if (c > 0 && !wait_done(c - 1)) ok = false;  // none in flight when the block ends
  }
  ok = __syncthreads_and(ok);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (!ok) {
    if (threadIdx.x == 0) atomicExch(a.err, 1);
  } else if (threadIdx.x < kGradLoaders) {
    const int row = m0 + (warp & 3) * 32 + lane, c0 = 16 * (warp >> 2);
    uint32_t r[16];
    tmem_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0, r);
    if (row < a.M) {
      float* out = a.out32 + (int64_t)row * a.ldo + n0 + c0;
#pragma unroll
      for (int j = 0; j < 16; j += 4)
        red_add4(out + j, __uint_as_float(r[j]), __uint_as_float(r[j + 1]), __uint_as_float(r[j + 2]),
                 __uint_as_float(r[j + 3]));
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, kGradN);
}

}  // namespace mlp
}  // namespace o2f
