// Scoring kernels of the learned distance model (mlp.cuh).
//
// Scoring some thousand sets is about 0.1 GFLOP: what it costs is launches and the
// round trips between them.  So the whole forward pass of 128 sets is one block of
// one launch: activations go from TMEM through registers into the next product's
// shared-memory operand (18 us for 8192 sets at n = 256, where one launch per
// product, bias and conversion took eleven).
//
// Every product runs on the fifth-generation tensor cores: tcgen05.mma
// kind::f16 (bf16 x bf16 -> fp32), M = 128, N = 64 or 128, K = 16 per
// instruction, issued by one thread, accumulators in TMEM, completion by
// tcgen05.commit to an mbarrier.  Operands lie in shared memory in the
// canonical K-major layout without swizzle, in slices of 64 along K (8 x 8 "core
// matrices" of 128 contiguous bytes, K-adjacent cores 128 bytes apart, 8-row
// groups 1024 bytes apart); the weights and embeddings are kept in that layout in
// global memory, so they are copied as they are.  Every wait is bounded: a wait
// that runs out sets the caller's error word to kErrorWait and the block frees its
// TMEM and stops.
#include "mlp.cuh"

#include <algorithm>
#include <cmath>

namespace sw {
namespace mlp {

namespace {
constexpr int kRows = 128;      // sets per block (the MMA's M)
constexpr int kThreads = 256;   // warps w and w + 4 share rows 32 (w % 4) ..; each takes half of the columns
constexpr u32 kWaitLimit = 1u << 24;
constexpr u32 kSlice = kRows * 64 * 2;  // bytes of a 128-row operand slice; 64-row ones are half

// Shared memory of the forward block: A and B operands (two slices each),
// mbarrier and TMEM address.  Asking for 100 KB keeps it to two blocks an SM,
// whose 256 TMEM columns each always fit.
constexpr u32 kFwdB = 2 * kSlice, kFwdBar = 4 * kSlice;
constexpr u32 kFwdSmem = 100 * 1024;
static_assert(kFwdBar + 32 <= kFwdSmem, "forward block's shared memory");

__device__ __forceinline__ u32 sm_addr(const void* p) { return (u32)__cvta_generic_to_shared(p); }

// byte offset of element (row r, k < 64) of a slice
__host__ __device__ __forceinline__ u32 core_offset(int r, int k) {
  return (u32)((r >> 3) * 1024 + (k >> 3) * 128 + (r & 7) * 16 + (k & 7) * 2);
}

// tcgen05 shared-memory descriptor: start address, leading-dimension byte
// offset (K-adjacent core matrices), stride byte offset (8-row groups),
// descriptor version 1, no swizzle
__device__ __forceinline__ uint64_t smem_desc(u32 addr) {
  const uint64_t start = (addr & 0x3FFFFu) >> 4;
  const uint64_t lbo = 128u >> 4, sbo = 1024u >> 4;
  return start | (lbo << 16) | (sbo << 32) | (1ull << 46);
}

// instruction descriptor, kind::f16: fp32 accumulator, bf16 A and B, both
// K-major, N >> 3 and M >> 4
__device__ __forceinline__ u32 instr_desc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((u32)(n >> 3) << 17) | ((u32)(kRows >> 4) << 24);
}

// One thread: D (TMEM column d, N columns) = or += A · B over `slices` slices.
__device__ __forceinline__ void issue_mma(u32 d, u32 a, u32 b, u32 b_slice, int slices, int n_cols, bool accumulate) {
  const u32 idesc = instr_desc(n_cols);
  for (int s = 0; s < slices; ++s)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint64_t da = smem_desc(a + s * kSlice + i * 256);  // K = 16 i: two cores of 128 bytes further
      const uint64_t db = smem_desc(b + s * b_slice + i * 256);
      const u32 acc = accumulate || s || i ? 1u : 0u;
      asm volatile(
          "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
          "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
          "l"(da), "l"(db), "r"(idesc), "r"(acc)
          : "memory");
    }
}

__device__ __forceinline__ bool bar_wait(u32 bar, u32 parity) {
  for (u32 it = 0; it < kWaitLimit; ++it) {
    u32 ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// A block's tensor-core state.
struct Tc {
  u32 tmem, bar, parity;
  u32* err;
  __device__ void open(u32 bar_addr, u32 slot_addr, const u32* slot, u32 columns, u32* error) {
    bar = bar_addr;
    err = error;
    parity = 0;
    if (threadIdx.x == 0) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < 32) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_addr), "r"(columns)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    tmem = *slot;
  }
  // operands written by all threads become visible to the tensor cores
  __device__ void publish() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  }
  __device__ void commit() {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
  }
  // the committed products are done (the same answer in every thread)
  __device__ bool wait() {
    const bool ok = __syncthreads_and(bar_wait(bar, parity));
    parity ^= 1u;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (!ok && threadIdx.x == 0) atomicExch(err, kErrorWait);
    return ok;
  }
  __device__ void close(u32 columns) {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (threadIdx.x < 32)
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(columns) : "memory");
  }
};

// 32 columns from column c of the warp's rows (lane = row).
__device__ __forceinline__ void ld32(u32 tmem, int row0, u32 c, float* v) {
  u32 r[32];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    u32* const p = r + 16 * h;
    const u32 addr = tmem + ((u32)row0 << 16) + c + 16 * h;
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(p[0]), "=r"(p[1]), "=r"(p[2]), "=r"(p[3]), "=r"(p[4]), "=r"(p[5]), "=r"(p[6]), "=r"(p[7]), "=r"(p[8]),
          "=r"(p[9]), "=r"(p[10]), "=r"(p[11]), "=r"(p[12]), "=r"(p[13]), "=r"(p[14]), "=r"(p[15])
        : "r"(addr)
        : "memory");
  }
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ u32 pack2(float lo, float hi) {
  const __nv_bfloat162 b = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const u32*>(&b);
}
__device__ __forceinline__ float unpack(u32 pair, int i) {
  return __uint_as_float(i ? pair & 0xffff0000u : pair << 16);
}

// 32 values of row r, columns c .. c + 31 (c % 32 == 0): bf16 into a K-major
// operand (K = columns).
__device__ __forceinline__ void put_rows(const float* v, int r, int c, uint8_t* op) {
  u32 p[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) p[i] = pack2(v[2 * i], v[2 * i + 1]);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint4 q = make_uint4(p[4 * i], p[4 * i + 1], p[4 * i + 2], p[4 * i + 3]);
    *reinterpret_cast<uint4*>(op + (c >> 6) * kSlice + core_offset(r, (c & 63) + 8 * i)) = q;
  }
}
__device__ __forceinline__ void copy_in(uint8_t* dst, const bf16* src, int bytes) {
  for (int i = threadIdx.x; i < bytes / 16; i += kThreads)
    reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(src)[i];
}
}  // namespace

// ---- forward ----
__global__ void __launch_bounds__(kThreads) k_forward(const u64* __restrict__ rows, int W, int n, u32 count,
                                                      const bf16* __restrict__ staged_e,
                                                      const bf16* __restrict__ weights,
                                                      const float* __restrict__ params, float* __restrict__ y,
                                                      u32* err) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t *const sA = smem, *const sB = smem + kFwdB;
  u32* const slot = reinterpret_cast<u32*>(smem + kFwdBar + 16);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, q = warp & 3, half = warp >> 2;
  const u32 i0 = blockIdx.x * kRows;
  const int r = q * 32 + lane;
  const u32 row = i0 + r;
  const bool in = row < count;
  Tc tc;
  tc.open(sm_addr(smem + kFwdBar), sm_addr(slot), slot, 256, err);
  bool ok = true;
  // x = bits · E: columns 0 .. 63, two 64-state slices at a time
  const int slices = (n + 63) / 64;
  for (int s0 = 0; s0 < slices && ok; s0 += 2) {
    const int cnt = min(2, slices - s0);
    for (int e = tid; e < cnt * kRows * 8; e += kThreads) {
      const int sl = e >> 10, rr = (e >> 3) & 127, g = e & 7;
      const u64 w = i0 + rr < count ? rows[(size_t)(i0 + rr) * W + s0 + sl] : 0ULL;
      const u32 b = (u32)(w >> (56 - 8 * g));  // states 8 g .. 8 g + 7: bits 7 .. 0
      uint4 v;
      v.x = (b & 0x80 ? 0x3F80u : 0u) | (b & 0x40 ? 0x3F800000u : 0u);  // bf16 ones
      v.y = (b & 0x20 ? 0x3F80u : 0u) | (b & 0x10 ? 0x3F800000u : 0u);
      v.z = (b & 0x08 ? 0x3F80u : 0u) | (b & 0x04 ? 0x3F800000u : 0u);
      v.w = (b & 0x02 ? 0x3F80u : 0u) | (b & 0x01 ? 0x3F800000u : 0u);
      *reinterpret_cast<uint4*>(sA + sl * kSlice + core_offset(rr, 8 * g)) = v;
    }
    copy_in(sB, staged_e + (size_t)s0 * 64 * kEmb, cnt * 64 * kEmb * 2);
    tc.publish();
    if (tid == 0) {
      issue_mma(tc.tmem, sm_addr(sA), sm_addr(sB), kSlice / 2, cnt, kEmb, s0 > 0);
      tc.commit();
    }
    ok = tc.wait();
  }
  if (ok) {
    float v[32];
    ld32(tc.tmem, q * 32, half * 32, v);
    put_rows(v, r, half * 32, sA);
    // h1 = relu(x · W1 + b1): columns 128 .. 255
    copy_in(sB, weights + kOffW1F, kStagedW1 * 2);
    tc.publish();
    if (tid == 0) {
      issue_mma(tc.tmem + 128, sm_addr(sA), sm_addr(sB), kSlice, 1, kHidden, false);
      tc.commit();
    }
    ok = tc.wait();
  }
  if (ok) {
#pragma unroll
    for (int cb = 0; cb < 2; ++cb) {
      const int c = half * 64 + cb * 32;
      float v[32];
      ld32(tc.tmem + 128, q * 32, c, v);
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = fmaxf(v[i] + __ldg(params + kOffB1 + c + i), 0.0f);
      put_rows(v, r, c, sA);
    }
    // h2 = relu(h1 · W2 + b2): columns 0 .. 127
    copy_in(sB, weights + kOffW2F, kStagedW2 * 2);
    tc.publish();
    if (tid == 0) {
      issue_mma(tc.tmem, sm_addr(sA), sm_addr(sB), kSlice, 2, kHidden, false);
      tc.commit();
    }
    ok = tc.wait();
  }
  if (ok) {
    // y = h2 · w3 + b3.  Column l + 32 t joins sum l in the order t = 0 .. 3 (t = 0, 1 in the
    // warps of half 0, which pass their sums on), and the 32 sums fold in
    // halves: one fixed order of additions, whatever the batch.
    float* const s_part = reinterpret_cast<float*>(sA);  // [32][128]; the products have read the operands
    float part[32];
    auto head = [&](int cb) {
      const int c = half * 64 + cb * 32;
      float v[32];
      ld32(tc.tmem, q * 32, c, v);
      u32 p[16];
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = fmaxf(v[i] + __ldg(params + kOffB2 + c + i), 0.0f);
#pragma unroll
      for (int i = 0; i < 16; ++i) p[i] = pack2(v[2 * i], v[2 * i + 1]);
#pragma unroll
      for (int i = 0; i < 32; ++i) part[i] += unpack(p[i / 2], i & 1) * __ldg(params + kOffW3 + c + i);
    };
    if (half == 0) {
#pragma unroll
      for (int i = 0; i < 32; ++i) part[i] = 0.0f;
      head(0);
      head(1);
#pragma unroll
      for (int i = 0; i < 32; ++i) s_part[i * kRows + r] = part[i];
    }
    __syncthreads();
    if (half == 1) {
#pragma unroll
      for (int i = 0; i < 32; ++i) part[i] = s_part[i * kRows + r];
      head(0);
      head(1);
#pragma unroll
      for (int o = 16; o; o >>= 1)
#pragma unroll
        for (int i = 0; i < o; ++i) part[i] += part[i + o];
      if (in) y[row] = part[0] + params[kOffB3];
    }
  }
  tc.close(256);
}

void forward(const u64* rows, int W, int n, u32 count, const bf16* staged_e, const bf16* weights, const float* params,
             float* y, u32* err, cudaStream_t s) {
  if (!count) return;
  const u32 blocks = (count + kRows - 1) / kRows;
  ensure_smem_limit((const void*)k_forward, kFwdSmem);
  k_forward<<<blocks, kThreads, kFwdSmem, s>>>(rows, W, n, count, staged_e, weights, params, y, err);
  SW_LAUNCH_CHECK();
}

// ---- embeddings ----
// Block of 128 states: feat · Phi is one K = 16 product.
__global__ void __launch_bounds__(kThreads) k_embed(const float* __restrict__ feat, const float* __restrict__ params,
                                                    int n, bf16* __restrict__ staged, u32* err) {
  __shared__ __align__(1024) uint8_t sA[kSlice];
  __shared__ __align__(1024) uint8_t sB[kSlice / 2];
  __shared__ __align__(16) uint64_t s_bar[2];
  __shared__ u32 slot;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, q = warp & 3, half = warp >> 2;
  const int s0 = blockIdx.x * kRows;
  Tc tc;
  tc.open(sm_addr(s_bar), sm_addr(&slot), &slot, 64, err);
  for (int e = tid; e < kRows * kFeat; e += kThreads) {
    const int m = e / kFeat, f = e % kFeat;
    const float v = s0 + m < n ? feat[(size_t)(s0 + m) * kFeat + f] : 0.0f;
    *reinterpret_cast<bf16*>(sA + core_offset(m, f)) = __float2bfloat16(v);
  }
  for (int e = tid; e < kEmb * kFeat; e += kThreads) {
    const int j = e % kEmb, f = e / kEmb;
    *reinterpret_cast<bf16*>(sB + core_offset(j, f)) = __float2bfloat16(params[kOffPhi + f * kEmb + j]);
  }
  tc.publish();
  if (tid == 0) {
    const uint64_t da = smem_desc(sm_addr(sA)), db = smem_desc(sm_addr(sB));
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tc.tmem),
        "l"(da), "l"(db), "r"(instr_desc(kEmb)), "r"(0u)
        : "memory");
    tc.commit();
  }
  if (tc.wait()) {
    const int r = q * 32 + lane, st = s0 + r;
    float v[32];
    ld32(tc.tmem, q * 32, half * 32, v);
    if (st < (n + 63) / 64 * 64) {  // states past the last one: zero embeddings to the slice's end
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const int j = half * 32 + i;
        const float a = st < n ? v[i] + params[kOffC + j] : 0.0f;
        staged[(size_t)(st >> 6) * 64 * kEmb + core_offset(j, st & 63) / 2] = __float2bfloat16(fmaxf(a, 0.0f));
      }
    }
  }
  tc.close(64);
}

void embed(const float* feat, const float* params, int n, bf16* staged, u32* err, cudaStream_t s) {
  k_embed<<<(n + kRows - 1) / kRows, kThreads, 0, s>>>(feat, params, n, staged, err);
  SW_LAUNCH_CHECK();
}

// ---- weights ----
// bf16 copies of W1[i][j] and W2[i][j] where the products read them, as B(N = j,
// K = i).
__device__ __forceinline__ void stage_weight(bf16* w, int e, float value) {
  const bf16 b = __float2bfloat16(value);
  if (e >= kOffW1 && e < kOffB1) {
    const int i = (e - kOffW1) / kHidden, j = (e - kOffW1) % kHidden;
    w[kOffW1F + core_offset(j, i) / 2] = b;
  } else if (e >= kOffW2 && e < kOffB2) {
    const int i = (e - kOffW2) / kHidden, j = (e - kOffW2) % kHidden;
    w[kOffW2F + (i >> 6) * (128 * 64) + core_offset(j, i & 63) / 2] = b;
  }
}

__global__ void k_stage_weights(const float* __restrict__ p, bf16* __restrict__ w) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e < kParams) stage_weight(w, e, p[e]);
}

void stage_weights(const float* p, bf16* weights, cudaStream_t s) {
  k_stage_weights<<<(kParams + 255) / 256, 256, 0, s>>>(p, weights);
  SW_LAUNCH_CHECK();
}

}  // namespace mlp
}  // namespace sw
