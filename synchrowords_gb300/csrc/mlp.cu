// Kernels of the learned distance model (mlp.cuh).
//
// A training step on a batch of a few hundred sets is 1.5 GFLOP: what it costs is
// launches and the round trips between them.  So the whole forward pass of a
// block of 128 sets is one block of one launch, and the whole backward pass
// another: the activations of a block go from TMEM through registers into the
// next product's shared-memory operand, and only what the other pass needs is
// written out.  (One launch per product, bias and conversion took 45 launches and
// 540 us a step at batch 512.)
//
// Every product runs on the fifth-generation tensor cores: tcgen05.mma
// kind::f16 (bf16 x bf16 -> fp32), M = 128, N = 64 or 128, K = 16 per
// instruction, issued by one thread, accumulators in TMEM, completion by
// tcgen05.commit to an mbarrier.  Operands lie in shared memory in the
// canonical K-major layout without swizzle, in slices of 64 along K (8 x 8 "core
// matrices" of 128 contiguous bytes, K-adjacent cores 128 bytes apart, 8-row
// groups 1024 bytes apart); the weights and embeddings are kept in that layout in
// global memory, so they are copied as they are.  Every wait is bounded: a wait
// that runs out sets an error word (tc_error()) and the block frees its TMEM and
// stops.
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
// Backward block: four operands of two slices, the sets' rows, mbarrier; one block an SM (512 TMEM columns).
constexpr u32 kBwdB = 2 * kSlice, kBwdC = 4 * kSlice, kBwdT = 6 * kSlice, kBwdRows = 8 * kSlice,
              kBwdBar = kBwdRows + kRows * 8 * 8;
constexpr u32 kBwdSmem = kBwdBar + 32;

__device__ u32 g_tc_error = 0;

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
  __device__ void open(u32 bar_addr, u32 slot_addr, const u32* slot, u32 columns) {
    bar = bar_addr;
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
    if (!ok && threadIdx.x == 0) atomicExch(&g_tc_error, 1u);
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
// operand (K = columns) and, if given, into a global row.
__device__ __forceinline__ void put_rows(const float* v, int r, int c, uint8_t* op, bf16* global) {
  u32 p[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) p[i] = pack2(v[2 * i], v[2 * i + 1]);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint4 q = make_uint4(p[4 * i], p[4 * i + 1], p[4 * i + 2], p[4 * i + 3]);
    *reinterpret_cast<uint4*>(op + (c >> 6) * kSlice + core_offset(r, (c & 63) + 8 * i)) = q;
    if (global) reinterpret_cast<uint4*>(global)[i] = q;
  }
}
// ... transposed: bf16 pairs p (columns c ..) into an operand whose K is the row.
__device__ __forceinline__ void put_columns(const u32* p, int r, int c, uint8_t* op, u32 slice) {
  uint8_t* const o = op + (r >> 6) * slice;
#pragma unroll
  for (int i = 0; i < 32; ++i)
    *reinterpret_cast<uint16_t*>(o + core_offset(c + i, r & 63)) = (uint16_t)(i & 1 ? p[i / 2] >> 16 : p[i / 2]);
}

// Sums of 32 columns over the warp's rows: lane l gets column l's (31 exchanges).
__device__ __forceinline__ float column_sums(float* v) {
  const u32 lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const float send = up ? v[i] : v[i + o], keep = up ? v[i + o] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  return v[0];
}

__device__ __forceinline__ void copy_in(uint8_t* dst, const bf16* src, int bytes) {
  for (int i = threadIdx.x; i < bytes / 16; i += kThreads)
    reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(src)[i];
}
}  // namespace

// ---- forward ----
template <bool kTrain>
__global__ void __launch_bounds__(kThreads) k_forward(const u64* __restrict__ rows, int W, int n, u32 count,
                                                      const bf16* __restrict__ staged_e,
                                                      const bf16* __restrict__ weights,
                                                      const float* __restrict__ params, float* __restrict__ y,
                                                      Activations act) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t *const sA = smem, *const sB = smem + kFwdB;
  u32* const slot = reinterpret_cast<u32*>(smem + kFwdBar + 16);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, q = warp & 3, half = warp >> 2;
  const u32 i0 = blockIdx.x * kRows;
  const int r = q * 32 + lane;
  const u32 row = i0 + r;
  const bool in = row < count;
  Tc tc;
  tc.open(sm_addr(smem + kFwdBar), sm_addr(slot), slot, 256);
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
    put_rows(v, r, half * 32, sA, kTrain && in ? act.x + (size_t)row * kEmb + half * 32 : nullptr);
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
      u32 open = 0;
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        v[i] += __ldg(params + kOffB1 + c + i);
        open |= v[i] > 0.0f ? 1u << i : 0u;
        v[i] = fmaxf(v[i], 0.0f);
      }
      put_rows(v, r, c, sA, kTrain && in ? act.h1 + (size_t)row * kHidden + c : nullptr);
      if (kTrain && in) act.open1[(size_t)row * 4 + (c >> 5)] = open;
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
      u32 open = 0;
      u32 p[16];
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        v[i] += __ldg(params + kOffB2 + c + i);
        open |= v[i] > 0.0f ? 1u << i : 0u;
        v[i] = fmaxf(v[i], 0.0f);
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) p[i] = pack2(v[2 * i], v[2 * i + 1]);
#pragma unroll
      for (int i = 0; i < 32; ++i) part[i] += unpack(p[i / 2], i & 1) * __ldg(params + kOffW3 + c + i);
      if (kTrain && in) {
        uint4* const o = reinterpret_cast<uint4*>(act.h2 + (size_t)row * kHidden + c);
#pragma unroll
        for (int i = 0; i < 4; ++i) o[i] = make_uint4(p[4 * i], p[4 * i + 1], p[4 * i + 2], p[4 * i + 3]);
        act.open2[(size_t)row * 4 + (c >> 5)] = open;
      }
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
             float* y, const Activations& act, cudaStream_t s) {
  if (!count) return;
  const u32 blocks = (count + kRows - 1) / kRows;
  if (act.h2) {
    ensure_smem_limit((const void*)k_forward<true>, kFwdSmem);
    k_forward<true><<<blocks, kThreads, kFwdSmem, s>>>(rows, W, n, count, staged_e, weights, params, y, act);
  } else {
    ensure_smem_limit((const void*)k_forward<false>, kFwdSmem);
    k_forward<false><<<blocks, kThreads, kFwdSmem, s>>>(rows, W, n, count, staged_e, weights, params, y, act);
  }
  SW_LAUNCH_CHECK();
}

// ---- loss ----
// Warp per row.  The ranking term pairs the rows of one group (one BFS layer):
// for t_a < t_b, w / rows * softplus(y_a - y_b), so that a set nearer to a
// singleton scores lower than its sibling.  (One thread per row walked the batch
// with dependent loads: 75 us at 512 rows.)
__global__ void __launch_bounds__(256) k_loss(const float* __restrict__ y, const float* __restrict__ tgt,
                                              const uint32_t* __restrict__ grp, int rows, float w,
                                              float* __restrict__ dy, float* loss) {
  __shared__ float s_sum[8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, i = blockIdx.x * 8 + warp;
  float l = 0.0f;
  if (i < rows) {
    const float yi = y[i], ti = tgt[i];
    float g = 0.0f;
    if (grp) {
      const uint32_t gi = grp[i];
      for (int j0 = 0; j0 < rows; j0 += 32) {
        const int j = j0 + lane;
        float term = 0.0f;
        if (j < rows && grp[j] == gi) {
          const float tj = tgt[j];
          if (ti < tj) {  // i should score below j
            const float z = yi - y[j];
            term = 1.0f / (1.0f + __expf(-z));
            l += z > 20.0f ? z : log1pf(__expf(z));
          } else if (tj < ti) {  // j should score below i
            term = -(1.0f / (1.0f + __expf(-(y[j] - yi))));
          }
        }
#pragma unroll
        for (int x = 0; x < 32; ++x) g += __shfl_sync(0xffffffffu, term, x);  // in the order of j
      }
#pragma unroll
      for (int o = 16; o; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
      l *= w / (float)rows;
    }
    if (lane == 0) {
      const float d = yi - ti;
      l += d * d / (float)rows;
      dy[i] = 2.0f * d / (float)rows + (grp ? w * g / (float)rows : 0.0f);
    }
  }
  if (lane == 0) s_sum[warp] = i < rows ? l : 0.0f;
  __syncthreads();
  if (threadIdx.x == 0) {
    float b = 0.0f;
    for (int x = 0; x < 8; ++x) b += s_sum[x];
    atomicAdd(loss, b);
  }
}

void loss(const float* y, const float* t, const uint32_t* grp, int rows, float w, float* dy, float* loss,
          cudaStream_t s) {
  if (!rows) return;
  k_loss<<<(rows + 7) / 8, 256, 0, s>>>(y, t, w > 0.0f ? grp : nullptr, rows, w, dy, loss);
  SW_LAUNCH_CHECK();
}

// ---- backward ----
// TMEM columns: dH1 and then the dE tiles 0 .. 127, dW2 128 .. 255, dX 256 .. 319,
// dW1 384 .. 511.
__global__ void __launch_bounds__(kThreads, 1) k_backward(const u64* __restrict__ rows, int W, int n, u32 count,
                                                          const float* __restrict__ dy,
                                                          const bf16* __restrict__ weights,
                                                          const float* __restrict__ params, Activations act,
                                                          float* grad, float* de) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t *const sA = smem, *const sB = smem + kBwdB, *const sC = smem + kBwdC, *const sT = smem + kBwdT;
  u64* const s_rows = reinterpret_cast<u64*>(smem + kBwdRows);  // [128][8]
  u32* const slot = reinterpret_cast<u32*>(smem + kBwdBar + 16);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, q = warp & 3, half = warp >> 2;
  const u32 i0 = blockIdx.x * kRows;
  const int r = q * 32 + lane;
  const u32 row = i0 + r;
  const bool in = row < count;
  const int words = (n + 63) / 64;
  Tc tc;
  tc.open(sm_addr(smem + kBwdBar), sm_addr(slot), slot, 512);
  for (int e = tid; e < kRows * words; e += kThreads) {
    const int rr = e / words, w = e - rr * words;
    s_rows[rr * 8 + w] = i0 + rr < count ? rows[(size_t)(i0 + rr) * W + w] : 0ULL;
  }
  const float d = in ? dy[row] : 0.0f;
  if (half == 0) {
    float b = d;
#pragma unroll
    for (int o = 16; o; o >>= 1) b += __shfl_xor_sync(0xffffffffu, b, o);
    if (lane == 0) atomicAdd(grad + kOffB3, b);
  }
  // head: dw3, db2, dH2 = dy w3^T * [h2 open] (rows and columns); h1 by columns
#pragma unroll
  for (int cb = 0; cb < 2; ++cb) {
    const int c = half * 64 + cb * 32;
    const u32 open = in ? act.open2[(size_t)row * 4 + (c >> 5)] : 0u;
    float v[32];
    u32 p[16];
    const uint4* h = reinterpret_cast<const uint4*>(act.h2 + (size_t)row * kHidden + c);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint4 x = in ? h[i] : make_uint4(0, 0, 0, 0);
      p[4 * i] = x.x;
      p[4 * i + 1] = x.y;
      p[4 * i + 2] = x.z;
      p[4 * i + 3] = x.w;
    }
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = d * unpack(p[i / 2], i & 1);
    atomicAdd(grad + kOffW3 + c + lane, column_sums(v));
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = (open >> i) & 1u ? d * __ldg(params + kOffW3 + c + i) : 0.0f;
    put_rows(v, r, c, sA, nullptr);
#pragma unroll
    for (int i = 0; i < 16; ++i) p[i] = pack2(v[2 * i], v[2 * i + 1]);
    put_columns(p, r, c, sT, kSlice);
    atomicAdd(grad + kOffB2 + c + lane, column_sums(v));
    h = reinterpret_cast<const uint4*>(act.h1 + (size_t)row * kHidden + c);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint4 x = in ? h[i] : make_uint4(0, 0, 0, 0);
      p[4 * i] = x.x;
      p[4 * i + 1] = x.y;
      p[4 * i + 2] = x.z;
      p[4 * i + 3] = x.w;
    }
    put_columns(p, r, c, sC, kSlice);
  }
  copy_in(sB, weights + kOffW2B, kStagedW2 * 2);
  tc.publish();
  if (tid == 0) {
    issue_mma(tc.tmem, sm_addr(sA), sm_addr(sB), kSlice, 2, kHidden, false);        // dH1 = dH2 · W2^T
    issue_mma(tc.tmem + 128, sm_addr(sC), sm_addr(sT), kSlice, 2, kHidden, false);  // dW2 = h1^T · dH2
    tc.commit();
  }
  bool ok = tc.wait();
  if (ok) {
#pragma unroll
    for (int cb = 0; cb < 2; ++cb) {
      const int c = half * 64 + cb * 32;
      const u32 open = in ? act.open1[(size_t)row * 4 + (c >> 5)] : 0u;
      float v[32];
      ld32(tc.tmem, q * 32, c, v);
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = (open >> i) & 1u ? v[i] : 0.0f;
      put_rows(v, r, c, sA, nullptr);
      u32 p[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) p[i] = pack2(v[2 * i], v[2 * i + 1]);
      put_columns(p, r, c, sT, kSlice);
      atomicAdd(grad + kOffB1 + c + lane, column_sums(v));
      ld32(tc.tmem + 128, q * 32, c, v);
      float4* const g = reinterpret_cast<float4*>(grad + kOffW2 + (size_t)r * kHidden + c);
#pragma unroll
      for (int i = 0; i < 8; ++i) atomicAdd(g + i, make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]));
    }
    {  // x by columns: rows 0 .. 63 of the operand, the others zero
      u32 p[16];
      const uint4* const h = reinterpret_cast<const uint4*>(act.x + (size_t)row * kEmb + half * 32);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint4 x = in ? h[i] : make_uint4(0, 0, 0, 0);
        p[4 * i] = x.x;
        p[4 * i + 1] = x.y;
        p[4 * i + 2] = x.z;
        p[4 * i + 3] = x.w;
      }
      put_columns(p, r, half * 32, sC, kSlice);
      for (int e = tid; e < 1024; e += kThreads)
        *reinterpret_cast<uint4*>(sC + (e >> 9) * kSlice + kSlice / 2 + (e & 511) * 16) = make_uint4(0, 0, 0, 0);
    }
    copy_in(sB, weights + kOffW1B, kStagedW1 * 2);
    tc.publish();
    if (tid == 0) {
      issue_mma(tc.tmem + 256, sm_addr(sA), sm_addr(sB), kSlice / 2, 2, kEmb, false);  // dX = dH1 · W1^T
      issue_mma(tc.tmem + 384, sm_addr(sC), sm_addr(sT), kSlice, 2, kHidden, false);   // dW1 = x^T · dH1
      tc.commit();
    }
    ok = tc.wait();
  }
  if (ok) {
    float v[32];
    if (q < 2) {
#pragma unroll
      for (int cb = 0; cb < 2; ++cb) {
        const int c = half * 64 + cb * 32;
        ld32(tc.tmem + 384, q * 32, c, v);
        float4* const g = reinterpret_cast<float4*>(grad + kOffW1 + (size_t)r * kHidden + c);
#pragma unroll
        for (int i = 0; i < 8; ++i) atomicAdd(g + i, make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]));
      }
    }
    ld32(tc.tmem + 256, q * 32, half * 32, v);
    u32 p[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) p[i] = pack2(v[2 * i], v[2 * i + 1]);
    put_columns(p, r, half * 32, sB, kSlice / 2);
  }
  // dE += bits^T · dX, 128 states at a time
  for (int t0 = 0; t0 < n && ok; t0 += kRows) {
    for (int e = tid; e < kRows * 16; e += kThreads) {
      const int m = e & 127, kg = e >> 7, s = t0 + m;  // state s, rows 8 kg .. 8 kg + 7
      u32 b[4] = {0, 0, 0, 0};
      if (s < n) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if ((s_rows[(8 * kg + j) * 8 + (s >> 6)] >> (63 - (s & 63))) & 1ULL) b[j >> 1] |= j & 1 ? 0x3F800000u : 0x3F80u;
      }
      *reinterpret_cast<uint4*>(sA + (kg >> 3) * kSlice + core_offset(m, (kg & 7) * 8)) =
          make_uint4(b[0], b[1], b[2], b[3]);
    }
    tc.publish();
    if (tid == 0) {
      issue_mma(tc.tmem, sm_addr(sA), sm_addr(sB), kSlice / 2, 2, kEmb, false);
      tc.commit();
    }
    ok = tc.wait();
    if (ok) {
      float v[32];
      ld32(tc.tmem, q * 32, half * 32, v);
      if (t0 + r < n) {
        float4* const g = reinterpret_cast<float4*>(de + (size_t)(t0 + r) * kEmb + half * 32);
#pragma unroll
        for (int i = 0; i < 8; ++i) atomicAdd(g + i, make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]));
      }
    }
  }
  tc.close(512);
}

void backward(const u64* rows, int W, int n, u32 count, const float* dy, const bf16* weights, const float* params,
              const Activations& act, float* grad, float* de, cudaStream_t s) {
  if (!count) return;
  ensure_smem_limit((const void*)k_backward, kBwdSmem);
  k_backward<<<(count + kRows - 1) / kRows, kThreads, kBwdSmem, s>>>(rows, W, n, count, dy, weights, params, act, grad,
                                                                    de);
  SW_LAUNCH_CHECK();
}

bool tc_error() {
  u32 v = 0;
  SW_CUDA(cudaMemcpyFromSymbol(&v, g_tc_error, sizeof(u32)));
  return v != 0;
}

// ---- embeddings ----
// Block of 128 states: feat · Phi is one K = 16 product.
__global__ void __launch_bounds__(kThreads) k_embed(const float* __restrict__ feat, const float* __restrict__ params,
                                                    int n, float* __restrict__ epre, bf16* __restrict__ staged) {
  __shared__ __align__(1024) uint8_t sA[kSlice];
  __shared__ __align__(1024) uint8_t sB[kSlice / 2];
  __shared__ __align__(16) uint64_t s_bar[2];
  __shared__ u32 slot;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, q = warp & 3, half = warp >> 2;
  const int s0 = blockIdx.x * kRows;
  Tc tc;
  tc.open(sm_addr(s_bar), sm_addr(&slot), &slot, 64);
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
        float a = 0.0f;
        if (st < n) {
          a = v[i] + params[kOffC + j];
          epre[(size_t)st * kEmb + j] = a;
        }
        staged[(size_t)(st >> 6) * 64 * kEmb + core_offset(j, st & 63) / 2] = __float2bfloat16(fmaxf(a, 0.0f));
      }
    }
  }
  tc.close(64);
}

void embed(const float* feat, const float* params, int n, float* epre, bf16* staged, cudaStream_t s) {
  k_embed<<<(n + kRows - 1) / kRows, kThreads, 0, s>>>(feat, params, n, epre, staged);
  SW_LAUNCH_CHECK();
}

// Block of 32 states, thread (feature f, columns): dPhi += feat^T · bf16(de open),
// dc += column sums; de cleared.
constexpr int kEbStates = 32;
__global__ void __launch_bounds__(256) k_embed_back(const float* __restrict__ feat, const float* __restrict__ epre, int n,
                                                    float* __restrict__ de, float* grad) {
  __shared__ float s_d[kEbStates][kEmb];   // masked, fp32
  __shared__ float s_f[kEbStates][kFeat];  // rounded to bf16
  const int s0 = blockIdx.x * kEbStates, tid = threadIdx.x;
  for (int e = tid; e < kEbStates * kEmb; e += 256) {
    const int s = s0 + e / kEmb;
    float v = 0.0f;
    if (s < n) {
      const size_t at = (size_t)s * kEmb + e % kEmb;
      v = epre[at] > 0.0f ? de[at] : 0.0f;
      de[at] = 0.0f;
    }
    s_d[e / kEmb][e % kEmb] = v;
  }
  for (int e = tid; e < kEbStates * kFeat; e += 256) {
    const int s = s0 + e / kFeat;
    s_f[e / kFeat][e % kFeat] = s < n ? __bfloat162float(__float2bfloat16(feat[(size_t)s * kFeat + e % kFeat])) : 0.0f;
  }
  __syncthreads();
  const int j = tid & 63, fq = tid >> 6;  // features 4 fq .. 4 fq + 3
  float a[4] = {0, 0, 0, 0}, c = 0.0f;
  for (int s = 0; s < kEbStates; ++s) {
    const float v = s_d[s][j], b = __bfloat162float(__float2bfloat16(v));
    c += v;
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] += s_f[s][4 * fq + i] * b;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) atomicAdd(grad + kOffPhi + (4 * fq + i) * kEmb + j, a[i]);
  if (fq == 0) atomicAdd(grad + kOffC + j, c);
}

void embed_back(const float* feat, const float* epre, int n, float* de, float* grad, cudaStream_t s) {
  k_embed_back<<<(n + kEbStates - 1) / kEbStates, 256, 0, s>>>(feat, epre, n, de, grad);
  SW_LAUNCH_CHECK();
}

// ---- weights ----
// bf16 copies of W1[i][j] and W2[i][j] where the products read them: forward as
// B(N = j, K = i), backward as B(N = i, K = j).
__device__ __forceinline__ void stage_weight(bf16* w, int e, float value) {
  const bf16 b = __float2bfloat16(value);
  if (e >= kOffW1 && e < kOffB1) {
    const int i = (e - kOffW1) / kHidden, j = (e - kOffW1) % kHidden;
    w[kOffW1F + core_offset(j, i) / 2] = b;
    w[kOffW1B + (j >> 6) * (64 * 64) + core_offset(i, j & 63) / 2] = b;
  } else if (e >= kOffW2 && e < kOffB2) {
    const int i = (e - kOffW2) / kHidden, j = (e - kOffW2) % kHidden;
    w[kOffW2F + (i >> 6) * (128 * 64) + core_offset(j, i & 63) / 2] = b;
    w[kOffW2B + (j >> 6) * (128 * 64) + core_offset(i, j & 63) / 2] = b;
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

// Adam (Kingma & Ba 2015) with beta1 = 0.9, beta2 = 0.999, eps = 1e-8.
__global__ void k_adam(float* p, float* g, float* m, float* v, bf16* w, float lr, float c1, float c2) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= kParams) return;
  const float gr = g[e];
  g[e] = 0.0f;
  const float mm = 0.9f * m[e] + 0.1f * gr;
  const float vv = 0.999f * v[e] + 0.001f * gr * gr;
  m[e] = mm;
  v[e] = vv;
  const float np = p[e] - lr * (mm / c1) / (sqrtf(vv / c2) + 1e-8f);
  p[e] = np;
  stage_weight(w, e, np);
}

void adam(float* p, float* g, float* m, float* v, bf16* weights, float lr, int t, cudaStream_t s) {
  const float c1 = 1.0f - std::pow(0.9f, (float)t), c2 = 1.0f - std::pow(0.999f, (float)t);
  k_adam<<<(kParams + 255) / 256, 256, 0, s>>>(p, g, m, v, weights, lr, c1, c2);
  SW_LAUNCH_CHECK();
}

}  // namespace mlp
}  // namespace sw
