// Whole passes of the trace surrogate (sm_100a): one launch per layer.
//
// A layer is a small product (512 x 512 x 512 and down to 131072 x 4 x 16 at 512
// traces), so a pass is bound by launches and by the latency of each one, not by
// tensor or memory throughput.  layer_gemm therefore does a layer's whole step in
// one launch: the product on tcgen05.mma, fed by TMA, and in its epilogue what
// used to be launches of its own (the in-order sum of split K, bias and SiLU with
// the bf16 copy; backward, the activation's derivative).  The backward launch of a
// layer holds both of its products.  Split-K partials that need several CTAs and
// the bias gradients of all layers are finished by one launch at the end
// (finish_grads), and one launch updates all parameters (adam_all).  At 512 traces
// a training iteration takes 265 us instead of 1,230 (86 launches: products of
// 22-31 us from plain loads, 24 us a column sum, host calls for each), and 4,096
// predictions take 0.27 ms instead of 2.40, several batches sharing each launch.
// A layer's launch still costs about 10 us of latency (launch, tensor maps, TMA,
// epilogue), which is what bounds a pass.
//
// Results are those of the separate kernels bit for bit: the same splits of K in
// the same order, the same order of the column sums, the same elementwise
// arithmetic.
#include <algorithm>
#include <cmath>
#include <string>

#include "../../include/ifdtd_surrogate.h"
#include "errors.cuh"
#include "launch.cuh"
#include "silu.cuh"
#include "tc_common.cuh"

namespace ifdtd {
namespace tc {

int gemm_splits(int m, int n, int k, bool forward);  // gemm_tcgen05.cu

constexpr int LM = 128, LK = 64, LTHREADS = 256;
constexpr int kMaxLayerStages = 12;
constexpr int LA_BYTES = LM * LK * 2;

// One product of a launch: D (m x n, fp32) = op(A) op(B).  Operands K-major
// (rows of 64 K elements, loaded as 64 x rows boxes) or MN-major (rows of 64 M or N
// elements, 64 x 64 boxes side by side).
enum Epilogue : int { kStore = 0, kPartial = 1, kForward = 2, kBackward = 3 };
struct Job {
  CUtensorMap a, b;
  int m, n, nk;              // nk: chunks of 64 along K
  int a_mn, b_mn;            // operand is MN-major
  int tn, tiles_m, tiles_n;  // output tile 128 x tn
  int kps, out_splits;       // chunks per split; splits spread over CTAs (the others: accumulators of one CTA)
  int stages, stage_bytes;
  int epilogue, act;
  float* out;                // kForward: z (may be null); kBackward: dz; kStore: D; kPartial: (out_splits, m, n)
  const float* extra;        // kForward: bias; kBackward: z of the layer below
  __nv_bfloat16* out16;      // kForward: y (may be null); kBackward: dz as bf16
  int cols16, ld16;          // kBackward: row length and pitch of out16
};
struct Launch {
  Job job[2];
  int first_of_second;  // blocks of job 0
};

// MN-major operand with the 128-byte swizzle: rows of 64 elements along M or N
// (128 bytes), 8-row groups along K 1024 bytes apart (stride byte offset), blocks
// of 64 elements 8192 bytes apart (leading byte offset).  A K step of 16 advances
// the start address by 2048 bytes.
__device__ __forceinline__ uint64_t smem_desc_mn128(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)(8192u >> 4) << 16) | ((uint64_t)(1024u >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

__device__ __forceinline__ void tmem_ld16(uint32_t addr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(addr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int q = 0; q < 16; ++q) v[q] = __uint_as_float(r[q]);
}

// n <= 16 values to p; 16-byte stores where the address and count allow.
__device__ __forceinline__ void put16(float* p, const float (&v)[16], int n, bool vec) {
  if (vec) {
#pragma unroll
    for (int q = 0; q < 16; q += 4)
      if (q < n) *reinterpret_cast<float4*>(p + q) = make_float4(v[q], v[q + 1], v[q + 2], v[q + 3]);
  } else {
#pragma unroll
    for (int q = 0; q < 16; ++q)
      if (q < n) p[q] = v[q];
  }
}
__device__ __forceinline__ void put16(__nv_bfloat16* p, const float (&v)[16], int n, bool vec) {
  if (vec) {
#pragma unroll
    for (int q = 0; q < 16; q += 8)
      if (q < n) {
        __nv_bfloat162 h[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v[q + 2 * i], v[q + 2 * i + 1]);
        *reinterpret_cast<uint4*>(p + q) = *reinterpret_cast<uint4*>(h);
      }
  } else {
#pragma unroll
    for (int q = 0; q < 16; ++q)
      if (q < n) p[q] = __float2bfloat16(v[q]);
  }
}

// n <= 16 values from p (zero beyond), 16 bytes at a time where the address allows.
__device__ __forceinline__ void get16(const float* p, float (&v)[16], int n, bool vec) {
  if (vec) {
#pragma unroll
    for (int q = 0; q < 16; q += 4) {
      const float4 x = q < n ? __ldg(reinterpret_cast<const float4*>(p + q)) : make_float4(0.f, 0.f, 0.f, 0.f);
      v[q] = x.x;
      v[q + 1] = x.y;
      v[q + 2] = x.z;
      v[q + 3] = x.w;
    }
  } else {
#pragma unroll
    for (int q = 0; q < 16; ++q) v[q] = q < n ? __ldg(p + q) : 0.f;
  }
}

// One output tile (and split) per CTA of 256 threads.  Thread 0 streams the K
// chunks through the stage ring (all of them at once where they fit), issues the
// MMAs of chunk c into accumulator c / kps and commits them to the stage; then
// warps w and w + 4 read the TMEM lanes 32 (w % 4) .. + 31, alternate groups of 16
// columns each, and run the epilogue, whose other operands were loaded meanwhile.
// Every mbarrier wait is bounded; one that runs out sets the status bit and the CTA
// skips its epilogue after its own copies and MMAs have ended.  Two waits have no
// bound: tcgen05.alloc, while other CTAs of the SM hold the columns, and
// wait_previous, for the end of the launch before.  A CTA therefore lets the next
// launch begin only once its own columns are allocated: a CTA of the next launch may
// hold columns in wait_previous, and if this launch still needed them, neither would
// go on.  With that order a launch never waits for one that follows it, and CTAs of
// the same launch that wait for each other's columns end one after the other.
__global__ void __launch_bounds__(LTHREADS) layer_gemm(const __grid_constant__ Launch L) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full[kMaxLayerStages], empty[kMaxLayerStages], done;
  __shared__ float s_bias[LM];
  __shared__ uint32_t tmem_slot;
  __shared__ int failed;
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const bool second = (int)blockIdx.x >= L.first_of_second;
  const Job& J = L.job[second ? 1 : 0];
  int t = (int)blockIdx.x - (second ? L.first_of_second : 0);
  const int tm = t % J.tiles_m;
  t /= J.tiles_m;
  const int tile_n = t % J.tiles_n, split = t / J.tiles_n;
  const int c0 = J.out_splits > 1 ? split * J.kps : 0, c1 = J.out_splits > 1 ? min(c0 + J.kps, J.nk) : J.nk, n = c1 - c0;
  const int accs = J.out_splits > 1 ? 1 : (J.nk + J.kps - 1) / J.kps;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t cols = 32;
  while ((int)cols < accs * J.tn) cols *= 2;
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  __syncthreads();
  launch_next();
  auto load = [&](int c) {
    const int s = c % J.stages;
    const uint32_t as = smem_u32(smem + s * J.stage_bytes), bs = as + LA_BYTES, bar = smem_u32(&full[s]);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(J.stage_bytes) : "memory");
    const int k = (c0 + c) * LK;
    if (J.a_mn) {
      tma_load_2d(as, &J.a, tm * LM, k, bar);
      tma_load_2d(as + 8192, &J.a, tm * LM + 64, k, bar);
    } else {
      tma_load_2d(as, &J.a, k, tm * LM, bar);
    }
    if (J.b_mn)
      for (int q = 0; q < J.tn / 64; ++q) tma_load_2d(bs + q * 8192, &J.b, tile_n * J.tn + 64 * q, k, bar);
    else
      tma_load_2d(bs, &J.b, k, tile_n * J.tn, bar);
  };
  int loaded = 0;
  if (threadIdx.x == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&J.a)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&J.b)) : "memory");
    for (int s = 0; s < J.stages; ++s) {
      mbar_init_x(smem_u32(&full[s]), 1);
      mbar_init_x(smem_u32(&empty[s]), 1);
    }
    mbar_init_x(smem_u32(&done), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    failed = 0;
    wait_previous();
    for (; loaded < min(n, J.stages); ++loaded) load(loaded);
  } else {
    wait_previous();
  }
  // this thread's row and columns of the epilogue, and its first other operands
  const int row = tm * LM + 32 * (warp & 3) + lane, n0 = tile_n * J.tn, width = min(J.tn, J.n - n0), first = 16 * (warp >> 2);
  const bool vec = J.n % 4 == 0, back = J.epilogue == kBackward && J.act != 0 && row < J.m;
  if (J.epilogue == kForward)
    for (int i = threadIdx.x; i < width; i += LTHREADS) s_bias[i] = __ldg(J.extra + n0 + i);
  float z[16];
  const float* const zrow = J.extra + (size_t)row * J.n + n0;
  if (back && first < width) get16(zrow + first, z, width - first, vec);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  if (threadIdx.x == 0) {
    // fp32 accumulator, bf16 A and B, their majorness, N, M 128
    const uint32_t instr = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)J.a_mn << 15) | ((uint32_t)J.b_mn << 16) |
                           ((uint32_t)(J.tn >> 3) << 17) | ((uint32_t)(LM >> 4) << 24);
    int used = 0;
    bool ok = true;
    for (int c = 0; c < n && ok; ++c) {
      const int s = c % J.stages;
      ok = wait_bounded(smem_u32(&full[s]), (uint32_t)(c / J.stages) & 1u);
      if (!ok) break;
      used = c + 1;
      tc_fence_after();
      const uint32_t as = smem_u32(smem + s * J.stage_bytes), bs = as + LA_BYTES;
      const uint32_t d = tmem + (uint32_t)(accs > 1 ? c / J.kps * J.tn : 0);
      const bool fresh = accs > 1 ? c % J.kps == 0 : c == 0;
#pragma unroll
      for (int kk = 0; kk < LK / 16; ++kk) {
        const uint64_t ad = J.a_mn ? smem_desc_mn128(as + kk * 2048) : smem_desc_sw128(as + kk * 32);
        const uint64_t bd = J.b_mn ? smem_desc_mn128(bs + kk * 2048) : smem_desc_sw128(bs + kk * 32);
        asm volatile(
            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
            " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
            "l"(ad), "l"(bd), "r"(instr), "r"(fresh && kk == 0 ? 0u : 1u)
            : "memory");
      }
      if (c + 1 == n) break;
      tc_commit(smem_u32(&empty[s]));
      if (c >= 1 && c - 1 + J.stages < n) {
        // the stage of the chunk before is free once its MMAs are done
        ok = wait_bounded(smem_u32(&empty[(c - 1) % J.stages]), (uint32_t)((c - 1) / J.stages) & 1u);
        if (ok) load(loaded++);
      }
    }
    if (!ok) {
      failed = 1;
      for (int c = used; c < loaded; ++c) wait_bounded(smem_u32(&full[c % J.stages]), (uint32_t)(c / J.stages) & 1u);
    }
    tc_commit(smem_u32(&done));
  }
  __syncwarp();
  if (!wait_bounded(smem_u32(&done), 0u)) failed = 1;
  __syncthreads();
  tc_fence_after();
  if (!failed) {
    const uint32_t lane_base = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
    float* const out = J.out + ((J.epilogue == kPartial ? (size_t)split * J.m : (size_t)0) + row) * J.n + n0;
#pragma unroll 1
    for (int cb = first; cb < width; cb += 32) {
      float v[16];
      tmem_ld16(lane_base + (uint32_t)cb, v);
      for (int q = 1; q < accs; ++q) {  // splits of K in order
        float w[16];
        tmem_ld16(lane_base + (uint32_t)(q * J.tn + cb), w);
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] += w[i];
      }
      if (row >= J.m) continue;
      const int left = min(16, width - cb);
      const size_t at = (size_t)row * J.n + n0 + cb;
      if (J.epilogue == kForward) {
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = v[i] + (i < left ? s_bias[cb + i] : 0.f);
        if (J.out) put16(out + cb, v, left, vec);
        if (J.out16) {
          if (J.act) {
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = nn::silu(v[i]);
          }
          put16(J.out16 + at, v, left, J.n % 8 == 0);
        }
      } else if (J.epilogue == kBackward) {
        if (back) {
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = v[i] * nn::silu_grad(z[i]);
          if (cb + 32 < width) get16(zrow + cb + 32, z, width - cb - 32, vec);
        }
        put16(out + cb, v, left, vec);
        if (J.ld16 == J.cols16) {
          put16(J.out16 + at, v, left, J.n % 8 == 0);
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i)
            if (i < left) J.out16[(at + i) / J.cols16 * J.ld16 + (at + i) % J.cols16] = __float2bfloat16(v[i]);
        }
      } else {
        put16(out + cb, v, left, vec);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
  }
}

// dz (fp32, may be null where it equals dy) and its bf16 copy of the last layer.
__global__ void last_grad(int rows, int cols, int ld16, const float* __restrict__ z, const float* __restrict__ dy, int act,
                          float* __restrict__ dz, __nv_bfloat16* __restrict__ dz16) {
  launch_next();
  wait_previous();
  const size_t n = (size_t)rows * cols;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float v = act ? dy[i] * nn::silu_grad(z[i]) : dy[i];
    if (dz) dz[i] = v;
    dz16[ld16 == cols ? i : i / cols * ld16 + i % cols] = __float2bfloat16(v);
  }
}

// ---------------------------------------------------------------------------
// The end of a backward pass: split-K partials added in split order, and bias
// gradients.  A bias gradient sums its column in 256 interleaved partial sums
// (rows t, t + 256, ...; each in row order) added as a binary tree; bound by the
// latency of reaching the rows.  Few rows: a block takes all 256 sums of 16
// columns, each thread one column of 16 sums.  Many rows (tall): a block takes 8
// of the sums and up to 32 columns; all its threads bring the rows to shared
// memory with every load in flight, one thread per (sum, column) adds them in
// order, and the block that finishes a column group last (a ticket) adds the tree.
// One block per column walking its rows took 24 us a layer, 190 us a pass.
// ---------------------------------------------------------------------------
constexpr int kMaxJobs = 32, kT = 8, kColGroup = 32, kShortCols = 16, kPieceReals = 8192, kTallRows = 16 * 256;
struct SumJob {
  const float* x;
  float* out;
  int rows, cols, first;  // first: the job's first block
  float* part;            // (256, cols), tall jobs
  int* ticket;            // one per column group, zero between launches
};
struct AddJob {
  const float* partial;
  float* out;
  int splits, first;
  long long n;
};
struct FinishLaunch {
  SumJob sum[kMaxJobs];
  AddJob add[kMaxJobs];
  int sums, adds, add_blocks_from;
};
constexpr int kAddPerBlock = 256, kBatch = 32;  // kBatch: loads in flight per thread

// The tree over buf (256, w), then the column sums to out.
__device__ __forceinline__ void column_tree(float* buf, int w, float* out) {
  for (int h = 128; h > 0; h >>= 1) {
    for (int i = threadIdx.x; i < h * w; i += 256) buf[i] += buf[i + h * w];
    __syncthreads();
  }
  if (threadIdx.x < w) out[threadIdx.x] = buf[threadIdx.x];
}

__global__ void __launch_bounds__(256) finish_grads(const __grid_constant__ FinishLaunch F) {
  __shared__ float buf[kPieceReals];
  __shared__ int last;
  launch_next();
  wait_previous();
  const int b = blockIdx.x;
  if (b >= F.add_blocks_from) {
    int j = 0;
    while (j + 1 < F.adds && b >= F.add[j + 1].first) ++j;
    const AddJob& A = F.add[j];
    const long long i = (long long)(b - A.first) * kAddPerBlock + threadIdx.x;
    if (i < A.n) {
      const float* const p = A.partial + i;
      float acc = p[0];
      for (int z0 = 1; z0 < A.splits; z0 += kBatch) {
        float x[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u)
          if (z0 + u < A.splits) x[u] = p[(size_t)(z0 + u) * A.n];
#pragma unroll
        for (int u = 0; u < kBatch; ++u)
          if (z0 + u < A.splits) acc += x[u];
      }
      A.out[i] = acc;
    }
    return;
  }
  int j = 0;
  while (j + 1 < F.sums && b >= F.sum[j + 1].first) ++j;
  const SumJob& S = F.sum[j];
  if (S.rows < kTallRows) {
    const int c0 = (b - S.first) * kShortCols, w = min(kShortCols, S.cols - c0);
    const int c = threadIdx.x % kShortCols, t0 = threadIdx.x / kShortCols;
    if (c < w) {
      // 16 of the partial sums (rows t, then t + 256, ...)
      const float* const x = S.x + c0 + c;
      constexpr int kSums = kShortCols, kStep = 256 / kSums;
      float s[kSums];
#pragma unroll
      for (int u = 0; u < kSums; ++u) s[u] = 0.f;
      for (int r0 = 0; r0 < S.rows; r0 += 512) {
        float v[2 * kSums];
#pragma unroll
        for (int u = 0; u < 2 * kSums; ++u) {
          const int r = r0 + u / kSums * 256 + t0 + u % kSums * kStep;
          if (r < S.rows) v[u] = x[(size_t)r * S.cols];
        }
#pragma unroll
        for (int u = 0; u < 2 * kSums; ++u) {
          const int r = r0 + u / kSums * 256 + t0 + u % kSums * kStep;
          if (r < S.rows) s[u % kSums] += v[u];
        }
      }
#pragma unroll
      for (int u = 0; u < kSums; ++u) buf[(t0 + u * kStep) * w + c] = s[u];
    }
    __syncthreads();
    column_tree(buf, w, S.out + c0);
    return;
  }
  const int groups = (S.cols + kColGroup - 1) / kColGroup, g = (b - S.first) % groups, t0 = (b - S.first) / groups * kT;
  const int c0 = g * kColGroup, w = min(kColGroup, S.cols - c0);
  const int t = threadIdx.x / w, c = threadIdx.x % w;  // this thread's sum and column
  const bool adds = t < kT;
  const int per_sum = (S.rows + 255) / 256, piece = kPieceReals / (kT * w);  // rows of each sum, and of a piece
  const bool vec = S.cols % 4 == 0;
  float s = 0.f;
  for (int r0 = 0; r0 < per_sum; r0 += piece) {
    const int here = min(piece, per_sum - r0);
    // value i of the piece: row ((r0 + i / (kT w)) 256 + t0 + (i / w) % kT), column c0 + i % w
    if (vec) {
      const int w4 = w / 4, n4 = here * kT * w4;
      float4 v[kPieceReals / 4 / 256];
#pragma unroll
      for (int u = 0; u < kPieceReals / 4 / 256; ++u) {
        const int i = threadIdx.x + 256 * u, q = i / w4, row = (r0 + q / kT) * 256 + t0 + q % kT;
        if (i < n4 && row < S.rows) v[u] = *reinterpret_cast<const float4*>(S.x + (size_t)row * S.cols + c0 + 4 * (i - q * w4));
      }
#pragma unroll
      for (int u = 0; u < kPieceReals / 4 / 256; ++u)
        if (threadIdx.x + 256 * u < n4) reinterpret_cast<float4*>(buf)[threadIdx.x + 256 * u] = v[u];
    } else {
      for (int i = threadIdx.x; i < here * kT * w; i += 256) {
        const int q = i / w, row = (r0 + q / kT) * 256 + t0 + q % kT;
        if (row < S.rows) buf[i] = S.x[(size_t)row * S.cols + c0 + (i - q * w)];
      }
    }
    __syncthreads();
    if (adds) {
      const int valid = min(here, (S.rows - t0 - t + 255) / 256 - r0);  // rows of this sum in the piece
      const float* const p = buf + t * w + c;
      int q = 0;
      for (; q + 16 <= valid; q += 16) {
        float v[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) v[u] = p[(q + u) * kT * w];
#pragma unroll
        for (int u = 0; u < 16; ++u) s += v[u];
      }
      for (; q < valid; ++q) s += p[q * kT * w];
    }
    __syncthreads();
  }
  if (adds) S.part[(size_t)(t0 + t) * S.cols + c0 + c] = s;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(S.ticket + g, 1) == 256 / kT - 1;
  __syncthreads();
  if (!last) return;
  if (threadIdx.x == 0) S.ticket[g] = 0;
  __threadfence();
  for (int i = threadIdx.x; i < 256 * w; i += 256) buf[i] = __ldcg(S.part + (size_t)(i / w) * S.cols + c0 + i % w);
  __syncthreads();
  column_tree(buf, w, S.out + c0);
}

// Adam on every parameter tensor of a network in one launch (the arithmetic of
// the single-tensor kernel).
struct AdamJob {
  float *w, *m, *v;
  const float* g;
  __nv_bfloat16* w16;
  int n, first, vec;
};
struct AdamLaunch {
  AdamJob job[2 * kMaxJobs];
  int jobs;
};
constexpr int kAdamPerBlock = 1024;
// The roundings are those the single-tensor kernel is compiled to (fused multiply-adds spelled out).
__device__ __forceinline__ float adam_one(float& w, float g, float& m, float& v, float lr, float b1, float b2, float eps,
                                          float c1, float c2) {
  m = __fmaf_rn(1.f - b1, g, __fmul_rn(b1, m));
  v = __fmaf_rn(__fmul_rn(1.f - b2, g), g, __fmul_rn(b2, v));
  w = w - lr * (m / c1) / (sqrtf(v / c2) + eps);
  return w;
}
// A thread takes four consecutive parameters with 16-byte loads where the tensor allows.
__global__ void __launch_bounds__(256) adam_all(const __grid_constant__ AdamLaunch P, float lr, float b1, float b2,
                                                float eps, float c1, float c2) {
  wait_previous();
  int j = 0;
  while (j + 1 < P.jobs && (int)blockIdx.x >= P.job[j + 1].first) ++j;
  const AdamJob& A = P.job[j];
  const int i = ((int)blockIdx.x - A.first) * kAdamPerBlock + 4 * (int)threadIdx.x;
  if (A.vec && i < A.n) {
    float4 w = *reinterpret_cast<const float4*>(A.w + i), m = *reinterpret_cast<const float4*>(A.m + i);
    float4 v = *reinterpret_cast<const float4*>(A.v + i);
    const float4 g = *reinterpret_cast<const float4*>(A.g + i);
    __nv_bfloat162 h[2];
    h[0].x = __float2bfloat16(adam_one(w.x, g.x, m.x, v.x, lr, b1, b2, eps, c1, c2));
    h[0].y = __float2bfloat16(adam_one(w.y, g.y, m.y, v.y, lr, b1, b2, eps, c1, c2));
    h[1].x = __float2bfloat16(adam_one(w.z, g.z, m.z, v.z, lr, b1, b2, eps, c1, c2));
    h[1].y = __float2bfloat16(adam_one(w.w, g.w, m.w, v.w, lr, b1, b2, eps, c1, c2));
    *reinterpret_cast<float4*>(A.w + i) = w;
    *reinterpret_cast<float4*>(A.m + i) = m;
    *reinterpret_cast<float4*>(A.v + i) = v;
    if (A.w16) *reinterpret_cast<uint2*>(A.w16 + i) = *reinterpret_cast<uint2*>(h);
  } else {
    for (int k = i; k < min(i + 4, A.n); ++k) {
      const float w = adam_one(A.w[k], A.g[k], A.m[k], A.v[k], lr, b1, b2, eps, c1, c2);
      if (A.w16) A.w16[k] = __float2bfloat16(w);
    }
  }
}

namespace {

int failed_launch(const char* what, cudaError_t e) {
  return record_error(IFDTD_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

int pitch8(int cols) { return (cols + 7) / 8 * 8; }

// Fill the shape of a job.  a, b: bf16 matrices as they lie in memory, lda / ldb
// elements per row.  forward: whether the separate kernels would take this
// product's K in one piece when its 128 x 256 tiles fill enough SMs.  rule_m: the
// rows that decide the splits (those of one pass, where several passes share a launch).
bool shape_job(Job& J, int m, int n, int k, const void* a, int lda, bool a_mn, const void* b, int ldb, bool b_mn,
               bool forward, bool spread, int rule_m) {
  J.m = m;
  J.n = n;
  J.nk = (k + LK - 1) / LK;
  J.a_mn = a_mn;
  J.b_mn = b_mn;
  J.tiles_m = (m + LM - 1) / LM;
  const int want = gemm_splits(rule_m, n, k, forward);
  J.kps = (J.nk + want - 1) / want;
  const int splits = (J.nk + J.kps - 1) / J.kps;
  J.out_splits = spread ? splits : 1;
  const int accs = spread ? 1 : splits;
  // the widest tile whose tiles still cover most SMs (512 x 512: 64 CTAs of 128 x 32;
  // MN-major tiles are whole 64-element blocks)
  const int least = b_mn ? 64 : 32;
  int tn = 128;
  while (tn > least && (J.tiles_m * J.out_splits * ((n + tn - 1) / tn) < 100 || accs * tn > 512 || tn / 2 >= n)) tn /= 2;
  J.tn = tn;
  J.tiles_n = (n + tn - 1) / tn;
  J.stage_bytes = LA_BYTES + tn * LK * 2;
  const int chunks = J.out_splits > 1 ? J.kps : J.nk;
  J.stages = std::max(1, std::min({chunks, kMaxLayerStages, (220 * 1024) / J.stage_bytes}));
  return accs * tn <= 512 && encode_rows(&J.a, a, a_mn ? k : m, a_mn ? m : k, lda, a_mn ? 64 : LM) &&
         encode_rows(&J.b, b, b_mn ? k : n, b_mn ? n : k, ldb, b_mn ? 64 : tn);
}

int blocks_of(const Job& J) { return J.tiles_m * J.tiles_n * J.out_splits; }

int launch_jobs(Launch& L, int jobs, cudaStream_t st) {
  int blocks = 0;
  for (int q = 0; q < jobs; ++q) {
    if (q == 1) L.first_of_second = blocks;
    blocks += blocks_of(L.job[q]);
  }
  if (jobs == 1) L.first_of_second = blocks;
  // more CTAs than SMs: fewer stages each, so that they are resident together
  const int per_sm = std::min(8, (blocks + 147) / 148), budget = 220 * 1024 / per_sm - 2048;
  size_t smem = 0;
  for (int q = 0; q < jobs; ++q) {
    Job& J = L.job[q];
    J.stages = std::min(J.stages, std::max(2, budget / J.stage_bytes));
    smem = std::max(smem, (size_t)J.stages * J.stage_bytes + 1024);
  }
  // the opt-in above 48 KiB of dynamic shared memory holds per device; setting it is cheap
  cudaError_t e = cudaFuncSetAttribute(layer_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024);
  if (e == cudaSuccess) e = launch_after(layer_gemm, blocks, LTHREADS, smem, st, L);
  return e == cudaSuccess ? IFDTD_OK : failed_launch("layer_gemm", e);
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

int check_layers(const ifdtd_nn_layer* layers, int n, int rows, const void* x) {
  if (!layers || n < 1 || n > kMaxJobs || rows <= 0 || !x)
    return record_error(IFDTD_ERR_ARGUMENT, "bad network arguments");
  if (!aligned16(x)) return record_error(IFDTD_ERR_UNSUPPORTED, "network input is not 16-byte aligned");
  int64_t r = rows;
  for (int i = 0; i < n; ++i) {
    const ifdtd_nn_layer& l = layers[i];
    if (l.fan_in <= 0 || l.fan_out <= 0 || l.expand <= 0 || l.act < 0 || l.act > 1 || !l.w16 || !l.bias || (!l.z && i + 1 == n) ||
        (i + 1 < n && (!l.y || l.fan_out != l.expand * layers[i + 1].fan_in)))
      return record_error(IFDTD_ERR_ARGUMENT, "bad network layer");
    if (l.fan_in % 8 || !aligned16(l.w16) || !aligned16(l.z) || (l.y && !aligned16(l.y)))
      return record_error(IFDTD_ERR_UNSUPPORTED, "network layer needs fan_in in eights and 16-byte aligned arrays");
    // the epilogue's rows and columns are 32-bit; the separate kernels take larger layers
    if (r * std::max(l.fan_out, l.fan_in) >= (int64_t)1 << 31)
      return record_error(IFDTD_ERR_UNSUPPORTED, "network layer of 2^31 values or more");
    r *= l.expand;
  }
  return IFDTD_OK;
}

}  // namespace

cudaError_t net_status(int reset, int* out) {
  cudaError_t e = cudaMemcpyFromSymbol(out, g_status, sizeof(int));
  if (e == cudaSuccess && reset) {
    const int zero = 0;
    e = cudaMemcpyToSymbol(g_status, &zero, sizeof(int));
  }
  return e;
}

}  // namespace tc
}  // namespace ifdtd

using namespace ifdtd;
using namespace ifdtd::tc;

extern "C" {

int32_t ifdtd_nn_forward(const ifdtd_nn_layer* layers, int32_t n, int32_t rows, int32_t rows_per_pass, const void* x,
                         void* stream) {
  const int rc = check_layers(layers, n, rows, x);
  if (rc) return rc;
  if (rows_per_pass < 1 || rows % rows_per_pass) return ifdtd::record_error(IFDTD_ERR_ARGUMENT, "bad rows per pass");
  for (int i = 0; i < n; ++i) {
    const ifdtd_nn_layer& l = layers[i];
    Launch L;
    Job& J = L.job[0];
    if (!shape_job(J, rows, l.fan_out, l.fan_in, x, l.fan_in, false, l.w16, l.fan_in, false, true, false, rows_per_pass))
      return ifdtd::record_error(IFDTD_ERR_UNSUPPORTED, "network layer shape");
    J.epilogue = kForward;
    J.act = l.act;
    J.out = l.z;
    J.extra = l.bias;
    J.out16 = i + 1 < n ? (__nv_bfloat16*)l.y : nullptr;
    J.cols16 = J.ld16 = l.fan_out;
    const int e = launch_jobs(L, 1, (cudaStream_t)stream);
    if (e) return e;
    x = l.y;
    rows *= l.expand;
    rows_per_pass *= l.expand;
  }
  return IFDTD_OK;
}

int32_t ifdtd_nn_backward_bytes(const ifdtd_nn_layer* layers, int32_t n, int32_t rows, int64_t* out) {
  if (!layers || n < 1 || rows <= 0 || !out) return ifdtd::record_error(IFDTD_ERR_ARGUMENT, "bad network arguments");
  int64_t bytes = 0;
  for (int i = 0; i < n; ++i) {
    const ifdtd_nn_layer& l = layers[i];
    const int64_t splits = gemm_splits(l.fan_out, l.fan_in, rows, false);
    bytes += 4 * (splits > 4 ? splits * l.fan_out * (int64_t)l.fan_in : 0) + 4 * 256 * (int64_t)l.fan_out + 32;
    rows *= l.expand;
  }
  *out = bytes;
  return IFDTD_OK;
}

int32_t ifdtd_nn_backward(const ifdtd_nn_layer* layers, int32_t n, int32_t rows, const void* x, const float* grad,
                          int32_t* tickets, void* workspace, int64_t workspace_bytes, void* stream) {
  int rc = check_layers(layers, n, rows, x);
  if (rc) return rc;
  int64_t need = 0;
  rc = ifdtd_nn_backward_bytes(layers, n, rows, &need);
  if (rc) return rc;
  if (!grad || !tickets || !workspace || !aligned16(workspace) || workspace_bytes < need)
    return ifdtd::record_error(IFDTD_ERR_ARGUMENT, "bad backward arguments");
  if (!aligned16(grad)) return ifdtd::record_error(IFDTD_ERR_UNSUPPORTED, "gradient is not 16-byte aligned");
  int row_of[kMaxJobs];
  int tickets_at[kMaxJobs], n_tickets = 0;
  for (int i = 0, r = rows; i < n; ++i) {
    const ifdtd_nn_layer& l = layers[i];
    if (!l.z || !l.gw || !l.gb || !l.dz16 || (!l.dz && (i + 1 < n || l.act)))
      return ifdtd::record_error(IFDTD_ERR_ARGUMENT, "bad network gradient arrays");
    // the epilogues store gw, dz and dz16, and the bias sums read dz, 16 bytes at a time (gb by single values)
    if (!aligned16(l.dz16) || !aligned16(l.dz) || !aligned16(l.gw))
      return ifdtd::record_error(IFDTD_ERR_UNSUPPORTED, "network gradient arrays are not 16-byte aligned");
    row_of[i] = r;
    r *= l.expand;
    tickets_at[i] = n_tickets;
    n_tickets += (l.fan_out + kColGroup - 1) / kColGroup;
  }
  if (n_tickets > IFDTD_NN_TICKETS) return ifdtd::record_error(IFDTD_ERR_UNSUPPORTED, "network too wide for one backward pass");
  cudaStream_t st = (cudaStream_t)stream;
  const ifdtd_nn_layer& top = layers[n - 1];
  {
    const size_t values = (size_t)row_of[n - 1] * top.fan_out;
    const cudaError_t e = launch_after(last_grad, (int)std::min<size_t>((values + 255) / 256, 148 * 8), 256, 0, st,
                                       row_of[n - 1], top.fan_out, pitch8(top.fan_out), (const float*)top.z, grad, top.act,
                                       top.act ? top.dz : (float*)nullptr, (__nv_bfloat16*)top.dz16);
    if (e != cudaSuccess) return failed_launch("last_grad", e);
  }
  FinishLaunch F = {};
  float* ws = static_cast<float*>(workspace);
  auto take = [&](int64_t values) {
    float* p = ws;
    ws += (values + 3) / 4 * 4;
    return p;
  };
  int blocks = 0;
  for (int i = n - 1; i >= 0; --i) {
    const ifdtd_nn_layer& l = layers[i];
    const int r = row_of[i], ld = pitch8(l.fan_out);
    const void* in = i ? layers[i - 1].y : x;
    Launch L;
    // the weight gradient: both operands with K = rows outermost
    Job& G = L.job[0];
    const int splits = gemm_splits(l.fan_out, l.fan_in, r, false);
    if (!shape_job(G, l.fan_out, l.fan_in, r, l.dz16, ld, true, in, l.fan_in, true, false, splits > 4, l.fan_out))
      return ifdtd::record_error(IFDTD_ERR_UNSUPPORTED, "network layer shape");
    G.epilogue = kStore;
    G.act = 0;
    G.out = l.gw;
    G.extra = nullptr;
    G.out16 = nullptr;
    G.cols16 = G.ld16 = l.fan_in;
    if (G.out_splits > 1) {
      G.epilogue = kPartial;
      G.out = take((int64_t)G.out_splits * G.m * G.n);
      F.add[F.adds++] = {G.out, l.gw, G.out_splits, 0, (long long)G.m * G.n};
    }
    if (i > 0) {
      // the input's gradient through the activation of the layer below
      const ifdtd_nn_layer& p = layers[i - 1];
      Job& D = L.job[1];
      if (!shape_job(D, r, l.fan_in, l.fan_out, l.dz16, ld, false, l.w16, l.fan_in, true, false, false, r))
        return ifdtd::record_error(IFDTD_ERR_UNSUPPORTED, "network layer shape");
      D.epilogue = kBackward;
      D.act = p.act;
      D.out = p.dz;
      D.extra = p.z;
      D.out16 = (__nv_bfloat16*)p.dz16;
      D.cols16 = p.fan_out;
      D.ld16 = pitch8(p.fan_out);
    }
    rc = launch_jobs(L, i > 0 ? 2 : 1, st);
    if (rc) return rc;
    SumJob& S = F.sum[F.sums++];
    S.x = i + 1 == n && !l.act ? grad : l.dz;
    S.out = l.gb;
    S.rows = r;
    S.cols = l.fan_out;
    S.first = blocks;
    S.part = take(256 * (int64_t)l.fan_out);
    S.ticket = tickets + tickets_at[i];
    blocks += r < kTallRows ? (l.fan_out + kShortCols - 1) / kShortCols : 256 / kT * ((l.fan_out + kColGroup - 1) / kColGroup);
  }
  F.add_blocks_from = blocks;
  for (int q = 0; q < F.adds; ++q) {
    F.add[q].first = blocks;
    blocks += (int)((F.add[q].n + kAddPerBlock - 1) / kAddPerBlock);
  }
  const cudaError_t e = launch_after(finish_grads, blocks, 256, 0, st, F);
  return e == cudaSuccess ? IFDTD_OK : failed_launch("finish_grads", e);
}

int32_t ifdtd_nn_adam_all(const ifdtd_nn_param* params, int32_t n, float lr, float beta1, float beta2, float eps,
                          int32_t step, void* stream) {
  if (!params || n < 1 || n > 2 * kMaxJobs || step < 1) return ifdtd::record_error(IFDTD_ERR_ARGUMENT, "bad adam arguments");
  AdamLaunch P;
  int blocks = 0;
  for (int i = 0; i < n; ++i) {
    const ifdtd_nn_param& p = params[i];
    if (p.n <= 0 || !p.w || !p.g || !p.m || !p.v) return ifdtd::record_error(IFDTD_ERR_ARGUMENT, "bad adam arguments");
    const bool vec = p.n % 4 == 0 && aligned16(p.w) && aligned16(p.m) && aligned16(p.v) && aligned16(p.g) && aligned16(p.w16);
    P.job[i] = {p.w, p.m, p.v, p.g, (__nv_bfloat16*)p.w16, p.n, blocks, vec};
    blocks += (p.n + kAdamPerBlock - 1) / kAdamPerBlock;
  }
  P.jobs = n;
  const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
  const cudaError_t e = launch_after(adam_all, blocks, 256, 0, (cudaStream_t)stream, P, lr, beta1, beta2, eps, c1, c2);
  return e == cudaSuccess ? IFDTD_OK : failed_launch("adam_all", e);
}

}  // extern "C"
