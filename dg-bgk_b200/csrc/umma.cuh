// Blackwell (sm_100a) 5th-generation tensor-core GEMM for the warm-start
// MLP: C[M x N] = A[M x K] * B[N x K]^T with A and B in BF16, both K-major
// (row-major with the reduction index contiguous), accumulated in FP32 in
// tensor memory.
//
// One CTA computes one 128 x BN tile of C with 128 threads:
//   * an elected thread of warp 0 loads 128 x 64 (A) and BN x 64 (B) BF16
//     boxes per K-block with TMA (128-byte swizzle) into a ring of stages;
//   * an elected thread of warp 1 issues tcgen05.mma (kind::f16, M = 128,
//     N = BN, K = 16 per instruction, four per K-block) and frees each stage
//     with tcgen05.commit on the stage's "empty" mbarrier;
//   * all four warps read the accumulator with tcgen05.ld (warp w owns TMEM
//     lanes 32w..32w+31, i.e. rows 32w..32w+31 of the tile) and run the
//     epilogue.
// Every mbarrier wait is bounded; on expiry the CTA records an error flag,
// waits (bounded) for its own copies and MMAs, frees its tensor memory and
// returns.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "pdl.cuh"

namespace dgbgk {
namespace umma {

constexpr int BM = 128;        // tile rows (MMA M)
constexpr int BK = 64;         // K-block: 64 BF16 = one 128-byte swizzle row
constexpr unsigned WAIT_TRIES = 1u << 22;

__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void bar_init(uint64_t* b, uint32_t n) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr(b)), "r"(n) : "memory");
}
__device__ __forceinline__ void bar_expect(uint64_t* b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(saddr(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_try(uint64_t* b, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(saddr(b)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool bar_wait(uint64_t* b, uint32_t parity) {
  for (unsigned i = 0; i < WAIT_TRIES; ++i) {
    if (bar_try(b, parity)) return true;
    if (i > 32) __nanosleep(128);
  }
  return false;
}
__device__ __forceinline__ void tma2d(void* dst, const CUtensorMap* m, int x, int y, uint64_t* b) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::
          "r"(saddr(dst)),
      "l"(m), "r"(x), "r"(y), "r"(saddr(b))
      : "memory");
}

// Shared-memory matrix descriptor of a K-major BF16 tile whose 128-byte rows
// were written by TMA with the 128-byte swizzle: 8-row atoms of 1024 bytes
// stacked along M/N (stride byte offset 1024), descriptor version 1,
// layout type 2 (128-byte swizzle).  The start address advances by 32 bytes
// per K = 16 step inside the atom.
__device__ __forceinline__ uint64_t sdesc(const void* tile, int kbytes) {
  const uint64_t a = (uint64_t)((saddr(tile) + kbytes) >> 4) & 0x3FFFull;
  const uint64_t lbo = 1ull;               // unused by swizzled K-major layouts
  const uint64_t sbo = (1024ull >> 4);     // 8 rows x 128 bytes
  return a | (lbo << 16) | (sbo << 32) | (1ull << 46) | (2ull << 61);
}

// Instruction descriptor, kind::f16: D in FP32 (bits 4-5 = 1), A and B in
// BF16 (bits 7-9 = 1, bits 10-12 = 1), both K-major (bits 15, 16 = 0),
// N >> 3 in bits 17-22, M >> 4 in bits 24-28.
__host__ __device__ constexpr uint32_t idesc_bf16(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* b) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(saddr(b))
               : "memory");
}
__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(dst_smem)), "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// 32 columns of the warp's 32 TMEM lanes: thread t gets lane 32w+t
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,"
      "%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// Epilogue modes
enum Epi : int {
  EPI_TANH = 0,    // Y = tanh(C + bias): Y (BF16, [M][N]) and Y^T (BF16, [N][M])
  EPI_LINEAR = 1,  // Y = C + bias: FP32 [M][N]
  EPI_DTANH = 2,   // G = C * (1 - y^2), y = aux (BF16 [M][N]): G (BF16 [M][N]) and G^T (BF16 [N][M])
  EPI_F32 = 3,     // C: FP32 [M][N]
  EPI_LOSS = 4,    // d = C + bias - t: G = scale*d (BF16 [M][N]) and G^T, the sum of d^2/(M N) added to *loss
  EPI_ADAM = 5,    // C is the gradient of the weights w [M][N]: an Adam step on them and their BF16 copies
};

struct GemmArgs {
  const float* bias;         // [N] (EPI_TANH, EPI_LINEAR, EPI_LOSS)
  const __nv_bfloat16* aux;  // [M][N] (EPI_DTANH)
  __nv_bfloat16* out_bf;     // [M][N]
  __nv_bfloat16* out_bfT;    // [N][M]
  float* out_f;              // [M][N]
  // EPI_LOSS: row r's targets are ts[idx[r]*N ..]
  const float* ts;
  const int* idx;
  double* loss;
  float scale;
  // EPI_ADAM (out_bf, out_bfT: the weights' copies): columns from `live` on stay as they are
  float *w, *m, *v;
  int live;
  float lr, b1, b2, eps, c1, c2;
  int* err;  // set when a bounded wait expired
  int M, N, K;
};

// One Adam update of a weight and its moments.  The fused multiply-adds are
// written out: left to the compiler, the two places that inline this could
// round the moments differently, and BF16 copies of weights a last bit apart
// send a training run its own way.
__device__ __forceinline__ float adam_step(float x, float& m, float& v, float g, const GemmArgs& a) {
  m = __fmaf_rn(1.f - a.b1, g, __fmul_rn(a.b1, m));
  v = __fmaf_rn((1.f - a.b2) * g, g, __fmul_rn(a.b2, v));
  return x - a.lr * (m / a.c1) / (sqrtf(v / a.c2) + a.eps);
}

// One thread of a converged warp.  The loops of the copying and of the
// issuing thread take this and not lane == 0: the tensor instructions' operands
// are uniform registers, and where the compiler cannot see that one thread is
// active it moves them there anew for each instruction (K-block of 64, tile of
// 128 x 32: 0.29 -> 0.19 us).
__device__ __forceinline__ bool elect_one() {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(r));
  return r != 0;
}

// A stage holds SUB K-blocks.
template <int BN, int STAGES, int SUB, int EPI>
struct Smem {
  static constexpr int A_BYTES = BM * BK * 2;  // 16 KB
  static constexpr int B_BYTES = BN * BK * 2;
  static constexpr int BLOCK = A_BYTES + B_BYTES;
  static constexpr int STAGE = SUB * BLOCK;
  // EPI_ADAM, in the ring's place once the accumulator is complete: the tile
  // in FP32 (pitch BN + 4 floats: 16-byte rows on shifted banks) and the new
  // weights transposed in BF16 (pitch BM + 2: neighbouring columns on
  // neighbouring banks)
  static constexpr int PF = BN + 4, PT = BM + 2;
  static constexpr int EPILOGUE = EPI == EPI_ADAM ? BM * PF * 4 + BN * PT * 2 : 0;
  static constexpr int RING = STAGES * STAGE;
  static constexpr int TOTAL = 1024 + (RING > EPILOGUE ? RING : EPILOGUE);  // + 1024 alignment slack
};

__device__ __forceinline__ uint32_t bf16x2(float a, float b) {
  const __nv_bfloat162 p = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&p);
}

// C tile (m0, n0) by the CTA's 128 threads.  M, N, K: multiples of 128, BN,
// 64*SUB.
template <int BN, int STAGES, int SUB, int EPI>
__device__ __forceinline__ void gemm_tile(const CUtensorMap& ta, const CUtensorMap& tb, const GemmArgs& g, int m0,
                                          int n0) {
  static_assert(BN % 32 == 0 && BN >= 32 && BN <= 256, "MMA N");
  using S = Smem<BN, STAGES, SUB, EPI>;
  extern __shared__ __align__(1024) unsigned char sm_raw[];
  __shared__ uint64_t full[STAGES], empty[STAGES], done;
  __shared__ uint32_t tmem_base;
  __shared__ int fail, issued, consumed;
  __shared__ double red[4];
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  unsigned char* base = sm_raw + ((1024u - (saddr(sm_raw) & 1023u)) & 1023u);
  const int nk = g.K / (BK * SUB);
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      bar_init(&full[s], 1);
      bar_init(&empty[s], 1);
    }
    bar_init(&done, 1);
    fail = 0;
    issued = 0;
    consumed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tmem_alloc(&tmem_base, BN);
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = tmem_base;
  // the tensor memory is held: a CTA of the next kernel that waits for some
  // waits for CTAs that need nothing more
  grid_launch_dependents();
  grid_wait();  // the operands, and the readers of what the epilogue writes

  if (warp == 0 && elect_one()) {
    // producer: stage s = kb % STAGES once the MMAs of kb - STAGES have
    // released it (ph: parity of the round over the ring)
    int s = 0;
    uint32_t ph = 0;
    for (int kb = 0; kb < nk; ++kb) {
      if (kb >= STAGES && !bar_wait(&empty[s], ph ^ 1u)) {
        fail = 1;
        break;
      }
      unsigned char* st = base + s * S::STAGE;
      bar_expect(&full[s], S::STAGE);
#pragma unroll
      for (int u = 0; u < SUB; ++u) {
        tma2d(st + u * S::BLOCK, &ta, (kb * SUB + u) * BK, m0, &full[s]);
        tma2d(st + u * S::BLOCK + S::A_BYTES, &tb, (kb * SUB + u) * BK, n0, &full[s]);
      }
      issued = kb + 1;
      if (++s == STAGES) {
        s = 0;
        ph ^= 1u;
      }
    }
  } else if (warp == 1 && elect_one()) {
    // MMA issuer; the descriptors' address fields (16-byte units) are advanced
    // by additions.  A K-block of 64 took 0.32 us whatever the tile's width and
    // the ring's depth, most of it this thread's; with both changes above and
    // two K-blocks a stage 0.145 us (128 x 32 tile, 141 GB/s into the SM).
    constexpr uint32_t idesc = idesc_bf16(BM, BN);
    const uint64_t ad0 = sdesc(base, 0), bd0 = sdesc(base + S::A_BYTES, 0);
    uint64_t off = 0;
    int s = 0;
    uint32_t ph = 0;
    for (int kb = 0; kb < nk; ++kb) {
      if (!bar_wait(&full[s], ph)) {
        fail = 1;
        break;
      }
      fence_after();
#pragma unroll
      for (int u = 0; u < SUB; ++u)
#pragma unroll
        for (int k = 0; k < BK / 16; ++k)
          mma_bf16(tmem, ad0 + off + u * (S::BLOCK >> 4) + 2 * k, bd0 + off + u * (S::BLOCK >> 4) + 2 * k, idesc,
                   (kb | u | k) ? 1u : 0u);
      mma_commit(&empty[s]);  // the stage is free once these MMAs have read it
      consumed = kb + 1;
      off += S::STAGE >> 4;
      if (++s == STAGES) {
        s = 0;
        off = 0;
        ph ^= 1u;
      }
    }
    mma_commit(&done);  // the accumulator is complete
  }
  __syncwarp();
  // every thread: wait for the accumulator
  const bool ok = bar_wait(&done, 0);
  fence_after();
  // the failing thread set `fail` before its own wait: the vote is uniform
  if (__syncthreads_or((!ok || fail) ? 1 : 0)) {
    if (tid == 0) {
      atomicExch(g.err, 1);
      // the box copies still in flight land before the CTA leaves (bounded)
      for (int kb = consumed; kb < issued; ++kb) bar_wait(&full[kb % STAGES], (kb / STAGES) & 1);
    }
  } else if constexpr (EPI == EPI_ADAM) {
    // the gradient tile to shared memory (rows of the accumulator are lanes),
    // then whole rows of the weights and moments, BN/4 lanes a row
    float* const sf = reinterpret_cast<float*>(base);
    __nv_bfloat16* const stp = reinterpret_cast<__nv_bfloat16*>(base + BM * S::PF * 4);
    {
      const int row = 32 * warp + lane;
      for (int c0 = 0; c0 < BN; c0 += 32) {
        float v[32];
        tmem_ld32(tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)c0, v);
#pragma unroll
        for (int i = 0; i < 32; i += 4)
          *reinterpret_cast<float4*>(sf + row * S::PF + c0 + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
      }
    }
    __syncwarp();  // a warp reads the rows it has written
    constexpr int LPR = BN / 4, RPI = 32 / LPR, UR = 4;  // lanes a row, rows an instruction, rows in flight / RPI
    static_assert(32 % LPR == 0 && 32 % (RPI * UR) == 0, "rows of a warp");
    const int cl = 4 * (lane % LPR), rl = lane / LPR;
    for (int r0 = 0; r0 < 32; r0 += RPI * UR) {
      float4 x[UR], mm[UR], vv[UR];
#pragma unroll
      for (int u = 0; u < UR; ++u) {
        const size_t o = (size_t)(m0 + 32 * warp + r0 + u * RPI + rl) * g.N + n0 + cl;
        x[u] = *reinterpret_cast<const float4*>(g.w + o);
        mm[u] = *reinterpret_cast<const float4*>(g.m + o);
        vv[u] = *reinterpret_cast<const float4*>(g.v + o);
      }
#pragma unroll
      for (int u = 0; u < UR; ++u) {
        const int row = 32 * warp + r0 + u * RPI + rl;
        const float4 gr = *reinterpret_cast<const float4*>(sf + row * S::PF + cl);
        if (n0 + cl + 3 < g.live) {
          x[u].x = adam_step(x[u].x, mm[u].x, vv[u].x, gr.x, g);
          x[u].y = adam_step(x[u].y, mm[u].y, vv[u].y, gr.y, g);
          x[u].z = adam_step(x[u].z, mm[u].z, vv[u].z, gr.z, g);
          x[u].w = adam_step(x[u].w, mm[u].w, vv[u].w, gr.w, g);
        } else {
          if (n0 + cl < g.live) x[u].x = adam_step(x[u].x, mm[u].x, vv[u].x, gr.x, g);
          if (n0 + cl + 1 < g.live) x[u].y = adam_step(x[u].y, mm[u].y, vv[u].y, gr.y, g);
          if (n0 + cl + 2 < g.live) x[u].z = adam_step(x[u].z, mm[u].z, vv[u].z, gr.z, g);
        }
        const size_t o = (size_t)(m0 + row) * g.N + n0 + cl;
        *reinterpret_cast<float4*>(g.w + o) = x[u];
        *reinterpret_cast<float4*>(g.m + o) = mm[u];
        *reinterpret_cast<float4*>(g.v + o) = vv[u];
        uint2 b;
        b.x = bf16x2(x[u].x, x[u].y);
        b.y = bf16x2(x[u].z, x[u].w);
        *reinterpret_cast<uint2*>(g.out_bf + o) = b;
        __nv_bfloat16* t = stp + cl * S::PT + row;
        t[0] = __float2bfloat16_rn(x[u].x);
        t[S::PT] = __float2bfloat16_rn(x[u].y);
        t[2 * S::PT] = __float2bfloat16_rn(x[u].z);
        t[3 * S::PT] = __float2bfloat16_rn(x[u].w);
      }
    }
    __syncthreads();
    // the transposed copy: a warp writes a column's 128 rows
    for (int c = warp; c < BN; c += 4) {
      const uint32_t* src = reinterpret_cast<const uint32_t*>(stp + c * S::PT);
      uint32_t* dst = reinterpret_cast<uint32_t*>(g.out_bfT + (size_t)(n0 + c) * g.M + m0);
      dst[lane] = src[lane];
      dst[lane + 32] = src[lane + 32];
    }
  } else {
    // epilogue: row m0 + 32*warp + lane, 32 columns at a time
    const int row = m0 + 32 * warp + lane;
    double sq = 0.0;
    const float* trow = EPI == EPI_LOSS ? g.ts + (size_t)g.idx[row] * g.N : nullptr;
    for (int c0 = 0; c0 < BN; c0 += 32) {
      float v[32];
      const int col = n0 + c0;
      float4 t4[8];
      if (EPI == EPI_LOSS) {
#pragma unroll
        for (int i = 0; i < 8; ++i) t4[i] = *reinterpret_cast<const float4*>(trow + col + 4 * i);
      }
      tmem_ld32(tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)c0, v);
      if (EPI == EPI_TANH || EPI == EPI_LINEAR || EPI == EPI_LOSS) {
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] += g.bias[col + i];
      }
      if (EPI == EPI_TANH) {
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = tanhf(v[i]);
      } else if (EPI == EPI_DTANH) {
        const uint4* y = reinterpret_cast<const uint4*>(g.aux + (size_t)row * g.N + col);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint4 q = y[i];
          const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float lo = __uint_as_float(w[k] << 16), hi = __uint_as_float(w[k] & 0xffff0000u);
            v[8 * i + 2 * k] *= 1.f - lo * lo;
            v[8 * i + 2 * k + 1] *= 1.f - hi * hi;
          }
        }
      } else if (EPI == EPI_LOSS) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float t[4] = {t4[i].x, t4[i].y, t4[i].z, t4[i].w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float d = v[4 * i + k] - t[k];
            sq += (double)d * d;
            v[4 * i + k] = g.scale * d;
          }
        }
      }
      if (EPI == EPI_TANH || EPI == EPI_DTANH || EPI == EPI_LOSS) {
        uint4* o = reinterpret_cast<uint4*>(g.out_bf + (size_t)row * g.N + col);
#pragma unroll
        for (int i = 0; i < 4; ++i)
          o[i] = make_uint4(bf16x2(v[8 * i], v[8 * i + 1]), bf16x2(v[8 * i + 2], v[8 * i + 3]),
                            bf16x2(v[8 * i + 4], v[8 * i + 5]), bf16x2(v[8 * i + 6], v[8 * i + 7]));
        // transposed copy: for a fixed column the 32 lanes write 32 consecutive rows
#pragma unroll
        for (int i = 0; i < 32; ++i) g.out_bfT[(size_t)(col + i) * g.M + row] = __float2bfloat16_rn(v[i]);
      } else {
        float* o = g.out_f + (size_t)row * g.N + col;
#pragma unroll
        for (int i = 0; i < 32; i += 4) *reinterpret_cast<float4*>(o + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
      }
    }
    if (EPI == EPI_LOSS) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
      if (lane == 0) red[warp] = sq;
      __syncthreads();
      if (tid == 0) atomicAdd(g.loss, (red[0] + red[1] + red[2] + red[3]) / ((double)g.M * (double)g.N));
    }
  }
  fence_before();
  __syncthreads();
  if (warp == 0) tmem_free(tmem, BN);
}

// one GEMM: tile (blockIdx.y, blockIdx.x)
template <int BN, int STAGES, int SUB, int EPI>
__global__ void __launch_bounds__(128, 1) k_gemm(const __grid_constant__ CUtensorMap ta,
                                                 const __grid_constant__ CUtensorMap tb,
                                                 const __grid_constant__ GemmArgs g) {
  gemm_tile<BN, STAGES, SUB, EPI>(ta, tb, g, blockIdx.y * BM, blockIdx.x * BN);
}

// The weight gradients of up to GROUP layers with their Adam steps in one
// launch, so that the few tiles of the hidden layers run beside the output
// layer's.
constexpr int GROUP = 8;
struct GroupArgs {
  CUtensorMap ta[GROUP], tb[GROUP];
  GemmArgs g[GROUP];
  int end[GROUP];  // running sum of the layers' tiles
  int n;
};
template <int BN, int STAGES, int SUB>
__global__ void __launch_bounds__(128, 4) k_gemm_adam(const __grid_constant__ GroupArgs a) {
  int l = 0;
  while ((int)blockIdx.x >= a.end[l]) ++l;
  const int t = blockIdx.x - (l ? a.end[l - 1] : 0), nt = a.g[l].N / BN;
  gemm_tile<BN, STAGES, SUB, EPI_ADAM>(a.ta[l], a.tb[l], a.g[l], t / nt * BM, t % nt * BN);
}

}  // namespace umma
}  // namespace dgbgk
