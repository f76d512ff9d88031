// The warm-start network: an MLP with tanh hidden layers trained and run
// with the BF16 tensor-core GEMM of umma.cuh (FP32 accumulation, FP32
// master weights, Adam).  Layers: n_in (padded to 64) -> width x depth ->
// n_out.  All GEMMs are C = A B^T with both operands K-major, so the network
// keeps W and W^T in BF16 and every activation and gradient in both
// layouts:
//   forward   H_{l+1} = tanh(H_l W_l^T + b_l)       A = H_l,   B = W_l
//   output    P = H_L W_L^T + b_L                    (FP32; a forward call)
//   loss      dP = 2 (P - T) / (B n_out)             (BF16, both layouts; the
//             output layer's epilogue in a training step, P is not stored)
//   dW_l      = dZ_{l+1}^T H_l                        A = dZ^T,  B = H_l^T
//             (a training step: Adam in its epilogue, the gradient is not
//             stored)
//   dZ_l      = (dZ_{l+1} W_l) (1 - H_l^2)            A = dZ,    B = W_l^T
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <random>
#include <string>
#include <vector>

#include "../../include/dgbgk.h"
#include "umma.cuh"

namespace dgbgk {
void set_error(const std::string& m);
}

using namespace dgbgk;
using namespace dgbgk::umma;

#define MCK(x)                                                                       \
  do {                                                                               \
    cudaError_t e_ = (x);                                                            \
    if (e_ != cudaSuccess) {                                                         \
      set_error(std::string("CUDA error: ") + cudaGetErrorString(e_) + " (" #x ")"); \
      return DGBGK_ECUDA;                                                            \
    }                                                                                \
  } while (0)
#define MTRY(x)               \
  do {                        \
    int rc_ = (x);            \
    if (rc_ != 0) return rc_; \
  } while (0)

namespace {

constexpr int KPAD = 64;  // the input layer's K (n_in padded)

PFN_cuTensorMapEncodeTiled_v12000 encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    cudaDriverEntryPointQueryResult q;
    void* p = nullptr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
  }
  return fn;
}

// [rows][cols] BF16 row-major as a TMA tensor; box = 64 columns x box_rows
// rows, 128-byte swizzle (the layout the GEMM's descriptors describe).
int bf16_map(CUtensorMap* m, const void* p, int rows, int cols, int box_rows) {
  auto enc = encoder();
  if (!enc) {
    set_error("cuTensorMapEncodeTiled is not available from the driver");
    return DGBGK_ECUDA;
  }
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
  cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
  cuuint32_t es[2] = {1, 1};
  CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(p), dims, strides, box, es,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed for an MLP operand");
    return DGBGK_ECUDA;
  }
  return 0;
}

// One planned GEMM: its operand maps, tile and epilogue.
struct Gemm {
  CUtensorMap ta, tb;
  GemmArgs g;
  int bn, epi;
};

// Tile widths: 32 columns where 64 would leave SMs without a tile (the hidden
// layers, and the output layer's dZ, whose K is n_out), 64 otherwise.  The
// narrow tile's ring takes most of an SM: its CTAs are few, and what they
// need is loads in flight.  dZ of 128 x 512 with K = 32768: 175 us with four
// CTAs of 128 x 128 tiles, 75 with 16 of 128 x 32.  Many tiles: the CTAs an SM
// holds count, two of 64 columns against one of 128 in the same stages.
// Prediction of 1024 x 32768 with K = 512: 106.6 us against 114.7, of 128 rows
// 24.6 against 26.6, of 2048 199 against 213.
constexpr int STAGES32 = 5, STAGES64 = 2, STAGES_ADAM = 2;

int plan_gemm(Gemm& G, const __nv_bfloat16* A, const __nv_bfloat16* B, int M, int N, int K, int epi, GemmArgs g,
              int nsm) {
  if (M % BM || N % 64 || (K % (2 * BK) && !(K == BK && epi == EPI_TANH))) {
    set_error("MLP GEMM shape not a multiple of the tile");
    return DGBGK_EINVAL;
  }
  G.epi = epi;
  G.bn = epi != EPI_ADAM && epi != EPI_F32 && (long)(M / BM) * (N / 64) < nsm ? 32 : 64;
  MTRY(bf16_map(&G.ta, A, M, K, BM));
  MTRY(bf16_map(&G.tb, B, N, K, G.bn));
  G.g = g;
  G.g.M = M;
  G.g.N = N;
  G.g.K = K;
  return 0;
}

template <int BN, int STAGES, int SUB, int EPI> int launch_gemm(const Gemm& G, const GemmArgs& g, cudaStream_t st) {
  auto fn = k_gemm<BN, STAGES, SUB, EPI>;
  constexpr int bytes = Smem<BN, STAGES, SUB, EPI>::TOTAL;
  MCK(cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  launch_pdl(fn, dim3(g.N / BN, g.M / BM), dim3(128), bytes, st, G.ta, G.tb, g);
  MCK(cudaGetLastError());
  return 0;
}
// two K-blocks of 64 a stage; the input layer's forward has one in all
template <int EPI> int launch_gemm(const Gemm& G, const GemmArgs& g, cudaStream_t st) {
  if (EPI == EPI_TANH && g.K == BK)
    return G.bn == 32 ? launch_gemm<32, 1, 1, EPI_TANH>(G, g, st) : launch_gemm<64, 1, 1, EPI_TANH>(G, g, st);
  return G.bn == 32 ? launch_gemm<32, STAGES32, 2, EPI>(G, g, st) : launch_gemm<64, STAGES64, 2, EPI>(G, g, st);
}
int run_gemm(const Gemm& G, const GemmArgs& g, cudaStream_t st) {
  switch (G.epi) {
    case EPI_TANH: return launch_gemm<EPI_TANH>(G, g, st);
    case EPI_LINEAR: return launch_gemm<EPI_LINEAR>(G, g, st);
    case EPI_DTANH: return launch_gemm<EPI_DTANH>(G, g, st);
    case EPI_LOSS: return launch_gemm<EPI_LOSS>(G, g, st);
    default: return launch_gemm<64, STAGES64, 2, EPI_F32>(G, g, st);
  }
}
int run_gemm(const Gemm& G, cudaStream_t st) { return run_gemm(G, G.g, st); }

// ----------------------------------------------------------- small kernels
// minibatch inputs: rows idx[r] of the set -> X0 (BF16, padded to KPAD, both
// layouts)
__global__ void k_gather(const float* __restrict__ xs, const int* __restrict__ idx, int n_in, int B,
                         __nv_bfloat16* x0, __nv_bfloat16* x0T) {
  const int r = blockIdx.x * blockDim.y + threadIdx.y, c = threadIdx.x;
  grid_launch_dependents();
  grid_wait();
  const __nv_bfloat16 v = __float2bfloat16_rn(c < n_in ? xs[(size_t)idx[r] * n_in + c] : 0.f);
  x0[(size_t)r * KPAD + c] = v;
  x0T[(size_t)c * B + r] = v;
}

// bias gradient: the sum over the batch of G[.., j], from G^T [N][B], by a warp
__device__ __forceinline__ float bias_grad(const __nv_bfloat16* __restrict__ row, int B, int lane) {
  float s = 0.f;
  for (int r = lane; r < B; r += 32) s += __bfloat162float(row[r]);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}
__global__ void k_bias_grad(const __nv_bfloat16* __restrict__ gT, int N, int B, float* db) {
  const int j = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (j >= N) return;
  const float s = bias_grad(gT + (size_t)j * B, B, lane);
  if (lane == 0) db[j] = s;
}
// the biases' gradients and Adam steps of up to BIAS_LAYERS layers
constexpr int BIAS_LAYERS = 8;
struct BiasArgs {
  const __nv_bfloat16* gT[BIAS_LAYERS];
  float *b[BIAS_LAYERS], *m[BIAS_LAYERS], *v[BIAS_LAYERS];
  int end[BIAS_LAYERS];  // running sum of the layers' widths
  int n, B;
};
__global__ void k_bias_adam(const __grid_constant__ BiasArgs a, const __grid_constant__ GemmArgs p) {
  int j = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  grid_launch_dependents();
  grid_wait();
  if (j >= a.end[a.n - 1]) return;
  int l = 0;
  while (j >= a.end[l]) ++l;
  if (l > 0) j -= a.end[l - 1];
  const float g = bias_grad(a.gT[l] + (size_t)j * a.B, a.B, lane);
  if (lane == 0) {
    float m = a.m[l][j], v = a.v[l][j];
    a.b[l][j] = adam_step(a.b[l][j], m, v, g, p);
    a.m[l][j] = m;
    a.v[l][j] = v;
  }
}

// FP32 -> BF16 copies of a weight matrix (both layouts)
__global__ void k_to_bf16(const float* __restrict__ w, int rows, int cols, __nv_bfloat16* wb, __nv_bfloat16* wbT) {
  const size_t n = (size_t)rows * cols;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int r = (int)(i / cols), c = (int)(i - (size_t)r * cols);
    const __nv_bfloat16 xb = __float2bfloat16_rn(w[i]);
    wb[i] = xb;
    wbT[(size_t)c * rows + r] = xb;
  }
}

// zeroed device allocation; the memset is complete on return, so work on
// any stream may use the buffer
template <class X> int mall(X** p, size_t n) {
  *p = nullptr;
  MCK(cudaMalloc((void**)p, std::max<size_t>(n, 1) * sizeof(X)));
  MCK(cudaMemset(*p, 0, std::max<size_t>(n, 1) * sizeof(X)));
  MCK(cudaDeviceSynchronize());
  return 0;
}
template <class X> void mfree(X*& p) {
  if (p) cudaFree((void*)p);
  p = nullptr;
}

// room for n values, the old ones freed first; none (cap 0) when the new
// allocation fails
template <class X> int room(X*& p, size_t& cap, size_t n) {
  if (n <= cap) return 0;
  cap = 0;
  mfree(p);
  MTRY(mall(&p, n));
  cap = n;
  return 0;
}

struct Layer {
  int in = 0, in_live = 0, out = 0;
  float *w = nullptr, *b = nullptr, *gw = nullptr, *gb = nullptr;
  float *mw = nullptr, *vw = nullptr, *mb = nullptr, *vb = nullptr;
  __nv_bfloat16 *wb = nullptr, *wbT = nullptr;
};

}  // namespace

struct dgbgk_mlp {
  int device = 0, nsm = 0, n_in = 0, width = 0, depth = 0, n_out = 0, B = 0;
  cudaStream_t st = nullptr;
  std::vector<Layer> L;                  // depth + 1 layers
  std::vector<__nv_bfloat16*> H, HT;     // activations 0..depth (0 = input), [B][in] and [in][B]
  std::vector<__nv_bfloat16*> G, GT;     // dZ of layers 1..depth, and dP (index depth+1)
  float* P = nullptr;
  double* loss = nullptr;                // one slot per training step (slot 0 otherwise)
  size_t loss_cap = 0;
  int* err = nullptr;
  float *xs = nullptr, *ts = nullptr;    // training set
  int nset = 0;
  int* idx = nullptr;
  size_t idx_cap = 0;
  float *xin = nullptr, *tin = nullptr;  // staging of one host batch
  int* iin = nullptr;
  long long adam_t = 0;
  std::vector<Gemm> fwd, bwd_dw, bwd_dx, adam_dw;
  Gemm out_loss;  // the output layer with the loss in its epilogue

  ~dgbgk_mlp() {
    cudaSetDevice(device);
    if (st) cudaStreamSynchronize(st);
    for (auto& l : L) {
      mfree(l.w), mfree(l.b), mfree(l.gw), mfree(l.gb), mfree(l.mw), mfree(l.vw), mfree(l.mb), mfree(l.vb);
      mfree(l.wb), mfree(l.wbT);
    }
    for (auto* p : H) mfree(p);
    for (auto* p : HT) mfree(p);
    for (auto* p : G) mfree(p);
    for (auto* p : GT) mfree(p);
    mfree(P), mfree(loss), mfree(err), mfree(xs), mfree(ts), mfree(idx);
    mfree(xin), mfree(tin), mfree(iin);
    if (st) cudaStreamDestroy(st);
  }

  int init(unsigned long long seed) {
    MCK(cudaSetDevice(device));
    MCK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    const int nl = depth + 1;
    L.resize(nl);
    std::mt19937_64 rng(seed);
    for (int l = 0; l < nl; ++l) {
      Layer& y = L[l];
      y.in = l == 0 ? KPAD : width;
      y.in_live = l == 0 ? n_in : width;
      y.out = l == depth ? n_out : width;
      const size_t nw = (size_t)y.out * y.in;
      MTRY(mall(&y.w, nw));
      MTRY(mall(&y.gw, nw));
      MTRY(mall(&y.mw, nw));
      MTRY(mall(&y.vw, nw));
      MTRY(mall(&y.b, y.out));
      MTRY(mall(&y.gb, y.out));
      MTRY(mall(&y.mb, y.out));
      MTRY(mall(&y.vb, y.out));
      MTRY(mall(&y.wb, nw));
      MTRY(mall(&y.wbT, nw));
      // Xavier-uniform weights, zero biases
      std::vector<float> hw(nw, 0.f);
      const float a = std::sqrt(6.f / (float)(y.in_live + y.out));
      std::uniform_real_distribution<float> U(-a, a);
      for (int r = 0; r < y.out; ++r)
        for (int c = 0; c < y.in_live; ++c) hw[(size_t)r * y.in + c] = U(rng);
      MCK(cudaMemcpyAsync(y.w, hw.data(), nw * 4, cudaMemcpyHostToDevice, st));
      MCK(cudaStreamSynchronize(st));
    }
    H.assign(nl, nullptr);
    HT.assign(nl, nullptr);
    for (int l = 0; l < nl; ++l) {
      const int c = L[l].in;
      MTRY(mall(&H[l], (size_t)B * c));
      MTRY(mall(&HT[l], (size_t)B * c));
    }
    G.assign(nl + 1, nullptr);
    GT.assign(nl + 1, nullptr);
    for (int l = 1; l <= nl; ++l) {
      const int c = l == nl ? n_out : width;
      MTRY(mall(&G[l], (size_t)B * c));
      MTRY(mall(&GT[l], (size_t)B * c));
    }
    MTRY(mall(&P, (size_t)B * n_out));
    MTRY(room(loss, loss_cap, 1));
    MTRY(mall(&err, 1));
    MTRY(mall(&xin, (size_t)B * n_in));
    MTRY(mall(&tin, (size_t)B * n_out));
    MTRY(mall(&iin, B));
    {
      std::vector<int> id(B);
      for (int r = 0; r < B; ++r) id[r] = r;
      MCK(cudaMemcpyAsync(iin, id.data(), B * sizeof(int), cudaMemcpyHostToDevice, st));
    }
    MTRY(refresh_bf16());
    return plan();
  }

  int refresh_bf16() {
    for (auto& y : L) {
      k_to_bf16<<<256, 256, 0, st>>>(y.w, y.out, y.in, y.wb, y.wbT);
      MCK(cudaGetLastError());
    }
    return 0;
  }

  int plan() {
    const int nl = depth + 1;
    fwd.assign(nl, Gemm{});
    bwd_dw.assign(nl, Gemm{});
    bwd_dx.assign(nl, Gemm{});
    adam_dw.assign(nl, Gemm{});
    for (int l = 0; l < nl; ++l) {
      Layer& y = L[l];
      GemmArgs g{};
      g.err = err;
      g.bias = y.b;
      if (l < depth) {
        g.out_bf = H[l + 1];
        g.out_bfT = HT[l + 1];
        MTRY(plan_gemm(fwd[l], H[l], y.wb, B, y.out, y.in, EPI_TANH, g, nsm));
      } else {
        g.out_f = P;
        MTRY(plan_gemm(fwd[l], H[l], y.wb, B, y.out, y.in, EPI_LINEAR, g, nsm));
        g.out_bf = G[nl];
        g.out_bfT = GT[nl];
        g.scale = 2.f / (float)((size_t)B * n_out);
        MTRY(plan_gemm(out_loss, H[l], y.wb, B, y.out, y.in, EPI_LOSS, g, nsm));
      }
      // dW_l = G_{l+1}^T H_l: [out][in], K = B
      GemmArgs gw{};
      gw.err = err;
      gw.out_f = y.gw;
      MTRY(plan_gemm(bwd_dw[l], GT[l + 1], HT[l], y.out, y.in, B, EPI_F32, gw, nsm));
      gw.w = y.w;
      gw.m = y.mw;
      gw.v = y.vw;
      gw.out_bf = y.wb;
      gw.out_bfT = y.wbT;
      gw.live = y.in_live;
      MTRY(plan_gemm(adam_dw[l], GT[l + 1], HT[l], y.out, y.in, B, EPI_ADAM, gw, nsm));
      // G_l = (G_{l+1} W_l) (1 - H_l^2): [B][in], K = out (not for the input layer)
      if (l > 0) {
        GemmArgs gx{};
        gx.err = err;
        gx.aux = H[l];
        gx.out_bf = G[l];
        gx.out_bfT = GT[l];
        MTRY(plan_gemm(bwd_dx[l], G[l + 1], y.wbT, B, y.in, y.out, EPI_DTANH, gx, nsm));
      }
    }
    return 0;
  }

  int forward() {
    for (int l = 0; l <= depth; ++l) MTRY(run_gemm(fwd[l], st));
    return 0;
  }

  // forward, and the loss (into *lslot) and its gradient at the output, of
  // the minibatch whose inputs are in H[0] and whose targets are rows id of t
  // (*lslot is zero before: a memset between two kernels would keep the second
  // from starting early)
  int forward_loss(const float* t, const int* id, double* lslot) {
    for (int l = 0; l < depth; ++l) MTRY(run_gemm(fwd[l], st));
    GemmArgs g = out_loss.g;
    g.ts = t;
    g.idx = id;
    g.loss = lslot;
    return run_gemm(out_loss, g, st);
  }

  // all gradients of the minibatch
  int backward() {
    for (int l = depth; l >= 0; --l) {
      MTRY(run_gemm(bwd_dw[l], st));
      k_bias_grad<<<(L[l].out + 7) / 8, 256, 0, st>>>(GT[l + 1], L[l].out, B, L[l].gb);
      MCK(cudaGetLastError());
      if (l > 0) MTRY(run_gemm(bwd_dx[l], st));
    }
    return 0;
  }

  // the same with an Adam step on every layer: every dZ, which needs the old
  // weights, before the weights' updates
  int backward_adam(float lr) {
    ++adam_t;
    GemmArgs p{};
    p.lr = lr;
    p.b1 = 0.9f;
    p.b2 = 0.999f;
    p.eps = 1e-8f;
    p.c1 = 1.f - std::pow(p.b1, (float)adam_t);
    p.c2 = 1.f - std::pow(p.b2, (float)adam_t);
    for (int l = depth; l > 0; --l) MTRY(run_gemm(bwd_dx[l], st));
    constexpr int bytes = Smem<64, STAGES_ADAM, 1, EPI_ADAM>::TOTAL;
    MCK(cudaFuncSetAttribute((const void*)k_gemm_adam<64, STAGES_ADAM, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             bytes));
    for (int l1 = depth; l1 >= 0; l1 -= GROUP) {
      GroupArgs a{};
      int tiles = 0;
      for (int l = l1; l >= 0 && l > l1 - GROUP; --l, ++a.n) {
        a.ta[a.n] = adam_dw[l].ta;
        a.tb[a.n] = adam_dw[l].tb;
        GemmArgs& g = a.g[a.n] = adam_dw[l].g;
        g.lr = p.lr;
        g.b1 = p.b1;
        g.b2 = p.b2;
        g.eps = p.eps;
        g.c1 = p.c1;
        g.c2 = p.c2;
        a.end[a.n] = tiles += (g.M / BM) * (g.N / 64);
      }
      launch_pdl(k_gemm_adam<64, STAGES_ADAM, 1>, dim3(tiles), dim3(128), bytes, st, a);
      MCK(cudaGetLastError());
    }
    for (int l0 = 0; l0 <= depth; l0 += BIAS_LAYERS) {
      BiasArgs a{};
      a.B = B;
      int rows = 0;
      for (int l = l0; l <= depth && l < l0 + BIAS_LAYERS; ++l, ++a.n) {
        a.gT[a.n] = GT[l + 1];
        a.b[a.n] = L[l].b;
        a.m[a.n] = L[l].mb;
        a.v[a.n] = L[l].vb;
        a.end[a.n] = rows += L[l].out;
      }
      launch_pdl(k_bias_adam, dim3((rows + 7) / 8), dim3(256), 0, st, a, p);
      MCK(cudaGetLastError());
    }
    return 0;
  }

  int gather(const float* x, const int* id) {
    launch_pdl(k_gather, dim3(B / 4), dim3(KPAD, 4), 0, st, x, id, n_in, B, H[0], HT[0]);
    MCK(cudaGetLastError());
    return 0;
  }

  int check_err() {
    int e = 0;
    MCK(cudaMemcpyAsync(&e, err, sizeof(int), cudaMemcpyDeviceToHost, st));
    MCK(cudaStreamSynchronize(st));
    if (e) {
      set_error("MLP GEMM: a bounded device wait expired");
      return DGBGK_ECUDA;
    }
    return 0;
  }

  // n <= B host rows x[n][n_in] (and t[n][n_out]) -> the minibatch
  // buffers; rows past n repeat nothing meaningful (their inputs are zero
  // and their outputs are not read back)
  int load_batch_host(const float* x, const float* t, int n) {
    if (n < B) MCK(cudaMemsetAsync(xin, 0, (size_t)B * n_in * 4, st));
    MCK(cudaMemcpyAsync(xin, x, (size_t)n * n_in * 4, cudaMemcpyHostToDevice, st));
    if (t) MCK(cudaMemcpyAsync(tin, t, (size_t)n * n_out * 4, cudaMemcpyHostToDevice, st));
    return gather(xin, iin);
  }
};

extern "C" {

int dgbgk_mlp_create(int n_in, int width, int depth, int n_out, int batch, unsigned long long seed, int device,
                     dgbgk_mlp** out) {
  if (!out || n_in < 1 || n_in > KPAD || width < 128 || width % 128 || depth < 1 || n_out < 128 || n_out % 128 ||
      batch < 128 || batch % 128) {
    set_error("dgbgk_mlp_create: n_in <= 64, width/n_out/batch multiples of 128, depth >= 1");
    return DGBGK_EINVAL;
  }
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) {
    set_error("dgbgk_mlp_create: no such CUDA device");
    return DGBGK_ECUDA;
  }
  cudaDeviceProp prop;
  MCK(cudaGetDeviceProperties(&prop, device));
  if (prop.major != 10) {
    set_error("dgbgk_mlp_create: this build targets sm_100a (B200)");
    return DGBGK_ECUDA;
  }
  std::unique_ptr<dgbgk_mlp> m(new dgbgk_mlp());
  m->device = device;
  m->nsm = prop.multiProcessorCount;
  m->n_in = n_in;
  m->width = width;
  m->depth = depth;
  m->n_out = n_out;
  m->B = batch;
  MTRY(m->init(seed));
  *out = m.release();
  return DGBGK_OK;
}

long long dgbgk_mlp_param_count(const dgbgk_mlp* m) {
  if (!m) return -1;
  long long n = 0;
  for (const auto& y : m->L) n += (long long)y.out * y.in + y.out;
  return n;
}

// flat layout per layer: W [out][in] (input layer in = 64, columns past
// n_in zero), then b [out]
int dgbgk_mlp_get_params(dgbgk_mlp* m, float* p) {
  if (!m || !p) return set_error("NULL argument"), DGBGK_EINVAL;
  MCK(cudaSetDevice(m->device));
  MCK(cudaStreamSynchronize(m->st));
  size_t o = 0;
  for (const auto& y : m->L) {
    const size_t nw = (size_t)y.out * y.in;
    MCK(cudaMemcpyAsync(p + o, y.w, nw * 4, cudaMemcpyDeviceToHost, m->st));
    o += nw;
    MCK(cudaMemcpyAsync(p + o, y.b, y.out * 4, cudaMemcpyDeviceToHost, m->st));
    o += y.out;
  }
  MCK(cudaStreamSynchronize(m->st));
  return 0;
}

int dgbgk_mlp_set_params(dgbgk_mlp* m, const float* p) {
  if (!m || !p) return set_error("NULL argument"), DGBGK_EINVAL;
  MCK(cudaSetDevice(m->device));
  size_t o = 0;
  for (auto& y : m->L) {
    const size_t nw = (size_t)y.out * y.in;
    MCK(cudaMemcpyAsync(y.w, p + o, nw * 4, cudaMemcpyHostToDevice, m->st));
    o += nw;
    MCK(cudaMemcpyAsync(y.b, p + o, y.out * 4, cudaMemcpyHostToDevice, m->st));
    o += y.out;
  }
  MTRY(m->refresh_bf16());
  MCK(cudaStreamSynchronize(m->st));
  return 0;
}

// y[n][n_out] = network(x[n][n_in]); n rows in chunks of the batch size
int dgbgk_mlp_forward(dgbgk_mlp* m, const float* x, int n, float* y) {
  if (!m || !x || !y || n < 1) return set_error("NULL argument"), DGBGK_EINVAL;
  MCK(cudaSetDevice(m->device));
  for (int r0 = 0; r0 < n; r0 += m->B) {
    const int k = std::min(m->B, n - r0);
    MTRY(m->load_batch_host(x + (size_t)r0 * m->n_in, nullptr, k));
    MTRY(m->forward());
    MCK(cudaMemcpyAsync(y + (size_t)r0 * m->n_out, m->P, (size_t)k * m->n_out * 4, cudaMemcpyDeviceToHost, m->st));
    MCK(cudaStreamSynchronize(m->st));
    MTRY(m->check_err());
  }
  return 0;
}

// loss (mean squared error) and the gradient (flat, as the parameters) of
// one batch of exactly `batch` rows
int dgbgk_mlp_gradient(dgbgk_mlp* m, const float* x, const float* t, int n, double* loss, float* grad) {
  if (!m || !x || !t || n != m->B) return set_error("dgbgk_mlp_gradient: n must equal the batch size"), DGBGK_EINVAL;
  MCK(cudaSetDevice(m->device));
  MTRY(m->load_batch_host(x, t, n));
  MTRY(room(m->loss, m->loss_cap, 1));
  MCK(cudaMemsetAsync(m->loss, 0, sizeof(double), m->st));
  MTRY(m->forward_loss(m->tin, m->iin, m->loss));
  MTRY(m->backward());
  MTRY(m->check_err());
  if (loss) MCK(cudaMemcpyAsync(loss, m->loss, sizeof(double), cudaMemcpyDeviceToHost, m->st));
  if (grad) {
    size_t o = 0;
    for (const auto& y : m->L) {
      const size_t nw = (size_t)y.out * y.in;
      MCK(cudaMemcpyAsync(grad + o, y.gw, nw * 4, cudaMemcpyDeviceToHost, m->st));
      o += nw;
      MCK(cudaMemcpyAsync(grad + o, y.gb, y.out * 4, cudaMemcpyDeviceToHost, m->st));
      o += y.out;
    }
  }
  MCK(cudaStreamSynchronize(m->st));
  return 0;
}

// the training set: x[n][n_in], t[n][n_out] (host), kept on the device
int dgbgk_mlp_set_data(dgbgk_mlp* m, const float* x, const float* t, int n) {
  if (!m || !x || !t || n < 1) return set_error("NULL argument"), DGBGK_EINVAL;
  MCK(cudaSetDevice(m->device));
  MCK(cudaStreamSynchronize(m->st));
  mfree(m->xs);
  mfree(m->ts);
  m->nset = 0;
  MTRY(mall(&m->xs, (size_t)n * m->n_in));
  MTRY(mall(&m->ts, (size_t)n * m->n_out));
  MCK(cudaMemcpyAsync(m->xs, x, (size_t)n * m->n_in * 4, cudaMemcpyHostToDevice, m->st));
  MCK(cudaMemcpyAsync(m->ts, t, (size_t)n * m->n_out * 4, cudaMemcpyHostToDevice, m->st));
  MCK(cudaStreamSynchronize(m->st));
  m->nset = n;
  return 0;
}

// `iters` Adam steps on minibatches drawn without replacement per epoch
// (std::mt19937_64 seeded with `seed`); loss_hist[iters] (may be NULL)
// receives each step's minibatch loss.
int dgbgk_mlp_train(dgbgk_mlp* m, int iters, float lr, unsigned long long seed, double* loss_hist) {
  if (!m || iters < 0 || m->nset < 1) return set_error("dgbgk_mlp_train: no training set"), DGBGK_EINVAL;
  MCK(cudaSetDevice(m->device));
  const int B = m->B;
  if (iters == 0) return 0;
  MCK(cudaStreamSynchronize(m->st));
  MTRY(room(m->idx, m->idx_cap, (size_t)iters * B));
  MTRY(room(m->loss, m->loss_cap, (size_t)iters));
  std::vector<int> id((size_t)iters * B);
  std::mt19937_64 rng(seed);
  std::vector<int> perm(m->nset);
  for (int i = 0; i < m->nset; ++i) perm[i] = i;
  size_t pos = perm.size();
  for (size_t k = 0; k < id.size(); ++k) {
    if (pos == perm.size()) {
      std::shuffle(perm.begin(), perm.end(), rng);
      pos = 0;
    }
    id[k] = perm[pos++];
  }
  MCK(cudaMemcpyAsync(m->idx, id.data(), id.size() * sizeof(int), cudaMemcpyHostToDevice, m->st));
  MCK(cudaMemsetAsync(m->loss, 0, iters * sizeof(double), m->st));
  for (int it = 0; it < iters; ++it) {
    const int* id = m->idx + (size_t)it * B;
    MTRY(m->gather(m->xs, id));
    MTRY(m->forward_loss(m->ts, id, m->loss + it));
    MTRY(m->backward_adam(lr));
  }
  MTRY(m->check_err());
  if (loss_hist) {
    MCK(cudaMemcpyAsync(loss_hist, m->loss, iters * sizeof(double), cudaMemcpyDeviceToHost, m->st));
    MCK(cudaStreamSynchronize(m->st));
  }
  return 0;
}

void dgbgk_mlp_destroy(dgbgk_mlp* m) { delete m; }

}  // extern "C"
