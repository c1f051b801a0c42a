// Warm-start network: an MLP (Fourier features of the cell centre (x, y)
// plus (m, p, t, Mach, AoA) -> 4 hidden layers of 256 SiLU units -> 8
// outputs: the 4 conserved variables and the 4 adjoint components, both
// normalised by the caller), trained and run on the GPU by this file's own
// kernels.  Every matrix product is the tcgen05 GEMM of mlp_gemm.cuh (BF16
// weights and activations, FP32 accumulation); biases, Adam moments and
// master weights are FP32.
#include <cmath>
#include <cstring>
#include <random>
#include <string>
#include <vector>

#include "mlp.hpp"
#include "mlp_gemm.cuh"

namespace o2f {
namespace mlp {

// Layers as k_adam sees them: where a layer's weights start, end, and go.
struct Layers {
  int64_t w_off[5], w_end[5];
  int cols[5], rows[5];
  bf16 *W[5], *WT[5];
};

namespace {

constexpr int kIn = 7;         // x, y, m, p, t, Mach, AoA
constexpr int kFreq = 32;      // Fourier frequencies of (x, y)
constexpr int kFeat = 128;     // 2*kFreq sin/cos + kIn raw inputs, zero padded
constexpr int kWidth = 256;
constexpr int kHidden = 4;     // Layers holds kHidden + 1
constexpr int kOut = 8;
constexpr int kOutPad = 16;    // the output layer's GEMM tile width

int in_dim(int l) { return l == 0 ? kFeat : kWidth; }
int out_dim(int l) { return l == kHidden ? kOutPad : kWidth; }

// What a training step reads besides the data: Adam's bias corrections, the
// step's number (place of its loss), the rows of its batch.
struct StepHead {
  float c1, c2;
  int step, pad;
};

// 32 threads per row: one frequency each, and the raw inputs and the padding.
__global__ void k_features(int n, const float* __restrict__ inputs, const int* __restrict__ index,
                           const float* __restrict__ freq, bf16* __restrict__ X) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int i = (int)(t >> 5), f = (int)(t & 31);
  if (i >= n) return;
  const float* in = inputs + (int64_t)(index ? index[i] : i) * kIn;
  bf16* x = X + (int64_t)i * kFeat;
  const float px = in[0], py = in[1];
  const float arg = 6.283185307179586f * (freq[2 * f] * px + freq[2 * f + 1] * py);
  x[f] = __float2bfloat16_rn(sinf(arg));
  x[kFreq + f] = __float2bfloat16_rn(cosf(arg));
  x[2 * kFreq + f] = __float2bfloat16_rn(f < kIn ? in[f] : 0.f);
  x[3 * kFreq + f] = __float2bfloat16_rn(0.f);
}
static_assert(kFreq == 32 && kFeat == 4 * kFreq, "k_features' thread layout");

// Mean squared error over the 8 outputs; dY = d(loss)/dY (bf16, padded
// columns zero); loss accumulated into *loss.
__global__ void k_loss(int n, const float* __restrict__ Y, const float* __restrict__ targets,
                       const int* __restrict__ index, bf16* __restrict__ dY, float* loss,
                       const StepHead* head) {
  if (head) loss += head->step;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  float l = 0.f;
  if (i < n) {
    const float* t = targets + (int64_t)(index ? index[i] : i) * kOut;
    const float scale = 2.f / ((float)n * kOut);
    for (int j = 0; j < kOutPad; ++j) {
      float g = 0.f;
      if (j < kOut) {
        const float d = Y[(int64_t)i * kOutPad + j] - t[j];
        l += d * d;
        g = scale * d;
      }
      dY[(int64_t)i * kOutPad + j] = __float2bfloat16_rn(g);
    }
  }
  for (int o = 16; o > 0; o >>= 1) l += __shfl_down_sync(0xffffffffu, l, o);
  if ((threadIdx.x & 31) == 0 && loss) atomicAdd(loss, l / ((float)n * kOut));
}

// Adam on the FP32 master parameters, and the BF16 copies of the weights in
// both orientations (W: [out][in] for the forward GEMM, WT: [in][out] for the
// input gradients).
__global__ void k_adam(int64_t n, float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, float lr, float b1, float b2, float eps, const StepHead* head,
                       Layers ly) {
  const float c1 = head->c1, c2 = head->c2;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    w[i] = wi;
#pragma unroll
    for (int l = 0; l <= kHidden; ++l)
      if (i >= ly.w_off[l] && i < ly.w_end[l]) {
        const int j = (int)(i - ly.w_off[l]), r = j / ly.cols[l], c = j - r * ly.cols[l];
        const bf16 b = __float2bfloat16_rn(wi);
        ly.W[l][j] = b;
        ly.WT[l][(int64_t)c * ly.rows[l] + r] = b;
      }
  }
}

__global__ void k_pack(int rows, int cols, const float* __restrict__ w, bf16* __restrict__ W, bf16* __restrict__ WT) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (int64_t)rows * cols) return;
  const int r = (int)(i / cols), c = (int)(i % cols);
  const bf16 b = __float2bfloat16_rn(w[i]);
  W[i] = b;
  WT[(int64_t)c * rows + r] = b;
}

int blocks_of(int64_t n, int b) { return (int)((n + b - 1) / b); }

}  // namespace

Mlp::Mlp(int max_batch, float freq_scale, uint64_t seed, cudaStream_t stream)
    : max_batch_(max_batch), stream_(stream) {
  if (max_batch < 128 || max_batch > (1 << 20)) throw Error(O2F_ERR_ARG, "max_batch out of range [128, 2^20]");
  if (!(freq_scale > 0.f)) throw Error(O2F_ERR_ARG, "freq_scale must be positive");
  O2F_CUDA(cudaFuncSetAttribute(k_gemm_tc<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, gemm_smem_bytes<64>()));
  O2F_CUDA(cudaFuncSetAttribute(k_gemm_tc<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, gemm_smem_bytes<16>()));
  O2F_CUDA(cudaFuncSetAttribute(k_weight_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, kGradSmem));
  // parameter layout: W0, b0, W1, b1, ..., W4, b4
  int64_t off = 0;
  for (int l = 0; l <= kHidden; ++l) {
    w_off_[l] = off;
    off += (int64_t)out_dim(l) * in_dim(l);
    b_off_[l] = off;
    off += out_dim(l);
  }
  n_params_ = off;
  std::mt19937_64 rng(seed);
  std::normal_distribution<float> nd(0.f, 1.f);
  std::vector<float> p(n_params_, 0.f);
  for (int l = 0; l <= kHidden; ++l) {
    const float s = std::sqrt(2.f / (float)in_dim(l)) * (l == kHidden ? 0.1f : 1.f);
    const int rows = l == kHidden ? kOut : out_dim(l);  // padded output rows stay zero
    for (int64_t i = 0; i < (int64_t)rows * in_dim(l); ++i) p[w_off_[l] + i] = s * nd(rng);
  }
  std::vector<float> fr(2 * kFreq);
  for (auto& f : fr) f = freq_scale * nd(rng);
  params_ = arena_.alloc<float>(n_params_);
  grads_ = arena_.alloc<float>(n_params_);
  adam_m_ = arena_.alloc<float>(n_params_);
  adam_v_ = arena_.alloc<float>(n_params_);
  freq_ = arena_.alloc<float>(2 * kFreq);
  for (int l = 0; l <= kHidden; ++l) {
    const int64_t n = (int64_t)out_dim(l) * in_dim(l);
    Wb_[l] = arena_.alloc<bf16>(n);
    WTb_[l] = arena_.alloc<bf16>(n);
  }
  // activations, pre-activations and their gradients of every layer: one block
  bf16* act = arena_.alloc<bf16>((int64_t)max_batch * (kFeat + 3 * kHidden * kWidth));
  X0_ = act;
  act += (int64_t)max_batch * kFeat;
  for (auto* group : {Z_, A_, dZ_})
    for (int l = 0; l < kHidden; ++l, act += (int64_t)max_batch * kWidth) group[l] = act;
  Y_ = arena_.alloc<float>((int64_t)max_batch * kOutPad);
  dY_ = arena_.alloc<bf16>((int64_t)max_batch * kOutPad);
  static_assert(sizeof(StepHead) % sizeof(int) == 0, "head and indices in one buffer");
  step_in_ = arena_.alloc<int>(sizeof(StepHead) / sizeof(int) + max_batch);
  loss_ = arena_.alloc<float>(1);
  err_ = arena_.alloc<int>(1);
  O2F_CUDA(cudaMemcpyAsync(params_, p.data(), n_params_ * sizeof(float), cudaMemcpyHostToDevice, stream_));
  O2F_CUDA(cudaMemcpyAsync(freq_, fr.data(), fr.size() * sizeof(float), cudaMemcpyHostToDevice, stream_));
  O2F_CUDA(cudaMemsetAsync(adam_m_, 0, n_params_ * sizeof(float), stream_));
  O2F_CUDA(cudaMemsetAsync(adam_v_, 0, n_params_ * sizeof(float), stream_));
  O2F_CUDA(cudaMemsetAsync(err_, 0, sizeof(int), stream_));
  pack();
  sync();
}

void Mlp::sync() {
  O2F_CUDA(cudaStreamSynchronize(stream_));
  int e = 0;
  O2F_CUDA(cudaMemcpy(&e, err_, sizeof(int), cudaMemcpyDeviceToHost));
  if (e) {
    O2F_CUDA(cudaMemset(err_, 0, sizeof(int)));
    throw Error(O2F_ERR_CUDA, "tensor-core GEMM: an mbarrier wait exceeded its limit");
  }
}

void Mlp::pack() {
  for (int l = 0; l <= kHidden; ++l) {
    const int64_t n = (int64_t)out_dim(l) * in_dim(l);
    k_pack<<<blocks_of(n, 256), 256, 0, stream_>>>(out_dim(l), in_dim(l), params_ + w_off_[l], Wb_[l], WTb_[l]);
  }
  O2F_CUDA(cudaGetLastError());
}

Mlp::~Mlp() {
  // the destructor's frees wait for the device
  if (graph_) cudaGraphExecDestroy(graph_);
  for (auto& e : slot_free_)
    if (e) cudaEventDestroy(e);
  for (auto& e : fork_)
    if (e) cudaEventDestroy(e);
  for (auto& e : join_)
    if (e) cudaEventDestroy(e);
  for (auto& c : capture_)
    if (c) cudaStreamDestroy(c);
  if (slots_) {
    cudaStreamSynchronize(stream_);
    cudaFreeHost(slots_);
  }
}

GemmArgs Mlp::args() const {
  GemmArgs a{};
  a.err = err_;
  return a;
}

// Forward pass of n feature rows (X0_ filled): Z_/A_ per hidden layer, the
// first `outputs` columns of the last layer into y (row stride `outputs`).
void Mlp::forward(int n, float* y, int outputs, cudaStream_t s) {
  const bf16* x = X0_;
  for (int l = 0; l <= kHidden; ++l) {
    GemmArgs a = args();
    a.M = n;
    a.K = in_dim(l);
    a.A = x;
    a.lda = in_dim(l);
    a.B = Wb_[l];
    a.ldb = in_dim(l);
    a.bias = params_ + b_off_[l];
    if (l < kHidden) {
      a.N = out_dim(l);
      a.epi = kEpiHidden;
      a.out = A_[l];
      a.pre = Z_[l];
      a.ldo = kWidth;
      k_gemm_tc<64><<<dim3(blocks_of(n, kTileM), blocks_of(a.N, 64)), gemm_threads(64), gemm_smem_bytes<64>(), s>>>(a);
      x = A_[l];
    } else {
      a.N = outputs;
      a.epi = kEpiLinear;
      a.out32 = y;
      a.ldo = outputs;
      k_gemm_tc<16><<<dim3(blocks_of(n, kTileM), 1), gemm_threads(16), gemm_smem_bytes<16>(), s>>>(a);
    }
    ++launches_;
  }
  O2F_CUDA(cudaGetLastError());
}

// Backward pass from dY_ into grads_ (zero on entry).  The chain of input
// gradients runs on s; a layer's weight and bias gradients, which nothing in
// the chain needs, on side[l] (null: on s too).
void Mlp::backward(int n, cudaStream_t s, const cudaStream_t* side) {
  const bf16* g = dY_;  // gradient w.r.t. the output of layer l
  for (int l = kHidden; l >= 0; --l) {
    const int N = out_dim(l), K = in_dim(l);
    const cudaStream_t sl = side ? side[l] : s;
    if (side) {
      O2F_CUDA(cudaEventRecord(fork_[l], s));
      O2F_CUDA(cudaStreamWaitEvent(sl, fork_[l], 0));
    }
    // dW_l[n][k] = sum_m g(m, n) below(m, k), db_l[n] = sum_m g(m, n): the
    // batch is the reduction axis
    GemmArgs w = args();
    w.M = N;
    w.N = K;
    w.K = n;
    w.A = g;
    w.lda = N;
    w.B = l > 0 ? A_[l - 1] : X0_;
    w.ldb = K;
    w.out32 = grads_ + w_off_[l];
    w.bias_grad = grads_ + b_off_[l];
    w.ldo = K;
    w.k_split = weight_grad_split(n);
    k_weight_grad<<<dim3(blocks_of(N, kTileM), K / kGradN + kBiasBlocks, blocks_of(n, w.k_split)), kGradThreads,
                    kGradSmem, sl>>>(w);
    if (side) O2F_CUDA(cudaEventRecord(join_[l], sl));
    ++launches_;
    if (l == 0) break;
    // gradient w.r.t. the layer below's pre-activation: (g W_l) * silu'(Z_{l-1})
    GemmArgs d = args();
    d.M = n;
    d.N = K;
    d.K = N;
    d.A = g;
    d.lda = N;
    d.B = WTb_[l];
    d.ldb = N;
    d.epi = kEpiBackAct;
    d.out = dZ_[l - 1];  // one per layer: its weight gradient may still be reading it
    d.zprev = Z_[l - 1];
    d.ldo = kWidth;
    k_gemm_tc<64>
        <<<dim3(blocks_of(n, kTileM), blocks_of(K, 64)), gemm_threads(64), gemm_smem_bytes<64>(), s>>>(d);
    ++launches_;
    g = dZ_[l - 1];
  }
  if (side)
    for (auto& e : join_) O2F_CUDA(cudaStreamWaitEvent(s, e, 0));
  O2F_CUDA(cudaGetLastError());
}

void Mlp::load_batch(const float* inputs_dev, const int* index_dev, int n, cudaStream_t s) {
  k_features<<<blocks_of((int64_t)n * 32, 128), 128, 0, s>>>(n, inputs_dev, index_dev, freq_, X0_);
  O2F_CUDA(cudaGetLastError());
  ++launches_;
}

void Mlp::set_data(const float* inputs, const float* targets, int64_t n) {
  if (n <= 0) throw Error(O2F_ERR_ARG, "empty data set");
  if (n > data_cap_) {  // device buffers grow only: repeated calls reuse them
    data_in_ = arena_.alloc<float>(n * kIn);
    data_out_ = arena_.alloc<float>(n * kOut);
    data_cap_ = n;
  }
  n_data_ = n;
  O2F_CUDA(cudaMemcpyAsync(data_in_, inputs, n * kIn * sizeof(float), cudaMemcpyHostToDevice, stream_));
  O2F_CUDA(cudaMemcpyAsync(data_out_, targets, n * kOut * sizeof(float), cudaMemcpyHostToDevice, stream_));
  sync();
}

void Mlp::train(int steps, int batch, float lr, uint64_t seed, float* loss_hist) {
  if (!n_data_) throw Error(O2F_ERR_STATE, "no training data (o2f_mlp_set_data)");
  if (steps <= 0 || batch < 1 || batch > max_batch_) throw Error(O2F_ERR_ARG, "steps or batch out of range");
  if (!(lr > 0.f)) throw Error(O2F_ERR_ARG, "lr must be positive");
  std::mt19937_64 rng(seed);
  std::uniform_int_distribution<int64_t> pick(0, n_data_ - 1);
  if (steps > loss_cap_) {
    loss_buf_ = arena_.alloc<float>(steps);
    loss_cap_ = steps;
  }
  O2F_CUDA(cudaMemsetAsync(loss_buf_, 0, steps * sizeof(float), stream_));
  const size_t slot_ints = sizeof(StepHead) / sizeof(int) + (size_t)max_batch_;
  if (!slots_) {
    O2F_CUDA(cudaMallocHost(&slots_, kSlots * slot_ints * sizeof(int)));
    for (auto& e : slot_free_) O2F_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    for (auto& e : fork_) O2F_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    for (auto& e : join_) O2F_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    for (auto& c : capture_) O2F_CUDA(cudaStreamCreateWithFlags(&c, cudaStreamNonBlocking));
  }
  build_graph(batch, lr);
  // The host draws the batches some steps ahead of the device: pinned slots,
  // each free again once its copy has been made.
  for (int s = 0; s < steps; ++s) {
    int* slot = slots_ + (size_t)(s % kSlots) * slot_ints;
    if (s >= kSlots) O2F_CUDA(cudaEventSynchronize(slot_free_[s % kSlots]));
    ++adam_t_;
    const float b1 = 0.9f, b2 = 0.999f;
    StepHead head{1.f - std::pow(b1, (float)adam_t_), 1.f - std::pow(b2, (float)adam_t_), s, 0};
    std::memcpy(slot, &head, sizeof(head));
    int* idx = slot + sizeof(StepHead) / sizeof(int);
    for (int i = 0; i < batch; ++i) idx[i] = (int)pick(rng);
    O2F_CUDA(cudaMemcpyAsync(step_in_, slot, sizeof(StepHead) + sizeof(int) * batch, cudaMemcpyHostToDevice, stream_));
    O2F_CUDA(cudaEventRecord(slot_free_[s % kSlots], stream_));
    O2F_CUDA(cudaGraphLaunch(graph_, stream_));
    launches_ += graph_launches_;
  }
  sync();
  if (loss_hist) O2F_CUDA(cudaMemcpy(loss_hist, loss_buf_, steps * sizeof(float), cudaMemcpyDeviceToHost));
}

// One training step as a graph: its batch, rates and loss place come from
// step_in_.  Captured on streams of its own (the caller's may be one that
// cannot be captured) and launched on the caller's.
void Mlp::build_graph(int batch, float lr) {
  if (graph_ && graph_batch_ == batch && graph_lr_ == lr && graph_data_ == data_in_ && graph_loss_ == loss_buf_) return;
  if (graph_) {
    O2F_CUDA(cudaGraphExecDestroy(graph_));
    graph_ = nullptr;
  }
  cudaStream_t s = capture_[0];
  const cudaStream_t* side = capture_ + 1;  // one per layer
  const StepHead* head = reinterpret_cast<const StepHead*>(step_in_);
  const int* index = step_in_ + sizeof(StepHead) / sizeof(int);
  const int64_t before = launches_;
  cudaGraph_t graph = nullptr;
  O2F_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
  try {
    O2F_CUDA(cudaEventRecord(fork_[0], s));  // the gradients are zeroed beside the forward pass
    O2F_CUDA(cudaStreamWaitEvent(side[0], fork_[0], 0));
    O2F_CUDA(cudaMemsetAsync(grads_, 0, n_params_ * sizeof(float), side[0]));
    O2F_CUDA(cudaEventRecord(join_[0], side[0]));
    load_batch(data_in_, index, batch, s);
    forward(batch, Y_, kOutPad, s);
    O2F_CUDA(cudaStreamWaitEvent(s, join_[0], 0));
    k_loss<<<blocks_of(batch, 128), 128, 0, s>>>(batch, Y_, data_out_, index, dY_, loss_buf_, head);
    backward(batch, s, side);
    k_adam<<<blocks_of(n_params_, 256), 256, 0, s>>>(n_params_, params_, grads_, adam_m_, adam_v_, lr, 0.9f, 0.999f,
                                                     1e-8f, head, layers());
    O2F_CUDA(cudaGetLastError());
  } catch (...) {
    cudaStreamEndCapture(s, &graph);
    if (graph) cudaGraphDestroy(graph);
    throw;
  }
  O2F_CUDA(cudaStreamEndCapture(s, &graph));
  const cudaError_t e = cudaGraphInstantiate(&graph_, graph, 0);
  cudaGraphDestroy(graph);
  if (e != cudaSuccess) graph_ = nullptr;
  O2F_CUDA(e);
  graph_launches_ = launches_ - before + 2;
  launches_ = before;
  graph_batch_ = batch;
  graph_lr_ = lr;
  graph_data_ = data_in_;
  graph_loss_ = loss_buf_;
}

Layers Mlp::layers() const {
  Layers ly{};
  for (int l = 0; l <= kHidden; ++l) {
    ly.w_off[l] = w_off_[l];
    ly.w_end[l] = b_off_[l];
    ly.rows[l] = out_dim(l);
    ly.cols[l] = in_dim(l);
    ly.W[l] = Wb_[l];
    ly.WT[l] = WTb_[l];
  }
  return ly;
}

void Mlp::predict(const float* inputs, int64_t n, float* out) {
  if (n <= 0) return;
  float* in_dev = arena_scratch_in(n);
  O2F_CUDA(cudaMemcpyAsync(in_dev, inputs, n * kIn * sizeof(float), cudaMemcpyHostToDevice, stream_));
  for (int64_t b0 = 0; b0 < n; b0 += max_batch_) {
    const int m = (int)std::min<int64_t>(max_batch_, n - b0);
    load_batch(in_dev + b0 * kIn, nullptr, m, stream_);
    forward(m, Y_, kOut, stream_);
    O2F_CUDA(cudaMemcpyAsync(out + b0 * kOut, Y_, (size_t)m * kOut * sizeof(float), cudaMemcpyDeviceToHost, stream_));
  }
  sync();
}

float* Mlp::arena_scratch_in(int64_t n) {
  if (scratch_cap_ < n) {
    scratch_in_ = arena_.alloc<float>(n * kIn);
    scratch_cap_ = n;
  }
  return scratch_in_;
}

void Mlp::gradients(const float* inputs, const float* targets, int n, float* grads_out, float* loss_out) {
  if (n < 1 || n > max_batch_) throw Error(O2F_ERR_ARG, "n out of range");
  float* in_dev = arena_scratch_in(n);
  if (!grad_targets_) grad_targets_ = arena_.alloc<float>((int64_t)max_batch_ * kOut);
  O2F_CUDA(cudaMemcpyAsync(in_dev, inputs, (size_t)n * kIn * sizeof(float), cudaMemcpyHostToDevice, stream_));
  O2F_CUDA(cudaMemcpyAsync(grad_targets_, targets, (size_t)n * kOut * sizeof(float), cudaMemcpyHostToDevice, stream_));
  O2F_CUDA(cudaMemsetAsync(loss_, 0, sizeof(float), stream_));
  load_batch(in_dev, nullptr, n, stream_);
  forward(n, Y_, kOutPad, stream_);
  k_loss<<<blocks_of(n, 128), 128, 0, stream_>>>(n, Y_, grad_targets_, nullptr, dY_, loss_, nullptr);
  O2F_CUDA(cudaMemsetAsync(grads_, 0, n_params_ * sizeof(float), stream_));
  backward(n, stream_, nullptr);
  sync();
  O2F_CUDA(cudaMemcpy(grads_out, grads_, n_params_ * sizeof(float), cudaMemcpyDeviceToHost));
  if (loss_out) O2F_CUDA(cudaMemcpy(loss_out, loss_, sizeof(float), cudaMemcpyDeviceToHost));
}

void Mlp::get_params(float* out, float* freq_out) {
  sync();
  O2F_CUDA(cudaMemcpy(out, params_, n_params_ * sizeof(float), cudaMemcpyDeviceToHost));
  if (freq_out) O2F_CUDA(cudaMemcpy(freq_out, freq_, 2 * kFreq * sizeof(float), cudaMemcpyDeviceToHost));
}

void Mlp::set_params(const float* in) {
  O2F_CUDA(cudaMemcpyAsync(params_, in, n_params_ * sizeof(float), cudaMemcpyHostToDevice, stream_));
  pack();
  sync();
}

}  // namespace mlp
}  // namespace o2f
