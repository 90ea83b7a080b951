// hw_mlp.cu -- the learned depth operator's per-point network (no counterpart in the
// reference): 5 features -> 32 -> 32 (tanh) -> K = 4 logits -> softmax weights over K
// reference-depth operators.  FP32 training on the GPU with hand-written kernels:
// forward + loss and backward with the parameter gradients summed per block, then the
// blocks' sums and Adam.  Inference writes the per-point weights that replace the
// interpolation weights (gamma_j) of the varying-depth operator HSS.
//
// Per-point training record (kRec floats): 5 features, then K*kBand band matrix
// G[m][j] = C^2(kappa_m, D_j) of the K learned references at the point's band
// wavenumbers kappa_m, then kBand targets T[m] = effective C^2(kappa_m) of the
// 16-reference operator at the point.  Loss per point: mean_m ((sum_j w_j G_mj - T_m)/T_m)^2.
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <string>
#include <vector>

namespace {

constexpr int kIn = 5, kH = 32, kK = 4, kBand = 8;
constexpr int kRec = kIn + kK * kBand + kBand;   // 45
// parameter layout: W1[kH][kIn], b1[kH], W2[kH][kH], b2[kH], W3[kK][kH], b3[kK]
constexpr int oW1 = 0, ob1 = oW1 + kH * kIn, oW2 = ob1 + kH, ob2 = oW2 + kH * kH, oW3 = ob2 + kH,
              ob3 = oW3 + kK * kH, kParams = ob3 + kK;
constexpr int kSub = 8;                       // threads of one record
constexpr int kTile = 32;                     // records a block holds at a time
constexpr int kBlock = kSub * kTile;
constexpr int kMaxBlocks = 2 * 148;           // partial sums kept (two blocks an SM)
constexpr int kPart = ((kParams + 1 + 31) / 32) * 32;   // floats of a block's sums: parameters, loss

struct Act {
  float h1[kH], h2[kH], w[kK];
};

__device__ __forceinline__ void forward(const float* __restrict__ P, const float* x, Act& a) {
  for (int i = 0; i < kH; ++i) {
    float s = P[ob1 + i];
    for (int j = 0; j < kIn; ++j) s += P[oW1 + i * kIn + j] * x[j];
    a.h1[i] = tanhf(s);
  }
  for (int i = 0; i < kH; ++i) {
    float s = P[ob2 + i];
    for (int j = 0; j < kH; ++j) s += P[oW2 + i * kH + j] * a.h1[j];
    a.h2[i] = tanhf(s);
  }
  float z[kK], zmax = -1e30f;
  for (int i = 0; i < kK; ++i) {
    float s = P[ob3 + i];
    for (int j = 0; j < kH; ++j) s += P[oW3 + i * kH + j] * a.h2[j];
    z[i] = s;
    zmax = fmaxf(zmax, s);
  }
  float den = 0.f;
  for (int i = 0; i < kK; ++i) {
    z[i] = expf(z[i] - zmax);
    den += z[i];
  }
  for (int i = 0; i < kK; ++i) a.w[i] = z[i] / den;
}

// sum over the eight threads of a record
__device__ __forceinline__ float sub_sum(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  return v + __shfl_xor_sync(0xffffffffu, v, 4);
}

// Loss and parameter gradients summed over n records: block b's sums into part[b][.].
// Eight threads share a record (four of the 32 hidden units each, one band wavenumber
// each in the loss), a block holds 32 records at a time and walks on by the grid.  A
// minibatch of 4096 is 128 blocks, one wave; with a thread to a record and 64 blocks of
// two warps it was bound by the latency of 4000 dependent multiply-adds a thread.  The
// parameters' owners sum over a tile's records from shared memory, and keep their sums in
// registers from tile to tile.
__global__ void __launch_bounds__(kBlock) k_mlp_grad(const float* __restrict__ P, const float* __restrict__ data,
                                                     int n, float* __restrict__ part) {
  constexpr int kRow = kH + 2;   // padded: two-float reads, records of a warp on other banks
  __shared__ float sP[kParams], sW2T[kH * kH];
  __shared__ float rec[kTile][kRec];
  __shared__ __align__(8) float h1[kTile][kRow], h2[kTile][kRow], d1[kTile][kRow], d2[kTile][kRow];
  __shared__ float dzs[kTile][kK];
  __shared__ float sl[kBlock / 32];
  const int t = threadIdx.x, r = t / kSub, sub = t % kSub;
  for (int i = t; i < kParams; i += kBlock) sP[i] = P[i];
  for (int i = t; i < kH * kH; i += kBlock) sW2T[(i % kH) * kH + i / kH] = P[oW2 + i];
  float g2[4] = {0.f, 0.f, 0.f, 0.f}, ge[2] = {0.f, 0.f}, loss = 0.f;
  const int i0 = 2 * (t / 16), j0 = 2 * (t % 16);   // this thread's 2 x 2 block of W2
  for (int base = blockIdx.x * kTile; base < n; base += gridDim.x * kTile) {
    const int cnt = n - base < kTile ? n - base : kTile;
    __syncthreads();   // the last tile's readers are done
    for (int i = t; i < cnt * kRec; i += kBlock) (&rec[0][0])[i] = data[size_t(base) * kRec + i];
    __syncthreads();
    const bool on = r < cnt;
    const float* x = rec[r];
    float a1[4], a2[4], dz[kK] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = sub + kSub * u;
      float s = sP[ob1 + i];
#pragma unroll
      for (int j = 0; j < kIn; ++j) s += sP[oW1 + i * kIn + j] * (on ? x[j] : 0.f);
      a1[u] = on ? tanhf(s) : 0.f;
      h1[r][i] = a1[u];
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < 4; ++u) a2[u] = sP[ob2 + sub + kSub * u];
#pragma unroll 8
    for (int j = 0; j < kH; ++j) {
      const float v = h1[r][j];
#pragma unroll
      for (int u = 0; u < 4; ++u) a2[u] += sW2T[j * kH + sub + kSub * u] * v;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      a2[u] = on ? tanhf(a2[u]) : 0.f;
      h2[r][sub + kSub * u] = a2[u];
    }
    // softmax of the four logits, the loss's band `sub`, dL/dz
    float z[kK], zmax = -1e30f;
#pragma unroll
    for (int k = 0; k < kK; ++k) {
      float s = 0.f;
#pragma unroll
      for (int u = 0; u < 4; ++u) s += sP[oW3 + k * kH + sub + kSub * u] * a2[u];
      z[k] = sP[ob3 + k] + sub_sum(s);
      zmax = fmaxf(zmax, z[k]);
    }
    float den = 0.f;
#pragma unroll
    for (int k = 0; k < kK; ++k) {
      z[k] = expf(z[k] - zmax);
      den += z[k];
    }
#pragma unroll
    for (int k = 0; k < kK; ++k) z[k] = z[k] / den;
    float e = 0.f, dp = 0.f, G[kK] = {0.f, 0.f, 0.f, 0.f};
    if (on) {
      const float T = x[kIn + kK * kBand + sub];
      float p = 0.f;
#pragma unroll
      for (int k = 0; k < kK; ++k) {
        G[k] = x[kIn + sub * kK + k];
        p += z[k] * G[k];
      }
      e = (p - T) / T;
      dp = 2.f * e / (T * kBand);
      loss += e * e / kBand;
    }
    float dw[kK], s = 0.f;
#pragma unroll
    for (int k = 0; k < kK; ++k) {
      dw[k] = sub_sum(dp * G[k]);
      s += z[k] * dw[k];
    }
#pragma unroll
    for (int k = 0; k < kK; ++k) dz[k] = z[k] * (dw[k] - s);
    if (sub < kK) dzs[r][sub] = sub == 0 ? dz[0] : (sub == 1 ? dz[1] : (sub == 2 ? dz[2] : dz[3]));
    // backward through the hidden layers (zero for records past the end: dz is)
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = sub + kSub * u;
      float v = 0.f;
#pragma unroll
      for (int k = 0; k < kK; ++k) v += sP[oW3 + k * kH + i] * dz[k];
      d2[r][i] = v * (1.f - a2[u] * a2[u]);
    }
    __syncwarp();
    float b1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
    for (int k = 0; k < kH; ++k) {
      const float v = d2[r][k];
#pragma unroll
      for (int u = 0; u < 4; ++u) b1[u] += sP[oW2 + k * kH + sub + kSub * u] * v;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) d1[r][sub + kSub * u] = b1[u] * (1.f - a1[u] * a1[u]);
    __syncthreads();
    // parameter gradients over the tile's records
#pragma unroll 4
    for (int q = 0; q < kTile; ++q) {
      const float2 d = *reinterpret_cast<const float2*>(&d2[q][i0]), h = *reinterpret_cast<const float2*>(&h1[q][j0]);
      g2[0] += d.x * h.x;
      g2[1] += d.x * h.y;
      g2[2] += d.y * h.x;
      g2[3] += d.y * h.y;
    }
    // the others: W1, b1, b2, W3, b3 in that order, two a thread
#pragma unroll
    for (int v = 0; v < 2; ++v) {
      int p = t + v * kBlock;
      float sum = ge[v];
      if (p < ob1) {
        const int i = p / kIn, j = p % kIn;
        for (int q = 0; q < cnt; ++q) sum += d1[q][i] * rec[q][j];
      } else if (p < oW2) {
        for (int q = 0; q < cnt; ++q) sum += d1[q][p - ob1];
      } else if ((p += kH * kH) < oW3) {
        for (int q = 0; q < cnt; ++q) sum += d2[q][p - ob2];
      } else if (p < ob3) {
        const int i = (p - oW3) / kH, j = (p - oW3) % kH;
        for (int q = 0; q < cnt; ++q) sum += dzs[q][i] * h2[q][j];
      } else if (p < kParams) {
        for (int q = 0; q < cnt; ++q) sum += dzs[q][p - ob3];
      }
      ge[v] = sum;
    }
  }
  float* out = part + size_t(blockIdx.x) * kPart;
#pragma unroll
  for (int v = 0; v < 4; ++v) out[oW2 + (i0 + v / 2) * kH + j0 + v % 2] = g2[v];
#pragma unroll
  for (int v = 0; v < 2; ++v) {
    int p = t + v * kBlock;
    if (p >= oW2) p += kH * kH;
    if (p < kParams) out[p] = ge[v];
  }
  for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
  if ((t & 31) == 0) sl[t >> 5] = loss;
  __syncthreads();
  if (t == 0) {
    float s = 0.f;
    for (int q = 0; q < kBlock / 32; ++q) s += sl[q];
    out[kParams] = s;
  }
}

// the blocks' sums of 32 consecutive entries of part: warp w adds every eighth block's,
// then the eight are added in shared memory; returns the sum of entry 32 blockIdx.x + lane
// in warp 0
__device__ __forceinline__ float sum_blocks(const float* __restrict__ part, int nb) {
  __shared__ float red[8][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const float* p = part + blockIdx.x * 32 + lane;
  float s = 0.f;
#pragma unroll 8
  for (int b = w; b < nb; b += 8) s += p[size_t(b) * kPart];
  red[w][lane] = s;
  __syncthreads();
  float v = 0.f;
  if (w == 0)
    for (int q = 0; q < 8; ++q) v += red[q][lane];
  return v;
}

// gradient and loss sums alone
__global__ void __launch_bounds__(256) k_mlp_sum(const float* __restrict__ part, int nb, float* __restrict__ grad,
                                                 float* __restrict__ loss) {
  const float s = sum_blocks(part, nb);
  const int p = blockIdx.x * 32 + (threadIdx.x & 31);
  if (threadIdx.x >= 32) return;
  if (p < kParams) grad[p] = s;
  else if (p == kParams) *loss = s;
}

// Adam on the mean gradient (the blocks' sum / n); the minibatch's loss sum into *loss
__global__ void __launch_bounds__(256) k_adam(float* __restrict__ P, const float* __restrict__ part, int nb,
                                              float* __restrict__ m1, float* __restrict__ m2, float inv_n, float lr,
                                              float b1, float b2, float eps, float c1, float c2, float* __restrict__ loss) {
  const float s = sum_blocks(part, nb);
  const int p = blockIdx.x * 32 + (threadIdx.x & 31);
  if (threadIdx.x >= 32) return;
  if (p == kParams) *loss = s;
  if (p >= kParams) return;
  const float g = s * inv_n;
  m1[p] = b1 * m1[p] + (1.f - b1) * g;
  m2[p] = b2 * m2[p] + (1.f - b2) * g * g;
  const float mh = m1[p] / c1, vh = m2[p] / c2;
  P[p] -= lr * mh / (sqrtf(vh) + eps);
}

int grad_blocks(int n) {
  const int b = (n - 1) / kTile + 1;
  return b < kMaxBlocks ? b : kMaxBlocks;
}

__global__ void k_mlp_infer(const float* __restrict__ P, const float* __restrict__ feat, int n,
                            double* __restrict__ w_out) {
  __shared__ float sP[kParams];
  for (int i = threadIdx.x; i < kParams; i += blockDim.x) sP[i] = P[i];
  __syncthreads();
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  float x[kIn];
  for (int j = 0; j < kIn; ++j) x[j] = feat[size_t(r) * kIn + j];
  Act a;
  forward(sP, x, a);
  for (int k = 0; k < kK; ++k) w_out[size_t(k) * n + r] = double(a.w[k]);   // [K][n]
}

std::string g_mlp_err;

}  // namespace

struct hw_mlp {
  float *P = nullptr, *m1 = nullptr, *m2 = nullptr, *grad = nullptr, *loss = nullptr, *part = nullptr;
  float* records = nullptr;       // device copy of the records a call is given, and its room
  size_t record_floats = 0;
  float* losses = nullptr;        // loss sum of every minibatch of a call
  size_t loss_floats = 0;
  cudaStream_t copy = nullptr;    // the records' way to the device, beside the training steps
  cudaEvent_t arrived = nullptr;
  int step = 0;
  int device = 0;
  std::string err;
};

#define MLP_CUDA(call)                                                             \
  do {                                                                             \
    cudaError_t e_ = (call);                                                       \
    if (e_ != cudaSuccess) {                                                       \
      mlp->err = std::string(#call) + ": " + cudaGetErrorString(e_);               \
      return 1;                                                                    \
    }                                                                              \
  } while (0)

extern "C" {

void hw_mlp_destroy(hw_mlp* mlp);

int hw_mlp_sizes(int* n_in, int* n_hidden, int* n_out, int* n_band, int* n_params) {
  if (n_in) *n_in = kIn;
  if (n_hidden) *n_hidden = kH;
  if (n_out) *n_out = kK;
  if (n_band) *n_band = kBand;
  if (n_params) *n_params = kParams;
  return kRec;
}

hw_mlp* hw_mlp_create(unsigned long long seed, int device) {
  hw_mlp* mlp = new hw_mlp();
  mlp->device = device;
  if (cudaSetDevice(device) != cudaSuccess) { g_mlp_err = "cudaSetDevice failed"; delete mlp; return nullptr; }
  // Xavier-uniform initialisation from a splitmix64 stream, zero biases
  std::vector<float> p(kParams, 0.f);
  unsigned long long s = seed;
  auto uni = [&]() {
    unsigned long long z = (s += 0x9E3779B97F4A7C15ULL);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    z ^= z >> 31;
    return double(z >> 11) * (1.0 / 9007199254740992.0);
  };
  auto fill = [&](int off, int fan_out, int fan_in) {
    const double a = std::sqrt(6.0 / (fan_in + fan_out));
    for (int i = 0; i < fan_out * fan_in; ++i) p[off + i] = float((2 * uni() - 1) * a);
  };
  fill(oW1, kH, kIn);
  fill(oW2, kH, kH);
  fill(oW3, kK, kH);
  bool ok = cudaMalloc(&mlp->P, sizeof(float) * kParams) == cudaSuccess &&
            cudaMalloc(&mlp->m1, sizeof(float) * kParams) == cudaSuccess &&
            cudaMalloc(&mlp->m2, sizeof(float) * kParams) == cudaSuccess &&
            cudaMalloc(&mlp->grad, sizeof(float) * kParams) == cudaSuccess &&
            cudaMalloc(&mlp->loss, sizeof(float)) == cudaSuccess &&
            cudaMalloc(&mlp->part, sizeof(float) * kMaxBlocks * kPart) == cudaSuccess &&
            cudaStreamCreateWithFlags(&mlp->copy, cudaStreamNonBlocking) == cudaSuccess &&
            cudaEventCreateWithFlags(&mlp->arrived, cudaEventDisableTiming) == cudaSuccess &&
            cudaMemcpy(mlp->P, p.data(), sizeof(float) * kParams, cudaMemcpyHostToDevice) == cudaSuccess &&
            cudaMemset(mlp->m1, 0, sizeof(float) * kParams) == cudaSuccess &&
            cudaMemset(mlp->m2, 0, sizeof(float) * kParams) == cudaSuccess;
  if (!ok) { g_mlp_err = "device allocation failed"; hw_mlp_destroy(mlp); return nullptr; }
  return mlp;
}

void hw_mlp_destroy(hw_mlp* mlp) {
  if (!mlp) return;
  if (mlp->copy) cudaStreamSynchronize(mlp->copy);
  for (float* p : {mlp->P, mlp->m1, mlp->m2, mlp->grad, mlp->loss, mlp->part, mlp->records, mlp->losses}) cudaFree(p);
  if (mlp->arrived) cudaEventDestroy(mlp->arrived);
  if (mlp->copy) cudaStreamDestroy(mlp->copy);
  delete mlp;
}

const char* hw_mlp_last_error(const hw_mlp* mlp) { return mlp ? mlp->err.c_str() : g_mlp_err.c_str(); }

int hw_mlp_get_params(hw_mlp* mlp, float* out) {
  MLP_CUDA(cudaMemcpy(out, mlp->P, sizeof(float) * kParams, cudaMemcpyDeviceToHost));
  return 0;
}

int hw_mlp_set_params(hw_mlp* mlp, const float* in) {
  MLP_CUDA(cudaMemcpy(mlp->P, in, sizeof(float) * kParams, cudaMemcpyHostToDevice));
  mlp->step = 0;
  MLP_CUDA(cudaMemset(mlp->m1, 0, sizeof(float) * kParams));
  MLP_CUDA(cudaMemset(mlp->m2, 0, sizeof(float) * kParams));
  return 0;
}

// Summed loss and parameter gradients over n device-resident records.
int hw_mlp_grad_device(hw_mlp* mlp, const float* data_dev, int n, float* grad_host, float* loss_host) {
  if (n <= 0) { mlp->err = "gradient: no records"; return 1; }
  const int nb = grad_blocks(n);
  k_mlp_grad<<<nb, kBlock>>>(mlp->P, data_dev, n, mlp->part);
  MLP_CUDA(cudaGetLastError());
  k_mlp_sum<<<kPart / 32, 256>>>(mlp->part, nb, mlp->grad, mlp->loss);
  MLP_CUDA(cudaGetLastError());
  if (grad_host) MLP_CUDA(cudaMemcpy(grad_host, mlp->grad, sizeof(float) * kParams, cudaMemcpyDeviceToHost));
  if (loss_host) MLP_CUDA(cudaMemcpy(loss_host, mlp->loss, sizeof(float), cudaMemcpyDeviceToHost));
  return 0;
}

namespace {
// room for `count` floats in a buffer of the handle's that grows and is kept
bool room(float*& p, size_t& have, size_t count) {
  if (count <= have) return true;
  cudaFree(p);
  p = nullptr;
  have = 0;
  if (cudaMalloc(&p, sizeof(float) * count) != cudaSuccess) return false;
  have = count;
  return true;
}
}  // namespace

// Adam over minibatches of `batch` host records; losses[epoch] = mean loss.  The records
// go to the device minibatch by minibatch while the first epoch's steps run, and nothing
// waits for a step's loss: the minibatches' sums come back once, at the end.
int hw_mlp_train(hw_mlp* mlp, const float* data_host, int n, int epochs, int batch, float lr, float* losses) {
  if (n < 0) { mlp->err = "training: n must not be negative"; return 1; }
  if (n == 0 || epochs <= 0) {   // no step to take, whatever the batch: the mean loss of no records
    for (int ep = 0; losses && ep < epochs; ++ep) losses[ep] = std::nanf("");
    return 0;
  }
  if (batch <= 0) { mlp->err = "training: batch must be positive"; return 1; }
  const int per = (n - 1) / batch + 1;
  if (!room(mlp->records, mlp->record_floats, size_t(n) * kRec) ||
      !room(mlp->losses, mlp->loss_floats, size_t(per) * epochs)) {
    cudaGetLastError();
    mlp->err = "training: out of device memory";
    return 1;
  }
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  // a former call's kernels may still read the records
  MLP_CUDA(cudaEventRecord(mlp->arrived, nullptr));
  MLP_CUDA(cudaStreamWaitEvent(mlp->copy, mlp->arrived, 0));
  for (int ep = 0; ep < epochs; ++ep) {
    for (int k = 0; k < per; ++k) {
      const size_t off = size_t(k) * batch;
      const int cnt = int(off + batch <= size_t(n) ? size_t(batch) : size_t(n) - off);
      float* d = mlp->records + off * kRec;
      if (ep == 0) {
        MLP_CUDA(cudaMemcpyAsync(d, data_host + off * kRec, sizeof(float) * size_t(cnt) * kRec, cudaMemcpyHostToDevice,
                                 mlp->copy));
        MLP_CUDA(cudaEventRecord(mlp->arrived, mlp->copy));
        MLP_CUDA(cudaStreamWaitEvent(nullptr, mlp->arrived, 0));
      }
      const int nb = grad_blocks(cnt);
      k_mlp_grad<<<nb, kBlock>>>(mlp->P, d, cnt, mlp->part);
      ++mlp->step;
      const float c1 = 1.f - std::pow(b1, float(mlp->step)), c2 = 1.f - std::pow(b2, float(mlp->step));
      k_adam<<<kPart / 32, 256>>>(mlp->P, mlp->part, nb, mlp->m1, mlp->m2, 1.f / cnt, lr, b1, b2, eps, c1, c2,
                                  mlp->losses + size_t(ep) * per + k);
      MLP_CUDA(cudaGetLastError());
    }
  }
  std::vector<float> sums(size_t(per) * epochs);
  MLP_CUDA(cudaMemcpy(sums.data(), mlp->losses, sizeof(float) * sums.size(), cudaMemcpyDeviceToHost));
  if (losses)
    for (int ep = 0; ep < epochs; ++ep) {
      double tot = 0.0;
      for (int k = 0; k < per; ++k) tot += sums[size_t(ep) * per + k];
      losses[ep] = float(tot / n);
    }
  return 0;
}

// Per-point softmax weights [K][n] (double) for n feature rows (host in, host out).
int hw_mlp_infer(hw_mlp* mlp, const float* feat_host, int n, double* w_host) {
  float* f = nullptr;
  double* w = nullptr;
  MLP_CUDA(cudaMalloc(&f, sizeof(float) * size_t(n) * kIn));
  MLP_CUDA(cudaMalloc(&w, sizeof(double) * size_t(n) * kK));
  MLP_CUDA(cudaMemcpy(f, feat_host, sizeof(float) * size_t(n) * kIn, cudaMemcpyHostToDevice));
  k_mlp_infer<<<(n + 255) / 256, 256>>>(mlp->P, f, n, w);
  MLP_CUDA(cudaGetLastError());
  MLP_CUDA(cudaMemcpy(w_host, w, sizeof(double) * size_t(n) * kK, cudaMemcpyDeviceToHost));
  cudaFree(f);
  cudaFree(w);
  return 0;
}

// host-buffer convenience for the gradient check
int hw_mlp_grad(hw_mlp* mlp, const float* data_host, int n, float* grad_host, float* loss_host) {
  if (!room(mlp->records, mlp->record_floats, size_t(n > 0 ? n : 0) * kRec)) {
    cudaGetLastError();
    mlp->err = "gradient: out of device memory";
    return 1;
  }
  MLP_CUDA(cudaMemcpy(mlp->records, data_host, sizeof(float) * size_t(n) * kRec, cudaMemcpyHostToDevice));
  return hw_mlp_grad_device(mlp, mlp->records, n, grad_host, loss_host);
}

}  // extern "C"
