// Host side of the learned cost model (hs_mlp_*): parameter storage on the
// device, seeded initialisation, inference, one-shot gradients, and the
// minibatch Adam training loop driving the K7 kernels.
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include "internal.h"

using namespace hisv;

struct hs_mlp {
  int in = 0, P = 0, sms = 148;
  float* d_params = nullptr;
  float* d_m = nullptr;
  float* d_v = nullptr;
  float* d_grad = nullptr;
  float* d_partial = nullptr;  // sms x P
  float* d_lpart = nullptr;    // sms
  int step = 0;                // Adam steps taken
  // a call's buffers, kept for the next one (CallBuffers)
  std::mutex mu;
  char* kept = nullptr;
  size_t kept_bytes = 0;
  int kept_dev = 0;
};

namespace {

// splitmix64: a small seeded generator, identical on every platform
struct Rng {
  uint64_t s;
  uint64_t next() {
    uint64_t z = (s += 0x9e3779b97f4a7c15ull);
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
  }
  double uniform() { return double(next() >> 11) * (1.0 / 9007199254740992.0); }
};

constexpr size_t kKeptBytes = size_t(16) << 20;

// A call's device buffers, cut from one block that the model keeps (up to 16 MiB)
// for its next call.  Allocating and freeing them in every call maps and unmaps
// device memory wherever no other allocation holds the driver's segment: an
// epoch of 8192 rows and the pricing of its rows took 0.8 or 2.1 ms, depending
// on what else the process had allocated.  Calls at the same time on one model
// take the kept block or one of their own.
class CallBuffers {
 public:
  explicit CallBuffers(hs_mlp* m) : m_(m) {}
  ~CallBuffers() {
    if (!base_) return;
    if (idle_ && bytes_ <= kKeptBytes) {
      std::lock_guard<std::mutex> lk(m_->mu);
      std::swap(base_, m_->kept);
      std::swap(bytes_, m_->kept_bytes);
      std::swap(dev_, m_->kept_dev);
    }
    if (base_) cudaFree(base_);
  }
  // room for four arrays of these sizes
  int get(size_t a, size_t b, size_t c, size_t d) {
    const size_t bytes = up(a) + up(b) + up(c) + up(d);
    HS_CUDA(cudaGetDevice(&dev_));
    {
      std::lock_guard<std::mutex> lk(m_->mu);
      if (m_->kept && m_->kept_dev == dev_ && m_->kept_bytes >= bytes) {
        std::swap(base_, m_->kept);
        bytes_ = m_->kept_bytes;
        m_->kept_bytes = 0;
      }
    }
    if (!base_) {
      HS_CUDA(device_malloc(&base_, bytes));
      bytes_ = bytes;
    }
    next_ = base_;
    return HS_OK;
  }
  template <class T>
  T* cut(size_t bytes) {
    T* p = reinterpret_cast<T*>(next_);
    next_ += up(bytes);
    return p;
  }
  // the device has finished with the buffers (or runs the next call's work
  // on them in the same stream, after this one's)
  int done() {
    idle_ = true;
    return HS_OK;
  }

 private:
  static size_t up(size_t b) { return (b + 255) & ~size_t(255); }
  hs_mlp* m_;
  char* base_ = nullptr;
  char* next_ = nullptr;
  size_t bytes_ = 0;
  int dev_ = 0;
  bool idle_ = false;
};

int blocks_for(const hs_mlp* m, int n) { return mlp_backward_blocks(n, m->sms); }

}  // namespace

extern "C" {

int hs_mlp_create(int in_dim, uint64_t seed, hs_mlp** out) {
  if (!out) return set_error(HS_E_INVALID, "null output");
  *out = nullptr;
  if (in_dim < 1 || in_dim > kMlpMaxIn)
    return set_error(HS_E_INVALID, "input width %d outside 1..%d", in_dim, kMlpMaxIn);
  int dev = 0, ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    return set_error(HS_E_NODEVICE, "no CUDA device");
  }
  auto* m = new hs_mlp;
  m->in = in_dim;
  m->P = mlp_num_params(in_dim);
  auto fail = [&](int rc) {
    hs_mlp_destroy(m);
    return rc;
  };
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&m->sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return fail(set_error(HS_E_CUDA, "device query"));
  const size_t pb = sizeof(float) * size_t(m->P);
  if (device_malloc(&m->d_params, pb) != cudaSuccess || device_malloc(&m->d_m, pb) != cudaSuccess ||
      device_malloc(&m->d_v, pb) != cudaSuccess || device_malloc(&m->d_grad, pb) != cudaSuccess ||
      device_malloc(&m->d_partial, pb * size_t(m->sms)) != cudaSuccess ||
      device_malloc(&m->d_lpart, sizeof(float) * size_t(m->sms)) != cudaSuccess) {
    cudaGetLastError();
    return fail(set_error(HS_E_NOMEM, "model buffers"));
  }
  // He-uniform weights (bound sqrt(6 / fan_in)), zero biases
  std::vector<float> p(m->P, 0.f);
  Rng r{seed};
  const int H = kMlpHidden;
  auto fill = [&](int off, int count, int fan_in) {
    const double a = std::sqrt(6.0 / fan_in);
    for (int i = 0; i < count; ++i) p[off + i] = float((2.0 * r.uniform() - 1.0) * a);
  };
  int off = 0;
  fill(off, H * in_dim, in_dim);
  off += H * in_dim + H;
  fill(off, H * H, H);
  off += H * H + H;
  fill(off, H * H, H);
  off += H * H + H;
  fill(off, H, H);
  int rc = hs_mlp_set_params(m, p.data());
  if (rc != HS_OK) return fail(rc);
  *out = m;
  return HS_OK;
}

int hs_mlp_num_params(const hs_mlp* m) { return m ? m->P : set_error(HS_E_INVALID, "null model"); }

int hs_mlp_get_params(hs_mlp* m, float* host) {
  if (!m || !host) return set_error(HS_E_INVALID, "null argument");
  HS_CUDA(cudaMemcpy(host, m->d_params, sizeof(float) * size_t(m->P), cudaMemcpyDeviceToHost));
  return HS_OK;
}

int hs_mlp_set_params(hs_mlp* m, const float* host) {
  if (!m || !host) return set_error(HS_E_INVALID, "null argument");
  const size_t pb = sizeof(float) * size_t(m->P);
  HS_CUDA(cudaMemcpy(m->d_params, host, pb, cudaMemcpyHostToDevice));
  HS_CUDA(cudaMemset(m->d_m, 0, pb));
  HS_CUDA(cudaMemset(m->d_v, 0, pb));
  m->step = 0;
  return HS_OK;
}

int hs_mlp_predict(hs_mlp* m, const float* x, int n, float* y_out) {
  if (!m || (n > 0 && (!x || !y_out)) || n < 0) return set_error(HS_E_INVALID, "bad arguments");
  if (n == 0) return HS_OK;
  const size_t xb = sizeof(float) * size_t(n) * m->in, yb = sizeof(float) * size_t(n);
  CallBuffers buf(m);
  HS_TRY(buf.get(xb, yb, 0, 0));
  float* dx = buf.cut<float>(xb);
  float* dy = buf.cut<float>(yb);
  HS_CUDA(cudaMemcpy(dx, x, xb, cudaMemcpyHostToDevice));
  HS_TRY(launch_mlp_forward(m->d_params, m->in, dx, n, dy, nullptr));
  HS_CUDA(cudaMemcpy(y_out, dy, yb, cudaMemcpyDeviceToHost));
  return buf.done();
}

int hs_mlp_gradients(hs_mlp* m, const float* x, const float* y, int n, float* grad_out,
                     float* loss_out) {
  if (!m || !x || !y || n < 1) return set_error(HS_E_INVALID, "bad arguments");
  const size_t xb = sizeof(float) * size_t(n) * m->in, yb = sizeof(float) * size_t(n);
  CallBuffers buf(m);
  HS_TRY(buf.get(xb, yb, sizeof(float), 0));
  float* dx = buf.cut<float>(xb);
  float* dy = buf.cut<float>(yb);
  float* dl = buf.cut<float>(sizeof(float));
  HS_CUDA(cudaMemcpy(dx, x, xb, cudaMemcpyHostToDevice));
  HS_CUDA(cudaMemcpy(dy, y, yb, cudaMemcpyHostToDevice));
  const int nblk = blocks_for(m, n);
  HS_TRY(launch_mlp_backward(m->d_params, m->in, dx, dy, nullptr, n, 2.f / float(n),
                             m->d_partial, m->d_lpart, nblk, nullptr));
  HS_TRY(launch_mlp_reduce(m->d_partial, m->d_lpart, nblk, m->P, m->d_grad, dl, nullptr));
  if (grad_out)
    HS_CUDA(cudaMemcpy(grad_out, m->d_grad, sizeof(float) * size_t(m->P), cudaMemcpyDeviceToHost));
  if (loss_out) {
    float l = 0.f;
    HS_CUDA(cudaMemcpy(&l, dl, sizeof(float), cudaMemcpyDeviceToHost));
    *loss_out = l / float(n);
  }
  return buf.done();
}

int hs_mlp_train(hs_mlp* m, const float* x, const float* y, int n, int epochs, int batch,
                 float lr, uint64_t seed, float* epoch_loss) {
  if (!m || !x || !y || n < 1 || epochs < 0 || batch < 1 || !(lr > 0.f))
    return set_error(HS_E_INVALID, "bad arguments");
  const int steps_per_epoch = (n + batch - 1) / batch;
  const size_t xb = sizeof(float) * size_t(n) * m->in, yb = sizeof(float) * size_t(n);
  const size_t ib = sizeof(int32_t) * size_t(n), lb = sizeof(float) * size_t(steps_per_epoch);
  CallBuffers buf(m);
  HS_TRY(buf.get(xb, yb, ib, lb));
  float* dx = buf.cut<float>(xb);
  float* dy = buf.cut<float>(yb);
  int32_t* didx = buf.cut<int32_t>(ib);
  float* dl = buf.cut<float>(lb);
  HS_CUDA(cudaMemcpy(dx, x, xb, cudaMemcpyHostToDevice));
  HS_CUDA(cudaMemcpy(dy, y, yb, cudaMemcpyHostToDevice));
  std::vector<int32_t> perm(n);
  std::vector<float> losses(steps_per_epoch);
  Rng r{seed};
  for (int e = 0; e < epochs; ++e) {
    for (int i = 0; i < n; ++i) perm[i] = i;
    for (int i = n - 1; i > 0; --i) std::swap(perm[i], perm[int(r.next() % uint64_t(i + 1))]);
    HS_CUDA(cudaMemcpy(didx, perm.data(), ib, cudaMemcpyHostToDevice));
    for (int st = 0; st < steps_per_epoch; ++st) {
      const int b0 = st * batch, nb = std::min(batch, n - b0);
      const int nblk = blocks_for(m, nb);
      HS_TRY(launch_mlp_backward(m->d_params, m->in, dx, dy, didx + b0, nb, 2.f / float(nb),
                                 m->d_partial, m->d_lpart, nblk, nullptr));
      HS_TRY(launch_mlp_adam(m->d_params, m->d_partial, m->d_lpart, nblk, m->d_m, m->d_v, m->P, lr,
                             0.9f, 0.999f, 1e-8f, ++m->step, dl + st, nullptr));
    }
    if (epoch_loss) {
      HS_CUDA(cudaMemcpy(losses.data(), dl, lb, cudaMemcpyDeviceToHost));
      double s = 0;
      for (float l : losses) s += l;
      epoch_loss[e] = float(s / n);  // mean squared error over the epoch
    }
  }
  HS_CUDA(cudaDeviceSynchronize());
  return buf.done();
}

int hs_mlp_destroy(hs_mlp* m) {
  if (!m) return HS_OK;
  for (float* p : {m->d_params, m->d_m, m->d_v, m->d_grad, m->d_partial, m->d_lpart})
    if (p) cudaFree(p);
  if (m->kept) cudaFree(m->kept);
  delete m;
  return HS_OK;
}

}  // extern "C"
