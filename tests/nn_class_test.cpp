// nn_class_test.cpp -- the reference-compatible NN class as a C++ program uses it: what a caller may read and write on the
// layers around NN::Forward.  Built and run by test_gpu_layers.py with a checkpoint of the network as its argument.
#include <math.h>
#include <stdint.h>
#include <stdio.h>

#include <vector>

#include "Layers.h"

namespace {

int g_failed = 0;
void expect(bool ok, const char* what) {
  if (ok) return;
  printf("FAILED: %s\n", what);
  ++g_failed;
}

template <class T>
std::vector<T> fetch(const void* dev, size_t n) {
  std::vector<T> v(n);
  cudaMemcpy(v.data(), dev, n * sizeof(T), cudaMemcpyDeviceToHost);
  return v;
}
std::vector<uint16_t> halves(const __half* dev, size_t n) { return fetch<uint16_t>(dev, n); }

void scale_on_device(float* dev, size_t n, float by) {
  std::vector<float> v = fetch<float>(dev, n);
  for (float& x : v) x *= by;
  cudaMemcpy(dev, v.data(), n * sizeof(float), cudaMemcpyHostToDevice);
}

// the BatchNorm layers of the network: after the first convolution, in the residual blocks, after the FC layers
std::vector<BatchNorm*> norms(NN& nn) {
  std::vector<BatchNorm*> out{static_cast<BatchNorm*>(nn.layers_[1])};
  for (int i = 3; i < 6; ++i)
    for (int k : {1, 4}) out.push_back(static_cast<BatchNorm*>(static_cast<ResConvLayer*>(nn.layers_[i])->layers_[k]));
  for (int i : {7, 10, 13}) out.push_back(static_cast<BatchNorm*>(nn.layers_[i]));
  return out;
}

__half* one_by_one(NN& nn, __half* x) {
  for (Layer* l : nn.layers_) x = l->Forward(x);
  return x;
}

float largest_difference(NN& a, NN& b, __half* frame) {
  const std::vector<__half> x = fetch<__half>(a.Forward(frame), numCtrls_), y = fetch<__half>(b.Forward(frame), numCtrls_);
  float most = 0.f;
  for (int i = 0; i < numCtrls_; ++i) most = fmaxf(most, fabsf(__half2float(x[i]) - __half2float(y[i])) / fmaxf(1.f, fabsf(__half2float(y[i]))));
  return most;
}

void compare(NN& a, NN& b, __half* frame, const char* when) {
  const std::vector<uint16_t> got = halves(a.Forward(frame), numCtrls_), want = halves(one_by_one(b, frame), numCtrls_);
  char what[128];
  snprintf(what, sizeof(what), "NN::Forward differs from its layers one by one, %s", when);
  expect(got == want, what);
  snprintf(what, sizeof(what), "a layer's output buffer differs after NN::Forward, %s", when);
  for (int i : {0, 6, 9, 12, 15}) {
    const size_t n = a.layers_[i]->outNCHW_;
    const __half *x = i == 0 ? static_cast<ConvLayer*>(a.layers_[i])->outData_ : static_cast<FCLayer*>(a.layers_[i])->outData_;
    const __half *y = i == 0 ? static_cast<ConvLayer*>(b.layers_[i])->outData_ : static_cast<FCLayer*>(b.layers_[i])->outData_;
    expect(halves(x, n) == halves(y, n), what);
  }
  const std::vector<BatchNorm*> na = norms(a), nb = norms(b);
  for (size_t i = 0; i < na.size(); ++i) expect(halves(na[i]->outData_, na[i]->outNCHW_) == halves(nb[i]->outData_, nb[i]->outNCHW_), what);
}

}  // namespace

int main(int argc, char** argv) {
  if (argc != 2) return 2;
  cudnnHandle_t handle;
  if (cudnnCreate(&handle) != 0) return 3;
  {
    NN a(handle, handle, 0, 0, false, argv[1]), b(handle, handle, 0, 0, false, argv[1]);
    std::vector<__half> host((size_t)3 * a.inWidth_ * a.inHeight_);
    for (size_t i = 0; i < host.size(); ++i) host[i] = __float2half((float)((i * 2654435761u >> 8) & 255) / 255.0f);
    __half* frame = nullptr;
    cudaMalloc(reinterpret_cast<void**>(&frame), host.size() * sizeof(__half));
    cudaMemcpy(frame, host.data(), host.size() * sizeof(__half), cudaMemcpyHostToDevice);

    compare(a, b, frame, "as loaded");
    const std::vector<uint16_t> before = halves(a.Forward(frame), numCtrls_);
    for (NN* nn : {&a, &b})
      for (BatchNorm* n : norms(*nn)) scale_on_device(n->bnScale_, n->paramCount_, 0.75f);
    compare(a, b, frame, "after the BatchNorm arrays were written on the device");
    expect(halves(a.Forward(frame), numCtrls_) != before, "the written BatchNorm arrays have no effect");

    // the fused launches, where a program asks for them: the same network with fewer roundings (the bound that
    // test_reference_network_sizes derives), and parameters that SyncWeights announces
    expect(a.UseFusedInference(), "the fused launches cover this size");
    expect(largest_difference(a, b, frame) < 8e-3f, "fused launches against the layers");
    for (NN* nn : {&a, &b})
      for (BatchNorm* n : norms(*nn)) {
        scale_on_device(n->bnScale_, n->paramCount_, 1.25f);
        n->SyncWeights();
      }
    expect(largest_difference(a, b, frame) < 8e-3f, "fused launches against the layers, after SyncWeights");
    cudaFree(frame);
  }
  cudnnDestroy(handle);
  if (g_failed == 0) printf("all as expected\n");
  return g_failed ? 1 : 0;
}
