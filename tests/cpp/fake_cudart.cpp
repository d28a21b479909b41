// Preloaded before libcudart: chosen calls return an error code instead of
// running, so that a test can make them fail without a fault on the device.
//   fake_fail(call, nth, code): the nth next run of `call` returns `code`.
//   fake_runs(call): runs of `call` so far (failed ones included).
//   fake_bytes(): bytes that cudaMalloc was asked for so far.
#include <cuda_runtime_api.h>
#include <dlfcn.h>

#include <cstring>

namespace {
struct Call {
  const char* name;
  long runs = 0, fail_in = 0;
  cudaError_t code = cudaSuccess;
};
long bytes = 0;
Call calls[] = {{"cudaMalloc"}, {"cudaGraphInstantiate"}};

void* real(const char* name) {
  void* const h = dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD);
  return dlsym(h, name);
}
// whether this run fails, and how
bool fails(Call& c) {
  ++c.runs;
  return c.fail_in > 0 && --c.fail_in == 0;
}
Call* find(const char* name) {
  for (Call& c : calls)
    if (!std::strcmp(c.name, name)) return &c;
  return nullptr;
}
}  // namespace

extern "C" {

void fake_fail(const char* name, long nth, int code) {
  Call* const c = find(name);
  c->fail_in = nth;
  c->code = static_cast<cudaError_t>(code);
}
long fake_runs(const char* name) { return find(name)->runs; }
long fake_bytes() { return bytes; }

cudaError_t cudaMalloc(void** p, size_t n) {
  bytes += static_cast<long>(n);
  if (fails(calls[0])) return calls[0].code;
  static const auto f = reinterpret_cast<cudaError_t (*)(void**, size_t)>(real("cudaMalloc"));
  return f(p, n);
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long flags) {
  if (fails(calls[1])) return calls[1].code;
  static const auto f =
      reinterpret_cast<cudaError_t (*)(cudaGraphExec_t*, cudaGraph_t, unsigned long long)>(
          real("cudaGraphInstantiate"));
  return f(e, g, flags);
}

}  // extern "C"
