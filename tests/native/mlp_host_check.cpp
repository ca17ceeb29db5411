// The host side of the sweep surrogate (boids_mlp.o) on a stand-in for the
// CUDA runtime that keeps to the latest moment the runtime's contract allows:
// nothing queued on a stream happens before something waits for it, and
// kernels do nothing.  Copies from host memory remember what the memory held
// when they were queued, so a caller that writes or frees it too early shows.
//
//   mlp_host_check train HIDDEN ROWS BATCH EPOCHS [FAIL_AT]
//       one training call; with FAIL_AT the so-many-th queued operation after
//       its start fails.  Prints "rc copies late pending orders distinct".
//   mlp_host_check image FAIL_AT
//       two forward calls, the first with its so-many-th operation failing (0:
//       none).  Prints "rc rc images", images: how often the second call laid
//       the weight image out.
#include <cuda_runtime_api.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <set>
#include <string>
#include <vector>

#include "boids.h"

namespace {

struct Op {
    std::function<void()> run;
    const void *host = nullptr;  // source in host memory (null: none)
};
std::vector<Op> queue_;          // one stream's worth: the library uses one
size_t done_ = 0;                // operations of it that have happened
std::map<void *, size_t> events_;
int late_ = 0, copies_ = 0, queued_ = 0, fail_at_ = 0;
cudaError_t last_ = cudaSuccess;
std::vector<std::vector<int>> orders_;  // index arrays that arrived, by their size
size_t order_bytes_ = 0;

void run_to(size_t end)
{
    for (; done_ < end; ++done_) queue_[done_].run();
}
void drain() { run_to(queue_.size()); }
int pending()
{
    int n = 0;
    for (size_t i = done_; i < queue_.size(); ++i) n += queue_[i].host != nullptr;
    return n;
}
cudaError_t put(Op op)
{
    if (++queued_ == fail_at_) return last_ = cudaErrorUnknown;
    queue_.push_back(std::move(op));
    return cudaSuccess;
}
std::map<const void *, std::string> &names()   // kernels, by their host stubs (registered before main)
{
    static std::map<const void *, std::string> n;
    return n;
}
std::map<std::string, int> launches_;          // those launched
cudaError_t launched(const void *f)
{
    const cudaError_t e = put(Op{[] {}, nullptr});
    if (e == cudaSuccess) ++launches_[names()[f]];
    return e;
}

}  // namespace

namespace boidsgpu {
int set_last_error(int code, const char *msg)
{
    std::fprintf(stderr, "%s\n", msg);
    return code;
}
}  // namespace boidsgpu

extern "C" {

void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *f, char *, const char *name, int, void *, void *, void *, void *, int *)
{
    names()[f] = name;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f)
{
    *k = (cudaKernel_t)f;
    return cudaSuccess;
}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void *) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *, dim3 *, size_t *, void *) { return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void **, size_t, cudaStream_t) { return launched(k); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *, const void *f, void **) { return launched(f); }

cudaError_t cudaMalloc(void **p, size_t n) { *p = std::calloc(n, 1); return cudaSuccess; }
cudaError_t cudaFree(void *p) { drain(); std::free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { *p = std::calloc(n, 1); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { drain(); std::free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { drain(); std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemset(void *d, int v, size_t n) { drain(); std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind kind, cudaStream_t)
{
    Op op;
    if (kind == cudaMemcpyHostToDevice) {
        const unsigned char *b = static_cast<const unsigned char *>(s);
        std::vector<unsigned char> was(b, b + n);
        op.host = s;
        op.run = [d, s, n, was] {
            ++copies_;
            late_ += std::memcmp(s, was.data(), n) != 0;
            std::memcpy(d, s, n);
            if (n == order_bytes_) orders_.emplace_back((const int *)s, (const int *)s + n / 4);
        };
    } else {
        op.run = [d, s, n] { std::memcpy(d, s, n); };
    }
    return put(std::move(op));
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t)
{
    return put(Op{[d, v, n] { std::memset(d, v, n); }, nullptr});
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { drain(); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { drain(); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned)
{
    *e = (cudaEvent_t)std::malloc(1);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) { events_[e] = queue_.size(); return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e)
{
    if (events_.count(e)) run_to(std::max(done_, events_[e]));
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { events_.erase(e); std::free(e); return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetLastError(void)
{
    const cudaError_t e = last_;
    last_ = cudaSuccess;
    return e;
}
const char *cudaGetErrorString(cudaError_t) { return "error of the stand-in"; }

}  // extern "C"

static int train(int hidden, int rows, int batch, int epochs, int fail_at)
{
    boids_mlp *m = nullptr;
    if (boids_mlp_create(8, hidden, 4, 1, 0, &m)) return 1;
    std::vector<float> x(8 * (size_t)rows, 0.5f), t(4 * (size_t)rows, 0.25f);
    order_bytes_ = sizeof(int) * (size_t)rows;
    queued_ = copies_ = late_ = 0;
    fail_at_ = fail_at;
    double loss = 0;
    const int rc = boids_mlp_train(m, x.data(), t.data(), rows, epochs, batch, 1e-3f, 7, &loss);
    const int left = pending();
    fail_at_ = 0;
    if (!left) drain();
    bool all = true;
    for (const auto &o : orders_) {  // each a permutation of the rows
        std::set<int> s(o.begin(), o.end());
        all = all && (int)s.size() == rows && *s.begin() == 0 && *s.rbegin() == rows - 1;
    }
    const std::set<std::vector<int>> distinct(orders_.begin(), orders_.end());
    std::printf("%d %d %d %d %d %d\n", rc, copies_, late_, left, all ? (int)orders_.size() : -1, (int)distinct.size());
    if (!left) boids_mlp_destroy(m);
    return 0;
}

static int image(int fail_at)
{
    boids_mlp *m = nullptr;
    if (boids_mlp_create(8, 256, 4, 1, 0, &m)) return 1;
    std::vector<float> x(8 * 100, 0.5f), y(4 * 100);
    queued_ = 0;
    fail_at_ = fail_at;
    const int rc1 = boids_mlp_forward(m, x.data(), 100, y.data());
    fail_at_ = 0;
    cudaGetLastError();
    launches_.clear();
    const int rc2 = boids_mlp_forward(m, x.data(), 100, y.data());
    int images = 0;
    for (const auto &l : launches_)
        if (l.first.find("k_mlp_tile_w") != std::string::npos) images += l.second;
    std::printf("%d %d %d\n", rc1, rc2, images);
    boids_mlp_destroy(m);
    return 0;
}

int main(int argc, char **argv)
{
    if (argc >= 6 && !std::strcmp(argv[1], "train"))
        return train(std::atoi(argv[2]), std::atoi(argv[3]), std::atoi(argv[4]), std::atoi(argv[5]),
                     argc > 6 ? std::atoi(argv[6]) : 0);
    if (argc == 3 && !std::strcmp(argv[1], "image")) return image(std::atoi(argv[2]));
    return 2;
}
