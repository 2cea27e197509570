// The training step's buffers when an allocation fails, with the allocator of the CUDA runtime replaced: no GPU needed.
#include "mlp.cuh"
#include <cstdio>
#include <cstdlib>
#include <map>

static std::map<void*, size_t> live;
static int fail_at = -1, calls = 0;

extern "C" cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) {
    if (calls++ == fail_at) return cudaErrorMemoryAllocation;
    *p = malloc(1);
    live[*p] = n;
    return cudaSuccess;
}
extern "C" cudaError_t cudaFreeAsync(void* p, cudaStream_t) {
    live.erase(p);
    free(p);
    return cudaSuccess;
}

namespace vsdmo {
cudaMemPool_t device_pool() { return nullptr; }
namespace mlp {
int wgrad_parts(int B) { return std::min(MAX_PARTS, B / 128); }
}
}  // namespace vsdmo

using namespace vsdmo;

static size_t bytes(const void* p) { return p ? live.at(const_cast<void*>(p)) : 0; }

int main() {
    for (int f = 0; f < 5; ++f) {
        mlp::TrainBuffers w;
        w.ensure(256, nullptr);
        calls = 0;
        fail_at = f;
        bool thrown = false;
        try {
            w.ensure(16384, nullptr);
        } catch (const Error&) {
            thrown = true;
        }
        fail_at = -1;
        if (!thrown) return 1;
        // a smaller batch than the one that failed: every buffer has to be there for it
        w.ensure(8192, nullptr);
        const size_t rows = 8192, parts = 64;
        if (bytes(w.part.p) < parts * mlp::TRAIN_PART * 4 || bytes(w.ws.p) < rows / 32 * (3 * mlp::HID + mlp::OUTP) * 4 ||
            bytes(w.loss_rows.p) < rows * 4 || bytes(w.loss.p) < 4 || bytes(w.idx.p) < 2 * rows * 4) {
            printf("allocation %d failed: buffers too small afterwards\n", f);
            return 2;
        }
    }
    DBuf<int> b(4, nullptr);
    calls = 0;
    fail_at = 0;
    try { b.alloc(8, nullptr); } catch (const Error&) {}
    if (b.p || b.n) return 3;
    return 0;
}
