// Tables built on the host for a kernel to read.  An asynchronous copy from
// pageable memory may read it after the call that queued it has returned (a GPU
// that addresses the host's pages need not stage it first), so a table belongs
// to its copy: copy() takes it over, and the destructor frees the tables
// only once the stream has passed the last of their copies, also when an error
// unwinds the caller.
#pragma once
#include <cuda_runtime.h>

#include <memory>
#include <utility>
#include <vector>

namespace rsg {

class HostTables {
  public:
    explicit HostTables(cudaStream_t st) : st(st) {}
    HostTables(const HostTables &) = delete;
    HostTables &operator=(const HostTables &) = delete;
    ~HostTables() {
        if (!last) return;
        cudaEventSynchronize(last);
        cudaEventDestroy(last);
    }
    template <class T>
    cudaError_t copy(T *dst, std::vector<T> &&table) {
        if (table.empty()) return cudaSuccess;
        if (!last) {
            cudaError_t e = cudaEventCreateWithFlags(&last, cudaEventDisableTiming);
            if (e != cudaSuccess) return e;
        }
        auto kept = std::make_shared<std::vector<T>>(std::move(table));
        tables.push_back(kept);
        cudaError_t e = cudaMemcpyAsync(dst, kept->data(), sizeof(T) * kept->size(),
                                        cudaMemcpyHostToDevice, st);
        const cudaError_t r = cudaEventRecord(last, st);
        if (r != cudaSuccess) cudaStreamSynchronize(st);  // no mark to wait for later
        return e != cudaSuccess ? e : r;
    }

  private:
    cudaStream_t st;
    cudaEvent_t last = nullptr;  // recorded after every copy
    std::vector<std::shared_ptr<void>> tables;
};

}  // namespace rsg
