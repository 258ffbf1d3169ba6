// tc_host.hpp -- host-side error plumbing shared by the translation units.
#pragma once

#include <cstdio>
#include <string>
#include <vector>
#include <cuda_runtime.h>

#include "tc_internal.cuh"

namespace tc {

void set_last_error(const std::string& msg);

// Number of kernels this library has launched (all devices, since load).
void count_launch();

// Evaluate a CUDA runtime call; on failure record the message and return TC_ERR_CUDA (2).
#define TC_CU(call)                                                                        \
    do {                                                                                   \
        cudaError_t e_ = (call);                                                           \
        if (e_ != cudaSuccess) {                                                           \
            ::tc::set_last_error(std::string(#call) + ": " + cudaGetErrorString(e_));      \
            return 2;                                                                      \
        }                                                                                  \
    } while (0)

// Propagate a non-zero status.
#define TC_TRY(expr)                                                                       \
    do {                                                                                   \
        int s_ = (expr);                                                                   \
        if (s_ != 0) return s_;                                                            \
    } while (0)

// Device memory from the library's stream-ordered pool on the current device, usable in the
// order of the library's stream (capi.cu); freed memory stays in the pool for the next call.
// Records a message and returns TC_ERR_NOMEM (5) on failure.
int dev_alloc(void** p, size_t bytes);
void dev_free(void* p);

// The dynamic shared memory that a kernel may be launched with belongs to the kernel: several
// threads launch it, with their own numbers of bins, so it is only ever raised.
int allow_smem(const void* kernel, size_t bytes);
template <class R, class... P>
int allow_smem(R (*kernel)(P...), size_t bytes) { return allow_smem((const void*)kernel, bytes); }

template <class T>
int dalloc(T** p, size_t count)
{
    *p = nullptr;
    return dev_alloc((void**)p, (count == 0 ? 1 : count) * sizeof(T));
}

template <class T>
void dfree(T*& p)
{
    if (p) dev_free((void*)p);
    p = nullptr;
}

#ifdef __CUDACC__
// A kernel launched with launch_chained has its blocks set up as those of the kernel before
// end; in after_previous, its first statement, they wait until all of that kernel's writes are
// visible.  (The kernel before gives no earlier sign: blocks set up while it still runs go where it
// has left room, not evenly over the SMs.  With one, builds of 400,000 points took 2.26 ms
// instead of 2.12, without chaining 2.16, and k-means of 2M points 32.8 instead of 28.9 and 32.0.)
__device__ __forceinline__ void after_previous() { cudaGridDependencySynchronize(); }

template <class... P, class... A>
int launch_chained(void (*kernel)(P...), int blocks, int threads, size_t smem, cudaStream_t st,
                   A... args)
{
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    count_launch();
    TC_CU(cudaLaunchKernelEx(&cfg, kernel, P(args)...));
    return 0;
}
#endif

// Tree build (tree_build.cu).

struct TreeBuild {                  // what a build works on
    BuildParams BP;
    Points bufs[2];
    Cells C;
    TCell* tcells;
    int *d_tops, *d_ntop, *d_err;
    int mintop, maxtop;
    BuildScratch* S;
};
struct BuildRun {                   // how far a build has come
    int lev = 0, total = 0, batch = 0;
    bool whole = false;             // one block builds the whole tree
};
struct BuildRead {                  // what the host reads of a build
    static constexpr int FIRST = 1024;
    int2 left;                      // tasks and chunks of the level after the queued ones
    int nsmall;                     // cells for k_subtree
    int ntop;
    int2 tops[FIRST];               // (first point, id)
};
// The build in three parts, so that several can run side by side: each of the first two
// queues its kernels on st and copies (kind) what the next part reads into *to, which has to
// be there before that one is called.
int tree_begin(const TreeBuild& B, BuildRun& R, BuildRead* to, cudaMemcpyKind kind, cudaStream_t st);
int tree_subtrees(const TreeBuild& B, BuildRun& R, const BuildRead& read, BuildRead* to,
                  cudaMemcpyKind kind, cudaStream_t st);
int tree_tops(const TreeBuild& B, const BuildRead& read, cudaStream_t st, std::vector<int>& tops_out);
int field_center(const BuildParams& BP, Points P, BuildScratch& S, cudaStream_t st,
                 double out[4]);
void launch_prepare(int n, int coords, int dkind, const double* x, const double* y,
                    const double* z, const double* d1, const double* d2, const double* w,
                    const double* wpos, Points P, cudaStream_t st);
int tcgen05_selftest(const float* A, const float* B, float* C, int N, int K, cudaStream_t st);
void launch_validate_tree(int ncap, const Cells& C, const int* tops, int ntop, int* err,
                          cudaStream_t st);

}  // namespace tc
