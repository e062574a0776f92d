// gdp_sequence.h -- device work in order, issued to a stream or added to a graph
// as a chain of nodes.
//
// Graphs are built from nodes and not captured from a stream. While a stream is
// captured, another thread that synchronises the device (destroying a context
// does, and any other code of the process may) ends the capture with an error,
// and the driver crashed when the graph of such a capture was destroyed.
#pragma once

#include <cuda_runtime.h>

namespace gdp {

class Sequence {
public:
    explicit Sequence(cudaStream_t s) : stream_(s) {}
    explicit Sequence(cudaGraph_t g) : graph_(g) {}

    cudaError_t kernel(const void *f, dim3 grid, dim3 block, void **args, size_t smem, bool cooperative = false) {
        if (!graph_)
            return cooperative ? cudaLaunchCooperativeKernel(f, grid, block, args, smem, stream_)
                               : cudaLaunchKernel(f, grid, block, args, smem, stream_);
        cudaKernelNodeParams p = {};
        p.func = const_cast<void *>(f);
        p.gridDim = grid;
        p.blockDim = block;
        p.sharedMemBytes = (unsigned)smem;
        p.kernelParams = args;  // copied
        cudaGraphNode_t node;
        cudaError_t e = cudaGraphAddKernelNode(&node, graph_, deps(), n_deps(), &p);
        if (e != cudaSuccess) return e;
        last_ = node;
        if (!cooperative) return cudaSuccess;
        cudaKernelNodeAttrValue v = {};
        v.cooperative = 1;
        return cudaGraphKernelNodeSetAttribute(node, cudaKernelNodeAttributeCooperative, &v);
    }
    cudaError_t copy(void *dst, const void *src, size_t bytes, cudaMemcpyKind kind) {
        if (!bytes) return cudaSuccess;
        if (!graph_) return cudaMemcpyAsync(dst, src, bytes, kind, stream_);
        cudaGraphNode_t node;
        const cudaError_t e = cudaGraphAddMemcpyNode1D(&node, graph_, deps(), n_deps(), dst, src, bytes, kind);
        if (e == cudaSuccess) last_ = node;
        return e;
    }
    cudaError_t clear(void *dst, size_t bytes) {
        if (!graph_) return cudaMemsetAsync(dst, 0, bytes, stream_);
        cudaMemsetParams p = {};
        p.dst = dst;
        p.elementSize = 1;
        p.width = bytes;
        p.height = 1;
        cudaGraphNode_t node;
        const cudaError_t e = cudaGraphAddMemsetNode(&node, graph_, deps(), n_deps(), &p);
        if (e == cudaSuccess) last_ = node;
        return e;
    }
    cudaError_t record(cudaEvent_t ev) {
        if (!graph_) return cudaEventRecord(ev, stream_);
        cudaGraphNode_t node;
        const cudaError_t e = cudaGraphAddEventRecordNode(&node, graph_, deps(), n_deps(), ev);
        if (e == cudaSuccess) last_ = node;
        return e;
    }

private:
    const cudaGraphNode_t *deps() const { return last_ ? &last_ : nullptr; }
    size_t n_deps() const { return last_ ? 1 : 0; }

    cudaStream_t stream_ = nullptr;
    cudaGraph_t graph_ = nullptr;
    cudaGraphNode_t last_ = nullptr;
};

}  // namespace gdp
