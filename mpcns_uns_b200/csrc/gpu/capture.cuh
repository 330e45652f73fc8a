#pragma once
#include <cuda_runtime_api.h>

namespace mhd
{
// The launches of enqueue() on stream s as an executable graph, or null where the stream cannot be captured, a launch
// inside fails (enqueue throws) or the graph cannot be instantiated.  Either way the capture has ended and no error is
// left behind, so that the caller can launch directly instead.
template <class F> cudaGraphExec_t capture_graph(cudaStream_t s, F &&enqueue)
{
    cudaGraphExec_t exec = nullptr;
    if (cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) == cudaSuccess)
    {
        bool ok = true;
        try
        {
            enqueue();
        }
        catch (...)
        {
            ok = false;
        }
        cudaGraph_t graph = nullptr;
        ok = cudaStreamEndCapture(s, &graph) == cudaSuccess && graph && ok;
        if (ok && cudaGraphInstantiate(&exec, graph, 0) != cudaSuccess) exec = nullptr;
        if (graph) cudaGraphDestroy(graph);
    }
    if (!exec) cudaGetLastError();
    return exec;
}
} // namespace mhd
