// plan.cu -- planned SpMM: one sparse matrix, many products.
//
// daspmm_spmm is stateless: every call recomputes the chunk boundaries of the
// balanced split (k_partition over rowPtr) before the gather, so a caller may
// change the matrix between calls.  A caller that multiplies the same matrix
// by many dense operands (an iterative solver, a GNN layer over one graph, a
// serving loop over a resident matrix) can instead create a plan: the
// boundaries, and the list of rows without nonzeros, are computed once into
// memory the plan owns, and each product is the worker-group window kernel,
// with no partition pass (and, where the matrix has rows without nonzeros, one
// small launch that clears them).  Between products nothing is reset: the
// split-row counters return to zero by themselves (the last piece of a row
// clears its counter), and each call counts its queue claims on from where the
// previous call's ended (a call makes exactly one claim per chunk group).
// Results are bit-identical to daspmm_spmm with the same configuration (same
// chunks, same order of summation).  Calls the planned form does not take
// (beta != 0, B or C off the window kernel's alignment, widths that are no
// multiple of 32) run the stateless path on the plan's workspace, and the next
// planned call first writes the boundaries again.
#include "internal.h"

#include <cuda_runtime.h>

#include <new>
#include <vector>

struct daspmm_plan_s {
    daspmm_config cfg;     // as the caller gave it
    daspmm::Resolved r;    // of operands aligned to 16 bytes
    int nr, nc, nnz, nv;
    const int *rowPtr, *colIdx;
    const float *values;
    void *ws = nullptr;
    size_t ws_bytes = 0;
    int *empty = nullptr;    // device: the rows without nonzeros
    int nempty = 0;
    bool fresh = false;      // the boundaries in the workspace are the plan's
    unsigned long long calls = 0;  // planned products since they were written
    int dev = 0;
};

namespace {

// Boundaries (k_partition, which also zeroes the queue heads and split-row
// counters) into the plan's workspace.
void refresh(daspmm_plan p, cudaStream_t st)
{
    daspmm::carve_and_partition(p->r, p->nr, p->nnz, p->nv, p->rowPtr, p->ws, p->ws_bytes, st);
    p->fresh = true;
    p->calls = 0;
}

// The rows without nonzeros, which the window kernel does not visit, from the
// row pointer (read once on the host).
daspmm_status list_empty_rows(daspmm_plan p, cudaStream_t st)
{
    std::vector<int> rp((size_t)p->nr + 1), list;
    cudaError_t e = cudaMemcpyAsync(rp.data(), p->rowPtr, sizeof(int) * rp.size(),
                                    cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return daspmm::cuda_fail(e);
    for (int r = 0; r < p->nr; ++r)
        if (rp[r] == rp[r + 1]) list.push_back(r);
    if (list.empty()) return DASPMM_OK;
    e = cudaMalloc(&p->empty, sizeof(int) * list.size());
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(p->empty, list.data(), sizeof(int) * list.size(),
                            cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return daspmm::cuda_fail(e);
    p->nempty = (int)list.size();
    return DASPMM_OK;
}

}  // namespace

extern "C" {

daspmm_status daspmm_plan_create(const daspmm_config *cfg, int nr, int nc, int nnz, int nv,
                                 const int *rowPtr, const int *colIdx, const float *values,
                                 void *stream, daspmm_plan *out)
{
    if (!out) return DASPMM_ERR_INVALID;
    *out = nullptr;
    daspmm_config c = cfg ? *cfg : daspmm_config{};
    if (!cfg) c.alg = DASPMM_ALG_CSR_BALANCED;
    if (c.alg != DASPMM_ALG_CSR_BALANCED) return DASPMM_ERR_UNSUPPORTED;
    if (nr < 0 || nc < 0 || nnz < 0 || nv < 1 || !rowPtr || (nnz > 0 && (!colIdx || !values)))
        return DASPMM_ERR_INVALID;
    daspmm::Resolved r;
    daspmm_status s = daspmm::resolve(&c, DASPMM_ROW_MAJOR, nr, nc, nnz, nv, nullptr, nullptr, &r);
    if (s != DASPMM_OK) return s;
    auto *p = new (std::nothrow) daspmm_plan_s();
    if (!p) return DASPMM_ERR_INVALID;
    p->cfg = c;
    p->r = r;
    p->nr = nr; p->nc = nc; p->nnz = nnz; p->nv = nv;
    p->rowPtr = rowPtr; p->colIdx = colIdx; p->values = values;
    cudaGetDevice(&p->dev);
    p->ws_bytes = daspmm::workspace_bytes(r, nv);
    cudaStream_t st = (cudaStream_t)stream;
    if (p->ws_bytes) {
        cudaError_t e = cudaMalloc(&p->ws, p->ws_bytes);
        if (e != cudaSuccess) {
            delete p;
            return daspmm::cuda_fail(e);
        }
    }
    if (r.pipe == 4 && nr > 0) {
        s = list_empty_rows(p, st);
        if (s == DASPMM_OK) {
            refresh(p, st);
            cudaError_t e = cudaStreamSynchronize(st);
            if (e != cudaSuccess) s = daspmm::cuda_fail(e);
        }
        if (s != DASPMM_OK) {
            cudaFree(p->ws);
            cudaFree(p->empty);
            delete p;
            return s;
        }
    }
    *out = p;
    return DASPMM_OK;
}

daspmm_status daspmm_plan_spmm(daspmm_plan p, const float *B, float *C, float beta, void *stream)
{
    if (!p) return DASPMM_ERR_INVALID;
    if (p->nr == 0) return DASPMM_OK;
    if (!B || !C) return DASPMM_ERR_INVALID;
    cudaStream_t st = (cudaStream_t)stream;
    if (beta == 0.0f && p->r.pipe == 4) {
        if (!p->fresh) refresh(p, st);
        if (daspmm::run_planned(p->r, p->nr, p->nc, p->nnz, p->nv, p->rowPtr, p->colIdx,
                                p->values, B, C, p->ws, p->ws_bytes, p->empty, p->nempty, p->calls, st)) {
            ++p->calls;
            cudaError_t e = cudaGetLastError();
            return e == cudaSuccess ? DASPMM_OK : daspmm::cuda_fail(e);
        }
    }
    // the stateless path on the plan's workspace, with the vectors that these addresses
    // allow (p->r's may be wider); it rewrites the boundaries and the queue heads, so the
    // next planned call refreshes them
    daspmm::Resolved r;
    const daspmm_status s = daspmm::resolve(&p->cfg, DASPMM_ROW_MAJOR, p->nr, p->nc, p->nnz, p->nv,
                                            B, C, &r);
    if (s != DASPMM_OK) return s;
    p->fresh = false;
    return daspmm::run_resolved(r, DASPMM_ROW_MAJOR, p->nr, p->nc, p->nnz, p->nv, p->rowPtr,
                                nullptr, p->colIdx, p->values, B, C, beta, p->ws, p->ws_bytes,
                                st);
}

daspmm_status daspmm_plan_config(daspmm_plan p, daspmm_config *out)
{
    if (!p || !out) return DASPMM_ERR_INVALID;
    *out = daspmm::to_config(p->r);
    return DASPMM_OK;
}

daspmm_status daspmm_plan_destroy(daspmm_plan p)
{
    if (!p) return DASPMM_OK;
    int cur = 0;
    cudaGetDevice(&cur);
    if (cur != p->dev) cudaSetDevice(p->dev);
    cudaError_t e = p->ws ? cudaFree(p->ws) : cudaSuccess;
    const cudaError_t e2 = p->empty ? cudaFree(p->empty) : cudaSuccess;
    if (e == cudaSuccess) e = e2;
    if (cur != p->dev) cudaSetDevice(cur);
    delete p;
    return e == cudaSuccess ? DASPMM_OK : daspmm::cuda_fail(e);
}

}  // extern "C"
