// Process-wide runtime (stream, reduction scratch) and vector helpers.
// Mirrors the reference's globals stream_interior / workspace
// (src/utils.hpp:38-45, created in src/init.cpp:200-230) and the vector
// helpers of src/Vector.hpp / src/CGData.hpp.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>

#include "hpcg_b200.h"
#include "internal.hpp"

namespace hpcg_b200 {

static Runtime g_rt;

Runtime& rt() { return g_rt; }

void throw_last(int code) { throw Error(code, hpcgb200_last_error()); }

void check_cuda(cudaError_t e, const char* what)
{
    if(e != cudaSuccess)
    {
        char buf[256];
        snprintf(buf, sizeof(buf), "CUDA error %d (%s) in %s", (int)e, cudaGetErrorString(e), what);
        throw Error(HPCGB200_ERR_CUDA, buf);
    }
}

namespace {

struct Chunk
{
    size_t bytes, used;
    int live;   // arrays not yet freed
    bool open;  // a scope may still place arrays in it
};

std::mutex g_chunks_mutex;
std::map<char*, Chunk> g_chunks;  // by base address
thread_local ArenaScope* t_arena = nullptr;

// Called with the mutex held: the chunk no scope fills any more.
char* close_chunk(char* base)
{
    if(!base) return nullptr;
    const auto it = g_chunks.find(base);
    it->second.open = false;
    if(it->second.live > 0) return nullptr;
    g_chunks.erase(it);
    return base;  // empty: the caller frees it
}

}  // namespace

ArenaScope::ArenaScope(long long rows) : outer_(t_arena)
{
    // kept per level-0 row of a problem whose vectors go into chunks: about 140 B on level 0 and
    // 50 for the coarse levels; of a larger one only the coarse levels' arrays do
    const size_t kept = rows * 8 < (long long)kArenaLargest ? (size_t)rows * 190 : 64u << 20;
    next_[kKept] = std::min(kArenaChunk, kept + (1u << 20));
    next_[kTemporary] = std::min<size_t>(kArenaChunk / 4, (size_t)rows * 48 + (1u << 20));
    t_arena = this;
}

ArenaScope::~ArenaScope()
{
    t_arena = outer_;
    for(char* base : chunk_)
    {
        char* empty;
        {
            std::lock_guard<std::mutex> lock(g_chunks_mutex);
            empty = close_chunk(base);
        }
        if(empty) cudaFree(empty);
    }
}

void* ArenaScope::take(size_t bytes, AllocKind kind)
{
    bytes = (bytes + 255) & ~(size_t)255;
    char* empty = nullptr;
    char* p = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_chunks_mutex);
        Chunk* c = chunk_[kind] ? &g_chunks[chunk_[kind]] : nullptr;
        if(!c || c->used + bytes > c->bytes)
        {
            void* base = nullptr;
            const size_t size = std::max(next_[kind], bytes);
            if(cudaMalloc(&base, size) != cudaSuccess)
            {
                cudaGetLastError();
                return nullptr;
            }
            empty = close_chunk(chunk_[kind]);
            chunk_[kind] = static_cast<char*>(base);
            c = &(g_chunks[chunk_[kind]] = Chunk{size, 0, 0, true});
            next_[kind] = std::max<size_t>(2u << 20, next_[kind] / 4);
        }
        p = chunk_[kind] + c->used;
        c->used += bytes;
        ++c->live;
    }
    if(empty) cudaFree(empty);
    return p;
}

void* device_alloc(size_t bytes, AllocKind kind)
{
    if(t_arena && bytes < kArenaLargest)
        if(void* p = t_arena->take(bytes, kind)) return p;
    void* p = nullptr;
    HB_HOST_CUDA(cudaMalloc(&p, bytes));
    return p;
}

void dfree(void* p)
{
    if(!p) return;
    {
        std::lock_guard<std::mutex> lock(g_chunks_mutex);
        auto it = g_chunks.upper_bound(static_cast<char*>(p));
        if(it != g_chunks.begin())
        {
            --it;
            Chunk& c = it->second;
            if(static_cast<char*>(p) < it->first + c.bytes)
            {
                if(--c.live > 0) return;
                if(c.open)
                {
                    c.used = 0;  // set-up work is stream ordered: the next arrays may take its place
                    return;
                }
                p = it->first;
                g_chunks.erase(it);
            }
        }
    }
    cudaFree(p);
}

void ensure_runtime()
{
    if(g_rt.initialized) return;
    int n = 0;
    if(cudaGetDeviceCount(&n) != cudaSuccess || n == 0)
        throw Error(HPCGB200_ERR_NO_DEVICE, "no CUDA device visible (libhpcgb200 has no CPU fallback)");
    HB_HOST_CUDA(cudaGetDevice(&g_rt.device));
    HB_HOST_CUDA(cudaStreamCreateWithFlags(&g_rt.stream, cudaStreamNonBlocking));
    void* p = nullptr;
    HB_HOST_CUDA(cudaMalloc(&p, sizeof(hb::ReduceScratch)));
    HB_HOST_CUDA(cudaMemset(p, 0, sizeof(hb::ReduceScratch)));
    g_rt.ws = static_cast<hb::ReduceScratch*>(p);
    HB_HOST_CUDA(cudaMalloc(&g_rt.d_scalar, 16 * sizeof(double)));
    HB_HOST_CUDA(cudaMallocHost(&g_rt.h_scalar, 16 * sizeof(double)));
    HB_HOST_CUDA(cudaMalloc(&g_rt.ref_status, sizeof(int)));
    HB_HOST_CUDA(cudaMemset(g_rt.ref_status, 0, sizeof(int)));
    g_rt.initialized = true;
}

}  // namespace hpcg_b200

using namespace hpcg_b200;

int HPCG_B200_Init(int device)
{
    try
    {
        if(g_rt.initialized) return 0;
        if(device >= 0) HB_HOST_CUDA(cudaSetDevice(device));
        ensure_runtime();
        return 0;
    }
    catch(const Error& e)
    {
        return report(e);
    }
}

extern "C" int hpcgb200_init(int device)
{
    try
    {
        if(g_rt.initialized)
        {
            if(device >= 0 && device != g_rt.device)
                return hb::record_error(HPCGB200_ERR_ARG, "the library runtime is bound to device %d already",
                                        g_rt.device);
            return 0;
        }
        int n = 0;
        if(cudaGetDeviceCount(&n) != cudaSuccess || n == 0)
            return hb::record_error(HPCGB200_ERR_NO_DEVICE, "no CUDA device visible");
        if(device >= n) return hb::record_error(HPCGB200_ERR_ARG, "device %d out of range (%d visible)", device, n);
        if(device >= 0) HB_HOST_CUDA(cudaSetDevice(device));
        ensure_runtime();
        return 0;
    }
    catch(const Error& e)
    {
        return report(e);
    }
}

cudaStream_t HPCG_B200_Stream()
{
    ensure_runtime();
    return g_rt.stream;
}

void HPCG_B200_SetStream(cudaStream_t s)
{
    ensure_runtime();
    g_rt.stream = s;
}

int HPCG_B200_Finalize()
{
    if(!g_rt.initialized) return 0;
    cudaStreamSynchronize(g_rt.stream);
    dfree(g_rt.ws);
    dfree(g_rt.d_scalar);
    dfree(g_rt.ref_status);
    if(g_rt.h_scalar) cudaFreeHost(g_rt.h_scalar);
    g_rt = Runtime{};
    return 0;
}

void CudaInitializeVector(Vector& v, local_int_t localLength)
{
    ensure_runtime();
    v.localLength = localLength;
    v.optimizationData = nullptr;
    v.d_values = dalloc<double>(localLength);
}

void CudaDeleteVector(Vector& v)
{
    dfree(v.d_values);
    v.d_values = nullptr;
    if(v.values) delete[] v.values;
    v.values = nullptr;
    v.localLength = 0;
}

void CudaZeroVector(Vector& v)
{
    ensure_runtime();
    HB_HOST_CUDA(cudaMemsetAsync(v.d_values, 0, sizeof(double) * v.localLength, g_rt.stream));
}

void CudaCopyVector(const Vector& v, Vector& w)
{
    ensure_runtime();
    HB_HOST_CUDA(cudaMemcpyAsync(w.d_values, v.d_values, sizeof(double) * v.localLength, cudaMemcpyDeviceToDevice,
                                 g_rt.stream));
}

void CudaFillRandomVector(Vector& v)
{
    ensure_runtime();
    std::vector<double> h(v.localLength);
    for(local_int_t i = 0; i < v.localLength; ++i) h[i] = rand() / (double)(RAND_MAX) + 1.0;
    HB_HOST_CUDA(cudaMemcpyAsync(v.d_values, h.data(), sizeof(double) * v.localLength, cudaMemcpyHostToDevice,
                                 g_rt.stream));
    HB_HOST_CUDA(cudaStreamSynchronize(g_rt.stream));
}

void CudaInitializeSparseCGData(SparseMatrix& A, CGData& data)
{
    CudaInitializeVector(data.r, A.localNumberOfRows);
    CudaInitializeVector(data.z, A.localNumberOfColumns);
    CudaInitializeVector(data.p, A.localNumberOfColumns);
    CudaInitializeVector(data.Ap, A.localNumberOfRows);
}

void CudaDeleteCGData(CGData& data)
{
    CudaDeleteVector(data.r);
    CudaDeleteVector(data.z);
    CudaDeleteVector(data.p);
    CudaDeleteVector(data.Ap);
}

void CudaCopyMatrixDiagonal(const SparseMatrix& A, Vector& diagonal)
{
    ensure_runtime();
    check(hpcgb200_copy_diagonal(A.localNumberOfRows, A.ell_col_ind, A.ell_val, diagonal.d_values, g_rt.stream));
}

void CudaReplaceMatrixDiagonal(SparseMatrix& A, const Vector& diagonal)
{
    ensure_runtime();
    LevelOpt* o = opt(A);
    check(hpcgb200_replace_diagonal(A.localNumberOfRows, diagonal.d_values, A.ell_col_ind, A.ell_val, A.inv_diag,
                                    o ? o->diag : nullptr, g_rt.stream));
    if(o && o->diag32) check(hb::launch_diag32(A.localNumberOfRows, o->diag, o->diag32, o->inv_diag32, g_rt.stream));
}

void ExchangeHalo(const SparseMatrix&, Vector&)
{
    // One rank: no neighbours, nothing to exchange (src/ExchangeHalo.cpp:67).
}
