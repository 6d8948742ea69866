// launch_single_cta.cu -- test hook for the tile pipeline's forward progress.
//
// The pipeline kernels (trtc_pipe.cuh) of 32-bit integers in grids of a given size.  A grid of one CTA
// holds the prefix CTA only, as when a long kernel on another stream leaves room for one.  And a kernel
// that keeps SMs busy for a bounded time.  Operators and keys are types of this file, so that these are instantiations of
// their own.
#include "trtc_launch.h"
#include "trtc_runtime.h"
#include "../device/trtc_pipe.cuh"

using namespace trtc_host;
using namespace trtc;

namespace {
struct IsOdd {
    template <class T> __device__ bool operator()(const T& x) const { return (x & 1) != 0; }
};
struct Same {
    template <class T> __device__ bool operator()(const T& a, const T& b) const { return a == b; }
};
struct Key {
    int v;
    __device__ bool operator==(const Key& o) const { return v == o.v; }
};
template <class F, class... A>
bool launch(F* kernel, unsigned ctas, unsigned threads, size_t smem, cudaStream_t s, A... args) {
    if (!TRTC_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem))) return false;
    kernel<<<ctas, threads, smem, s>>>(args...);
    count_launch();
    return TRTC_CUDA(cudaGetLastError());
}
__global__ void occupy_kernel(unsigned micros) {
    unsigned long long t0, t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    for (unsigned i = 0; i < (1u << 22); i++) {
        __nanosleep(1000);
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        if (t - t0 > (unsigned long long)micros * 1000ull) return;
    }
}
template <class T> VectorView<T> view(T* p, size_t n) {
    VectorView<T> v;
    v._data = p;
    v._size = n;
    return v;
}
}  // namespace

extern "C" int trtc_test_pipe_few_ctas(int what, unsigned ctas, int* keys, int* in, int* out, int* out2,
                                       unsigned long long n, unsigned long long* count, void* stream) {
    if (!ensure_device()) return -1;
    const cudaStream_t s = (cudaStream_t)stream;
    typedef CpipeShape<int> CS;
    typedef SpipeShape<Key, int> SS;
    constexpr int RI = 20, RS = 3, RC = 6000;  // (reduce_by_key: tiles of 5120, a ring of 6000 results)
    typedef RbkSmem<int, int, int, RI, RS, RC> RSM;
    const size_t tile = what <= 1 ? (size_t)CS::TILE : what <= 3 ? (size_t)SS::TILE : (size_t)RSM::TILE;
    const size_t tiles = (n + tile - 1) / tile;
    uint32_t e8 = 0;
    LookbackWs* w = n ? lookback_ws(s, tiles, sizeof(int), &e8) : nullptr;
    if (!w || ctas < 1 || ctas > tiles + 1) { set_error("pipeline test: bad size"); return -1; }
    LookbackState st;
    st.flags = w->flags;
    st.agg = w->agg;
    st.incl = w->incl;
    st.packed = w->packed;
    st.tile_ctr = w->tile_ctr;
    st.epoch8 = e8;
    st.err = device_error_word();
    st.result = w->result;
    LookbackState st2 = st;
    st2.packed = w->packed2;
    st2.flags = w->flags2;
    const uint32_t nt = (uint32_t)tiles;
    const VectorView<int> kv = view(keys, n), iv = view(in, n), ov = view(out, n), ov2 = view(out2, n);
    bool ok = false;
    if (what == 0)  // odd elements to out, the others to out2
        ok = launch(compact_pipe_kernel<CM_PRED, true, int, IsOdd, Nothing, VectorView<int>, VectorView<int>, CS::G, CS::ITEMS, CS::S, CS::RING>,
                    ctas, PipeShape<CS::G>::THREADS, CS::SMEM, s, in, IsOdd(), Nothing(), ov, ov2, (size_t)n, nt, st);
    else if (what == 1)  // unique
        ok = launch(compact_pipe_kernel<CM_UNIQUE_PRED, false, int, Same, Nothing, VectorView<int>, Nothing, CS::G, CS::ITEMS, CS::S, CS::RING>,
                    ctas, PipeShape<CS::G>::THREADS, CS::SMEM, s, in, Same(), Nothing(), ov, Nothing(), (size_t)n, nt, st);
    else if (what == 2)  // scan by key, inclusive, and exclusive behind 5
        ok = launch(scan_by_key_pipe_kernel<Key, int, 0>, ctas, PipeShape<SS::G>::THREADS, SS::SMEM, s, (Key*)keys, in, out, (size_t)n, nt, 0, st, st2);
    else if (what == 3)
        ok = launch(scan_by_key_pipe_kernel<Key, int, 1>, ctas, PipeShape<SS::G>::THREADS, SS::SMEM, s, (Key*)keys, in, out, (size_t)n, nt, 5, st, st2);
    else if (what == 4)  // keys to out2, sums to out
        ok = launch(rbk_pipe_kernel<VectorView<int>, VectorView<int>, VectorView<int>, VectorView<int>, int, Same, ::Plus, 2, RI, RS, RC>,
                    ctas, PipeShape<2>::THREADS, RSM::BYTES, s, kv, iv, ov2, ov, (size_t)n, nt, Same(), ::Plus(), st, st2);
    if (!ok || !TRTC_CUDA(cudaMemcpyAsync(count, w->result, 8, cudaMemcpyDeviceToHost, s))) return -1;
    return check_device_errors(s, "pipeline test") ? 0 : -1;
}

extern "C" int trtc_test_occupy(unsigned ctas, unsigned smem, unsigned micros, void* stream) {
    if (!ensure_device() || micros > 1000000u) return -1;
    return launch(occupy_kernel, ctas, 32u, smem, (cudaStream_t)stream, micros) ? 0 : -1;
}
