// op2g_vec.cu -- pointwise linear algebra of Dats (pyop2/types/dat.py:343-574
// runs each operation as a generated par_loop; the signatures are few and
// fixed, so here they are kernels of the library): r = a op b, r = a op s,
// r = -a and the inner product, on the owned values as flat arrays.
//
// All of them are bound by memory: 16-byte loads and stores where the arrays
// are aligned (any Dat's own allocation is), two packs in flight per thread.
// What they replace cost 30-170 us of host time per call (a loop built, and a
// Global uploaded and read back for every scalar and inner product) for a few
// microseconds of device time on a solver's vectors.  Per call on the GB300
// host, 274,625 doubles: a += b 30 -> 5 us, a * b 86 -> 22, a * s 170 -> 22,
// inner product 171 -> 22; two matrix-free CG iterations 3.12 -> 1.29 ms.
#include <cuda_runtime.h>

#include <cstdint>

#include "op2g_internal.h"

namespace {

#define CK(call)                                                   \
    do {                                                           \
        cudaError_t e_ = (call);                                   \
        if (e_ != cudaSuccess) return op2g::cuda_fail(e_, #call); \
    } while (0)

constexpr int VEC_T = 256;

int sms_of_current() {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 1;
}

// The C expression `a op b` of the element type.
template <class T, int OP>
__device__ __forceinline__ T apply(T a, T b) {
    if constexpr (OP == OP2G_VEC_ADD) return a + b;
    else if constexpr (OP == OP2G_VEC_SUB) return a - b;
    else if constexpr (OP == OP2G_VEC_MUL) return a * b;
    else if constexpr (OP == OP2G_VEC_DIV) return a / b;
    else return -a;
}

template <class T, int V>
struct alignas(V * sizeof(T)) Pack {
    T v[V];
};

// out[i] = a[i] op b[i], or op s when b is NULL.  out may be a or b: an
// element's inputs are read before it is written, by the same thread.
template <class T, int OP, int V>
__global__ void __launch_bounds__(VEC_T)
    k_vec(long long n, const T *a, const T *b, T s, T *out) {
    using P = Pack<T, V>;
    const long long np = n / V, stride = (long long)gridDim.x * VEC_T;
    const long long t = (long long)blockIdx.x * VEC_T + threadIdx.x;
    P sp;
#pragma unroll
    for (int k = 0; k < V; ++k) sp.v[k] = s;
    for (long long i = t; i < np; i += 2 * stride) {
        const long long j = i + stride;
        const bool two = j < np;
        P x0 = ((const P *)a)[i], y0 = sp, x1 = sp, y1 = sp;
        if (b) y0 = ((const P *)b)[i];
        if (two) {
            x1 = ((const P *)a)[j];
            if (b) y1 = ((const P *)b)[j];
        }
#pragma unroll
        for (int k = 0; k < V; ++k) x0.v[k] = apply<T, OP>(x0.v[k], y0.v[k]);
        ((P *)out)[i] = x0;
        if (two) {
#pragma unroll
            for (int k = 0; k < V; ++k) x1.v[k] = apply<T, OP>(x1.v[k], y1.v[k]);
            ((P *)out)[j] = x1;
        }
    }
    if (V > 1 && t < n - np * V) {   // the last few elements
        const long long i = np * V + t;
        out[i] = apply<T, OP>(a[i], b ? b[i] : s);
    }
}

template <class T, int OP>
op2g_status vec_launch(int64_t n, const void *a, const void *b, const void *s, void *out,
                       cudaStream_t st) {
    constexpr int V = 16 / sizeof(T);
    const T sv = s ? *(const T *)s : (T)0;
    const bool vec = (uintptr_t)a % 16 == 0 && (uintptr_t)b % 16 == 0 && (uintptr_t)out % 16 == 0;
    const int64_t items = vec ? n / V + 1 : n;
    int64_t g = (items + 2 * VEC_T - 1) / (2 * VEC_T);
    const int64_t small = (items + VEC_T - 1) / VEC_T, sms = sms_of_current();
    if (g < sms) g = small < sms ? small : sms;   // short vectors: a pack per thread first
    if (g > sms * 16) g = sms * 16;
    if (vec)
        k_vec<T, OP, V><<<(unsigned)g, VEC_T, 0, st>>>(n, (const T *)a, (const T *)b, sv, (T *)out);
    else
        k_vec<T, OP, 1><<<(unsigned)g, VEC_T, 0, st>>>(n, (const T *)a, (const T *)b, sv, (T *)out);
    CK(cudaGetLastError());
    return OP2G_OK;
}

template <class T>
op2g_status vec_op(int op, int64_t n, const void *a, const void *b, const void *s, void *out,
                   cudaStream_t st) {
    switch (op) {
        case OP2G_VEC_ADD: return vec_launch<T, OP2G_VEC_ADD>(n, a, b, s, out, st);
        case OP2G_VEC_SUB: return vec_launch<T, OP2G_VEC_SUB>(n, a, b, s, out, st);
        case OP2G_VEC_MUL: return vec_launch<T, OP2G_VEC_MUL>(n, a, b, s, out, st);
        case OP2G_VEC_DIV: return vec_launch<T, OP2G_VEC_DIV>(n, a, b, s, out, st);
        case OP2G_VEC_NEG: return vec_launch<T, OP2G_VEC_NEG>(n, a, b, s, out, st);
    }
    return op2g::fail(OP2G_ERR_INVALID, "unknown vector operation");
}

// ---------------------------------------------------------- inner product
constexpr int DOT_T = 256, DOT_CTAS_PER_SM = 4;

template <class T>
__device__ __forceinline__ T cta_sum(T v) {
    __shared__ T w[DOT_T / 32];
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
    if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = v;
    __syncthreads();
    T t = (T)0;
    if (threadIdx.x == 0)
        for (int k = 0; k < DOT_T / 32; ++k) t += w[k];
    return t;
}

// *out = sum a[i] b[i], accumulated in the element type: V partial sums per
// thread, then a tree per CTA, and the CTA that finishes last sums the CTAs'
// results (a fixed order, so repeated calls give the same bits).  The ticket
// is zero between calls.
template <class T, int V>
__global__ void __launch_bounds__(DOT_T)
    k_dot(long long n, const T *__restrict__ a, const T *__restrict__ b, T *part,
          unsigned *ticket, T *out) {
    using P = Pack<T, V>;
    const long long np = n / V, stride = (long long)gridDim.x * DOT_T;
    const long long t = (long long)blockIdx.x * DOT_T + threadIdx.x;
    T acc[V];
#pragma unroll
    for (int k = 0; k < V; ++k) acc[k] = (T)0;
    const bool same = a == b;
#pragma unroll 4
    for (long long i = t; i < np; i += stride) {
        const P x = ((const P *)a)[i];
        P y = x;
        if (!same) y = ((const P *)b)[i];
#pragma unroll
        for (int k = 0; k < V; ++k) acc[k] += x.v[k] * y.v[k];
    }
    T s = acc[0];
#pragma unroll
    for (int k = 1; k < V; ++k) s += acc[k];
    if (V > 1 && t < n - np * V) s += a[np * V + t] * b[np * V + t];
    s = cta_sum(s);
    __shared__ bool last;
    if (threadIdx.x == 0) {
        part[blockIdx.x] = s;
        __threadfence();
        last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    s = (T)0;
    for (unsigned i = threadIdx.x; i < gridDim.x; i += DOT_T) s += __ldcg(part + i);
    s = cta_sum(s);
    if (threadIdx.x == 0) {
        *out = s;
        *ticket = 0u;
    }
}

// What a calling thread keeps: 64 bytes of page-locked host memory for the
// result and, for the device it last used, the CTAs' results and the ticket.
// A call waits for its stream, so the next call of the thread finds them free.
struct DotState {
    void *host = nullptr, *dev = nullptr;
    int device = -1, ctas = 0;
    void drop() {
        if (dev) {
            int now = 0;
            cudaGetDevice(&now);
            cudaSetDevice(device);
            cudaFree(dev);
            cudaSetDevice(now);
        }
        dev = nullptr;
        device = -1;
    }
    ~DotState() {
        drop();
        if (host) cudaFreeHost(host);
    }
};

template <class T>
op2g_status dot(int64_t n, const void *a, const void *b, void *result, cudaStream_t st) {
    constexpr int V = 16 / sizeof(T);
    static thread_local DotState S;
    int dev = 0;
    CK(cudaGetDevice(&dev));
    if (!S.host) CK(cudaHostAlloc(&S.host, 64, cudaHostAllocPortable | cudaHostAllocMapped));
    if (S.device != dev) {
        S.drop();
        S.ctas = sms_of_current() * DOT_CTAS_PER_SM;
        CK(cudaMalloc(&S.dev, 64 + 8 * (size_t)S.ctas));
        S.device = dev;
        CK(cudaMemset(S.dev, 0, 64));
    }
    unsigned *ticket = (unsigned *)S.dev;
    T *part = (T *)((char *)S.dev + 64);
    const bool vec = (uintptr_t)a % 16 == 0 && (uintptr_t)b % 16 == 0;
    const int64_t items = vec ? n / V + 1 : n;
    int64_t g = (items + DOT_T - 1) / DOT_T;
    if (g > S.ctas) g = S.ctas;
    if (vec)
        k_dot<T, V><<<(unsigned)g, DOT_T, 0, st>>>(n, (const T *)a, (const T *)b, part, ticket,
                                                   (T *)S.host);
    else
        k_dot<T, 1><<<(unsigned)g, DOT_T, 0, st>>>(n, (const T *)a, (const T *)b, part, ticket,
                                                   (T *)S.host);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
        S.drop();   // the ticket may not be zero
        return op2g::cuda_fail(e, "inner product");
    }
    *(T *)result = *(volatile T *)S.host;
    return OP2G_OK;
}

}  // namespace

extern "C" {

op2g_status op2g_vec_op(int32_t op, int32_t dtype, int64_t n, const void *a, const void *b,
                        const void *scalar, void *out, void *stream) {
    if (n < 0 || (n > 0 && (!a || !out || (op != OP2G_VEC_NEG && !b == !scalar))))
        return op2g::fail(OP2G_ERR_INVALID, "op2g_vec_op needs a, out and one of b and scalar");
    if (n == 0) return OP2G_OK;
    cudaStream_t st = (cudaStream_t)stream;
    switch (dtype) {
        case OP2G_F64: return vec_op<double>(op, n, a, b, scalar, out, st);
        case OP2G_F32: return vec_op<float>(op, n, a, b, scalar, out, st);
        case OP2G_I32: return vec_op<int32_t>(op, n, a, b, scalar, out, st);
        case OP2G_U32: return vec_op<uint32_t>(op, n, a, b, scalar, out, st);
        case OP2G_I64: return vec_op<long long>(op, n, a, b, scalar, out, st);
        case OP2G_U64: return vec_op<unsigned long long>(op, n, a, b, scalar, out, st);
    }
    return op2g::fail(OP2G_ERR_UNSUPPORTED, "vector operations take 32- and 64-bit types");
}

op2g_status op2g_vec_dot(int32_t dtype, int64_t n, const void *a, const void *b, void *result,
                         void *stream) {
    if (n < 0 || !result || (n > 0 && (!a || !b)))
        return op2g::fail(OP2G_ERR_INVALID, "NULL argument");
    cudaStream_t st = (cudaStream_t)stream;
    const bool wide = dtype == OP2G_F64 || dtype == OP2G_I64 || dtype == OP2G_U64;
    if (n == 0 && (wide || dtype == OP2G_F32 || dtype == OP2G_I32 || dtype == OP2G_U32)) {
        if (wide) *(int64_t *)result = 0;
        else *(int32_t *)result = 0;
        return OP2G_OK;
    }
    switch (dtype) {
        case OP2G_F64: return dot<double>(n, a, b, result, st);
        case OP2G_F32: return dot<float>(n, a, b, result, st);
        // sums modulo 2^32 and 2^64 do not depend on the sign
        case OP2G_I32:
        case OP2G_U32: return dot<uint32_t>(n, a, b, result, st);
        case OP2G_I64:
        case OP2G_U64: return dot<unsigned long long>(n, a, b, result, st);
    }
    return op2g::fail(OP2G_ERR_UNSUPPORTED, "inner products take 32- and 64-bit types");
}

}  // extern "C"
