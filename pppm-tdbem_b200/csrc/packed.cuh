// What the step (step.cu) and its transpose (adjoint.cu) share on the device: dependent launches, the
// (single, double) x (Neumann, Dirichlet) arithmetic on register pairs, and warp sums of several
// values.
#pragma once
#include "common.cuh"

namespace pb
{

namespace
{

// Programmatic dependent launch along a chain of kernels (the step graph's main branch:
// corrected-cell stencil -> finish -> near -> next stencil; the reverse step's kernels): the dependent grid is scheduled while its predecessor's last
// blocks drain, and waits here, before its first read, until the predecessor has completed and
// its writes are visible.  Launched without the attribute, the wait returns at once.
__device__ inline void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... KArgs, typename... Args>
void launch_dependent(void (*kern)(KArgs...), dim3 grid, int block, cudaStream_t s, Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kern, ((KArgs)args)...);
}

constexpr unsigned kFull = 0xffffffffu;

template <typename T, int N>
struct alignas(16) Vec
{
    T v[N];
};

// A pair of floats in one 64-bit register pair, the operand of the packed instructions (kept packed
// throughout: taken apart and put together again it costs a move per half)
struct F32x2
{
    unsigned long long v;
};

template <typename R>
struct WRec;
template <>
struct WRec<float>
{
    using T = __half2;
    using W4 = Vec<__half2, 4>;
    using P = F32x2;
};
template <>
struct WRec<double>
{
    using T = double2;
    using W4 = Vec<double2, 4>;
    using P = double2;
};

__device__ inline F32x2 make_pair2(float x, float y)
{
    F32x2 p;
    asm("mov.b64 %0, {%1, %2};" : "=l"(p.v) : "f"(x), "f"(y));
    return p;
}
__device__ inline float2 halves(F32x2 p)
{
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(p.v));
    return f;
}
__device__ inline double2 make_pair2(double x, double y) { return make_double2(x, y); }
__device__ inline double2 halves(double2 p) { return p; }
template <typename P>
__device__ inline auto pair_sum(P p)
{
    const auto f = halves(p);
    return f.x + f.y;
}
// p with its second half replaced
template <typename P, typename R>
__device__ inline P with_y(P p, R y)
{
    return make_pair2(halves(p).x, y);
}

// component-wise a * b + c, a * b of (single, double) pairs
__device__ inline F32x2 fma2(F32x2 a, F32x2 b, F32x2 c)
{
    F32x2 d;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(d.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return d;
}
__device__ inline double2 fma2(double2 a, double2 b, double2 c)
{
    return make_double2(fma(a.x, b.x, c.x), fma(a.y, b.y, c.y));
}
__device__ inline F32x2 mul2(F32x2 a, F32x2 b)
{
    F32x2 d;
    asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
    return d;
}
__device__ inline double2 mul2(double2 a, double2 b) { return make_double2(a.x * b.x, a.y * b.y); }

__device__ inline F32x2 weight_pair(__half2 w)
{
    const float2 f = __half22float2(w);
    return make_pair2(f.x, f.y);
}
__device__ inline double2 weight_pair(double2 w) { return w; }

// the factors that a record's (single, double) sums enter the convolution with
__device__ inline F32x2 record_scale(const float2 *scale, long long i, float)
{
    const float2 s = scale[i];
    return make_pair2(-s.x, s.y);
}
__device__ inline double2 record_scale(const float2 *, long long, double) { return make_double2(-1.0, 1.0); }

// V sums over the warp at once (V a power of two, at most 32): each exchange halves the values a
// lane holds, so all V cost V - 1 + log2(32 / V) exchanges.  Lane l ends with the total of value
// l >> (5 - log2 V) in v[0].
template <typename R, int V>
__device__ inline void warp_sums(R (&v)[V], int lane)
{
    int off = 16;
#pragma unroll
    for (int half = V / 2; half > 0; half /= 2, off >>= 1)
    {
        const bool up = (lane & off) != 0;
#pragma unroll
        for (int i = 0; i < half; i++)
        {
            const R send = up ? v[i] : v[i + half], keep = up ? v[i + half] : v[i];
            v[i] = keep + __shfl_xor_sync(kFull, send, off);
        }
    }
    for (; off > 0; off >>= 1)
        v[0] += __shfl_xor_sync(kFull, v[0], off);
}

}  // namespace

}  // namespace pb
