// vec3.cuh -- the three right-hand sides of an upscaling solve as one vector element.
//
// The three directions of a batch share one matrix and one AMG hierarchy.  Kernels written for a vector
// element type VT run them together on V3: every matrix entry and column is read once for three products,
// and a gather fetches the three values of an unknown at once (one 16-byte load in FP32).
#pragma once

#include <type_traits>

namespace porsol {

template <class T>
struct V3;
template <>
struct alignas(16) V3<float> {
    float a, b, c, pad;   // padded to one 16-byte load
};
template <>
struct V3<double> {
    double a, b, c;
};

template <class VT>
struct ElementOf {
    using type = VT;
    static constexpr bool three = false;
};
template <class T>
struct ElementOf<V3<T>> {
    using type = T;
    static constexpr bool three = true;
};
template <class VT>
using scalar_t = typename ElementOf<VT>::type;
template <class VT>
constexpr bool is_v3 = ElementOf<VT>::three;
// FP64 element of the same width
template <class VT>
using wide_t = std::conditional_t<is_v3<VT>, V3<double>, double>;

#ifdef __CUDACC__
template <class T>
__device__ __forceinline__ V3<T> make_v3(T a, T b, T c)
{
    V3<T> v{};
    v.a = a;
    v.b = b;
    v.c = c;
    return v;
}
template <class T>
__device__ __forceinline__ V3<T> operator+(const V3<T>& x, const V3<T>& y) { return make_v3<T>(x.a + y.a, x.b + y.b, x.c + y.c); }
template <class T>
__device__ __forceinline__ V3<T> operator-(const V3<T>& x, const V3<T>& y) { return make_v3<T>(x.a - y.a, x.b - y.b, x.c - y.c); }
template <class T>
__device__ __forceinline__ V3<T> operator*(T s, const V3<T>& x) { return make_v3<T>(s * x.a, s * x.b, s * x.c); }
template <class T>
__device__ __forceinline__ V3<T> operator*(const V3<T>& x, T s) { return s * x; }
template <class T>
__device__ __forceinline__ V3<T>& operator+=(V3<T>& x, const V3<T>& y) { return x = x + y; }
// component by component (scales and coefficients per direction)
template <class T>
__device__ __forceinline__ V3<T> times(const V3<T>& x, const V3<T>& y) { return make_v3<T>(x.a * y.a, x.b * y.b, x.c * y.c); }

// acc + s x, contracted
template <class T>
__device__ __forceinline__ T multiply_add(T acc, T s, T x) { return acc + s * x; }
template <class T>
__device__ __forceinline__ V3<T> multiply_add(const V3<T>& acc, T s, const V3<T>& x)
{
    return make_v3<T>(acc.a + s * x.a, acc.b + s * x.b, acc.c + s * x.c);
}

template <class T>
__device__ __forceinline__ T shfl_xor(T v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
template <class T>
__device__ __forceinline__ V3<T> shfl_xor(const V3<T>& v, int o)
{
    return make_v3<T>(shfl_xor(v.a, o), shfl_xor(v.b, o), shfl_xor(v.c, o));
}

__device__ __forceinline__ double to_wide(float v) { return double(v); }
__device__ __forceinline__ double to_wide(double v) { return v; }
template <class T>
__device__ __forceinline__ V3<double> to_wide(const V3<T>& v) { return make_v3<double>(double(v.a), double(v.b), double(v.c)); }
template <class VT>
__device__ __forceinline__ VT from_wide(const wide_t<VT>& v)
{
    using T = scalar_t<VT>;
    if constexpr (is_v3<VT>) return make_v3<T>(T(v.a), T(v.b), T(v.c));
    else return T(v);
}
#endif

}  // namespace porsol
