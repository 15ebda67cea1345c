// Small complex transforms in registers and the two-step real transforms of
// fold rows built on them (fourier.cu).
#pragma once

#include <type_traits>

#include <cuda_runtime.h>

namespace lk::fft {

// cos(2 pi k / 32) for k in [0, 32).
__host__ __device__ constexpr float cos32(int k) {
    k &= 31;
    const int q = k <= 16 ? k : 32 - k;         // cos is even
    const int h = q <= 8 ? q : 16 - q;          // cos(pi - x) = -cos x
    constexpr float c[9] = {1.0f,         0.980785280f, 0.923879533f, 0.831469612f, 0.707106781f,
                            0.555570233f, 0.382683432f, 0.195090322f, 0.0f};
    return q <= 8 ? c[h] : -c[h];
}
__host__ __device__ constexpr float sin32(int k) { return cos32(k - 8); }

constexpr int bit_reverse(int i, int bits) {
    int r = 0;
    for (int b = 0; b < bits; ++b) {
        r |= ((i >> b) & 1) << (bits - 1 - b);
    }
    return r;
}

template <int I, int N, class F>
__device__ __forceinline__ void static_for(F&& f) {
    if constexpr (I < N) {
        f(std::integral_constant<int, I>{});
        static_for<I + 1, N>(f);
    }
}

// One radix-2 stage (blocks of M) of an N-point transform.
template <int N, int M, int SIGN>
__device__ __forceinline__ void fft_stage(float2 (&x)[N]) {
    static_for<0, N / 2>([&](auto ic) {
        constexpr int j = decltype(ic)::value % (M / 2), k = decltype(ic)::value / (M / 2) * M + j;
        constexpr int t32 = j * (32 / M);
        constexpr float c = cos32(t32), sn = static_cast<float>(SIGN) * sin32(t32);
        const float2 a = x[k], b = x[k + M / 2];
        float2 p;
        if constexpr (t32 == 0) {
            p = b;
        } else if constexpr (t32 == 8) {
            p = make_float2(-sn * b.y, sn * b.x);
        } else {
            p = make_float2(fmaf(b.x, c, -(b.y * sn)), fmaf(b.x, sn, b.y * c));
        }
        x[k] = make_float2(a.x + p.x, a.y + p.y);
        x[k + M / 2] = make_float2(a.x - p.x, a.y - p.y);
    });
    if constexpr (M < N) {
        fft_stage<N, 2 * M, SIGN>(x);
    }
}

// In-place radix-2 transform of N (a power of two up to 32) values in
// registers, natural order in and out: x_k = sum_j x_j exp(SIGN 2 pi i j k / N).
template <int N, int SIGN>
__device__ __forceinline__ void fft_reg(float2 (&x)[N]) {
    constexpr int BITS = N == 2 ? 1 : N == 4 ? 2 : N == 8 ? 3 : N == 16 ? 4 : 5;
    static_assert((1 << BITS) == N, "power of two up to 32");
    static_for<0, N>([&](auto ic) {
        constexpr int i = decltype(ic)::value, r = bit_reverse(i, BITS);
        if constexpr (r > i) {
            const float2 t = x[i];
            x[i] = x[r];
            x[r] = t;
        }
    });
    fft_stage<N, 2, SIGN>(x);
}

}  // namespace lk::fft
