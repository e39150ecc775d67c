// csrc/el_div.cuh against the compiler's division: the largest distance in ulps over random operands (hashed
// counters), printed for tests/test_gpu_div.py.
#include <cstdio>

#include "el_div.cuh"

__device__ unsigned long long mix(unsigned long long x) {  // splitmix64
    x += 0x9e3779b97f4a7c15ull;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
    return x ^ (x >> 31);
}
// a double of a random significand and an exponent in [lo, hi]
__device__ double value(unsigned long long h, int lo, int hi, bool sign) {
    const unsigned long long e = 1023ll + lo + (long long)((h >> 53) % (unsigned)(hi - lo + 1));
    const unsigned long long s = sign && (mix(h) & 1) ? 1ull << 63 : 0ull;
    return __longlong_as_double((long long)(s | (e << 52) | (h & 0xfffffffffffffull)));
}
__device__ unsigned long long ulps(double a, double b) {
    const long long x = __double_as_longlong(a), y = __double_as_longlong(b);
    if ((x < 0) != (y < 0)) return a == b ? 0ull : ~0ull;
    return x > y ? (unsigned long long)(x - y) : (unsigned long long)(y - x);
}

__global__ void check(unsigned long long n, int lo, int hi, unsigned long long* worst) {
    unsigned long long wd = 0, wi = 0;
    for (unsigned long long q = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; q < n;
         q += (unsigned long long)gridDim.x * blockDim.x) {
        const double den = value(mix(2 * q), lo, hi, false), num = value(mix(2 * q + 1), -60, 60, true);
        const unsigned long long d = ulps(el::div_newton(num, den), num / den), i = ulps(el::inverse(den), 1.0 / den);
        wd = d > wd ? d : wd;
        wi = i > wi ? i : wi;
    }
    atomicMax(worst, wd);
    atomicMax(worst + 1, wi);
}

int main() {
    unsigned long long *d, h[2];
    if (cudaMalloc(&d, sizeof(h)) != cudaSuccess) return 1;
    const int range[3][2] = {{-120, 119}, {-900, 900}, {-1, 1}};  // the floats', beyond, near 1
    for (auto& r : range) {
        cudaMemset(d, 0, sizeof(h));
        check<<<1024, 256>>>(1ull << 28, r[0], r[1], d);
        if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
        std::printf("%llu %llu\n", h[0], h[1]);
    }
    return 0;
}
