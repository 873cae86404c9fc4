// Straight-line quotients and square roots (csrc/exact_math.cuh) against the
// device's IEEE division and square root: prints the number of differences
// and the number of comparisons of each kind.
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <vector>

#include "exact_math.cuh"

using namespace gd2d;
typedef unsigned long long u64;
typedef unsigned __int128 u128;

enum { RANDOM, RANGE, SPECIAL, HARD_QUOTIENT, SQRT, HARD_SQRT, ZERO, KINDS };
struct Count {
    u64 bad[KINDS], n[KINDS];
};

__device__ u64 next(u64 &s) {  // splitmix64
    s += 0x9E3779B97F4A7C15ull;
    u64 z = s;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
// significand in [2^52, 2^53) times 2^(e - 52)
__device__ double make(u64 m, int e) {
    return __longlong_as_double((long long)((m & 0xFFFFFFFFFFFFFull) | ((u64)(e + 1023) << 52)));
}
__device__ void compare(Count *c, int kind, double a, double b) {
    atomicAdd(&c->n[kind], 1ull);
    if (__double_as_longlong(a) != __double_as_longlong(b)) atomicAdd(&c->bad[kind], 1ull);
}

__global__ void check(Count *c, u64 seed, int iters) {
    u64 s = seed + (u64)(blockIdx.x * blockDim.x + threadIdx.x) * 0x2545F4914F6CDD1Dull;
    for (int it = 0; it < iters; ++it) {
        const u64 ma = (next(s) >> 12) | (1ull << 52), mb = (next(s) >> 12) | (1ull << 52), w = next(s);
        const double sign = (w >> 63) ? -1.0 : 1.0;
        compare(c, RANDOM, div_rn(sign * make(ma, (int)(w % 61) - 30), make(mb, (int)((w >> 8) % 61) - 30)),
                sign * make(ma, (int)(w % 61) - 30) / make(mb, (int)((w >> 8) % 61) - 30));
        {  // the whole range of the callers' tests
            const double d = make(mb, (int)((w >> 8) % 899) - 700), n = sign * make(ma, (int)((w >> 24) % 1499) - 800);
            const double q = n / d;
            if (fabs(q) > 1e-300 && fabs(q) < 1e300) compare(c, RANGE, div_rn(n, d), q);
            const double x = make(ma, (int)((w >> 8) % 1399) - 700);
            compare(c, SQRT, sqrt_rn(x), sqrt(x));
        }
        {  // few-bit significands and those next to a power of two
            u64 m1 = ma >> ((w >> 3) % 50), m2 = mb >> ((w >> 10) % 50);
            while (!(m1 >> 52)) m1 <<= 1;
            while (!(m2 >> 52)) m2 <<= 1;
            if (w & 1) m1 = (1ull << 53) - 1 - ((w >> 20) % 1024);
            if (w & 2) m2 = (1ull << 53) - 2 - ((w >> 30) % 1024);  // (all ones: excluded by the callers)
            const double n = make(m1, (int)((w >> 8) % 61) - 30), d = make(m2, (int)((w >> 14) % 61) - 30);
            if (m2 != (1ull << 53) - 1) compare(c, SPECIAL, div_rn(n, d), n / d);
            compare(c, SQRT, sqrt_rn(n), sqrt(n));
        }
        // quotients next to a midpoint of two doubles: A 2^t = (2Q+1) D + k
        // with odd D and small odd k gives the distance k / (2 D) ulp
        const u64 D = mb | 1ull;
        u64 inv = D;
        for (int i = 0; i < 6; ++i) inv *= 2 - D * inv;
        long long k = (long long)((w >> 5) % 32) * 2 + 1;
        if (w & 16) k = -k;
        for (int t = 53; t <= 54 && D != (1ull << 53) - 1; ++t) {
            const u64 mod = (1ull << t) - 1;
            u64 r = ((u64)(-k) * inv) & mod;
            if (t == 53) r |= 1ull << 53;
            if (r < (1ull << 53)) continue;
            const __int128 v = (__int128)((u128)r * D) + k;
            const u64 A = (u64)((u128)v >> t);
            if (A < (1ull << 52) || A >= (1ull << 53) || ((u64)v & mod)) continue;
            compare(c, HARD_QUOTIENT, div_rn(make(A, 3), make(D, 5)), make(A, 3) / make(D, 5));
        }
    }
    const double d = make((1ull << 52) | (seed & 0xffff), (int)(threadIdx.x % 800) - 600);
    compare(c, ZERO, div_rn(0.0, d), 0.0);
    compare(c, ZERO, div_rn(-0.0, d), -0.0);
}

__global__ void check_sqrt(Count *c, const u64 *m, const int *odd, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
        for (int e = -40; e <= 40; e += 2) {
            const double x = make(m[i], odd[i] + e);
            compare(c, HARD_SQRT, sqrt_rn(x), sqrt(x));
        }
}

int main() {
    // arguments x = X 2^-t whose square root is next to a midpoint z 2^-53:
    // z^2 = -k modulo 2^t for small odd k, roots by Hensel lifting
    std::vector<u64> xs;
    std::vector<int> odd;
    for (int par = 0; par < 2; ++par) {
        const int t = 54 + par;
        const u64 mod = (1ull << t) - 1;
        for (long long k = -4095; k <= 4095; k += 2) {
            const u64 c = (u64)(-k) & mod;
            if ((c & 7) != 1) continue;
            u64 z = 1;
            for (int b = 3; b < t; ++b)
                if ((z * z - c) & ((1ull << (b + 1)) - 1)) z += 1ull << (b - 1);
            for (int v = 0; v < 4; ++v) {
                u64 r = (v & 1) ? (mod + 1 - z) & mod : z;
                if (v & 2) r = (r + (1ull << (t - 1))) & mod;
                if (r < (1ull << 53) || r >= (1ull << 54)) continue;
                const __int128 q = (__int128)((u128)r * r) + k;
                const u64 X = (u64)((u128)q >> t);
                if (((u64)q & mod) || X < (1ull << 52) || X >= (1ull << 53)) continue;
                xs.push_back(X);
                odd.push_back(par);
            }
        }
    }
    Count *c;
    u64 *dx;
    int *dodd;
    const int n = (int)xs.size();
    if (cudaMallocManaged(&c, sizeof *c) || cudaMalloc(&dx, 8 * n + 8) || cudaMalloc(&dodd, 4 * n + 4)) return 1;
    memset(c, 0, sizeof *c);
    cudaMemcpy(dx, xs.data(), 8 * n, cudaMemcpyHostToDevice);
    cudaMemcpy(dodd, odd.data(), 4 * n, cudaMemcpyHostToDevice);
    check_sqrt<<<n / 256 + 1, 256>>>(c, dx, dodd, n);
    check<<<148 * 4, 256>>>(c, 20240607ull, 100);
    if (cudaDeviceSynchronize() != cudaSuccess) return 2;
    for (int k = 0; k < KINDS; ++k) printf("%llu %llu\n", c->bad[k], c->n[k]);
    return 0;
}
