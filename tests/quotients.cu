/*
 * The quotients by FMA (csrc/quotient.cuh) against IEEE division, on the host and on the device:
 * built by test_quotients.py.  Operands come from a counter, by family; every one that the range
 * checks accept must give the division's bits, and ordinary ones must be accepted.
 */
#include "quotient.cuh"

namespace {

struct Counts {
    unsigned long long accepted, wrong, refused_ordinary;
};

__host__ __device__ uint64_t mix(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
__host__ __device__ double make(uint64_t fraction, int exponent, bool negative) {
    const uint64_t u = (fraction & 0xFFFFFFFFFFFFFull) | (uint64_t)(exponent + 1023) << 52 | (uint64_t)negative << 63;
    double x;
    memcpy(&x, &u, sizeof x);
    return x;
}
__host__ __device__ bool same(double x, double y) {
    uint64_t a, b;
    memcpy(&a, &x, sizeof a);
    memcpy(&b, &y, sizeof b);
    return a == b || (x == 0.0 && y == 0.0);
}

/* One numerator and divisor: family 0 any significands; 1 the divisor's next to all ones, by up to
 * 2^21 units; 2 the divisor's next to one, the numerator's next to all ones; 3 quotients next to a
 * short number; 4 exponents at the edges of the ranges. */
__host__ __device__ void operands(uint64_t seed, uint64_t k, int family, double &n, double &D) {
    const uint64_t r0 = mix(seed ^ mix(k)), r1 = mix(r0), r2 = mix(r1), r3 = mix(r2);
    uint64_t fd = r0, fn = r1;
    int ed = (int)(r2 % 900) - 450, en = (int)(r3 % 900) - 450;
    if (r3 >> 60 == 0) ed = en;
    const uint64_t small = r2 >> (43 + (int)(r3 >> 32) % 21);
    if (family == 1) fd = ~small;
    if (family == 2) fd = small, fn = ~(r3 >> 44);
    if (family == 4) {
        const int edges[8] = {-482, -481, -480, -479, 478, 479, 480, 481};
        ed = r2 & 8 ? edges[r2 & 7] : ed + ed / 15;
        en = (int)(r3 % 2040) - 1020;
    }
    D = make(fd, ed, r2 >> 63);
    n = make(fn, en, r3 >> 63);
    if (family == 3) n = make((r1 >> 40) << 40, en % 200, r3 >> 63) * D;
    if (family == 3 && (r0 & 1)) n = make(fn, en % 200, false), D = make((r0 >> 40) << 40, ed % 200, r2 >> 63);
    if (family == 0 && (r1 & 1023) == 0) n = 0.0;
}

__host__ __device__ void check(uint64_t seed, uint64_t k, int family, Counts &c) {
    double n, D;
    operands(seed, k, family, n, D);
    const bool good = mind::good_divisor(D);
    const bool ordinary = mind::in_binades(D, -300, 300) && mind::in_binades(n, -90, 90) &&
                          ((mind::magnitude_bits(D) + 1) & 0xFFFFFFFFFFFFFull) != 0;
    c.refused_ordinary += ordinary && !good;
    c.wrong += !good && mind::surely_good(D, 1.0);
    if (!good) return;
    const double want = n / D;
    const double x = mind::quotient(n, D, mind::reciprocal(D));
    const bool taken = mind::good_quotient(x, D);
    c.refused_ordinary += ordinary && !taken;
    c.wrong += mind::surely_good(D, x) && !taken;
    if (taken) {
        c.accepted += 1;
        c.wrong += !same(x, want);
    }
    if (mind::good_axial(n)) {
        c.accepted += 1;
        c.wrong += !same(mind::pivot_quotient(n, D), want);
    }
    c.wrong += !same(mind::reciprocal(D), 1.0 / D);
}

__global__ void check_kernel(uint64_t seed, uint64_t count, int family, Counts *out) {
    Counts c{};
    for (uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; k < count; k += (uint64_t)gridDim.x * blockDim.x)
        check(seed, k, family, c);
    atomicAdd(&out->accepted, c.accepted);
    atomicAdd(&out->wrong, c.wrong);
    atomicAdd(&out->refused_ordinary, c.refused_ordinary);
}

}  // namespace

extern "C" void check_on_host(uint64_t seed, uint64_t count, int family, unsigned long long *out) {
    Counts c{};
    for (uint64_t k = 0; k < count; ++k) check(seed, k, family, c);
    memcpy(out, &c, sizeof c);
}

extern "C" int check_on_device(uint64_t seed, uint64_t count, int family, unsigned long long *out) {
    Counts *d = nullptr;
    if (cudaMalloc(&d, sizeof(Counts)) != cudaSuccess) return 1;
    cudaMemset(d, 0, sizeof(Counts));
    check_kernel<<<592, 256>>>(seed, count, family, d);
    const cudaError_t e = cudaMemcpy(out, d, sizeof(Counts), cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e != cudaSuccess;
}
