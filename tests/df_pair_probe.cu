// Pairs of double-floats against single ones on the device (dfloat.h, df_solve.cuh): every
// operation on pairs, and the two exponentials of the SAE potential at once, must give the
// bits the single operations give.  counts[i]: mismatches of operation i.
#include "df_solve.cuh"

using namespace etraj;

__device__ const float g_exp2[2 * kExpTabN] = {ETRAJ_DF_EXP2_TABLE};

__device__ bool differ(df a, df b) {
    return __float_as_uint(a.hi) != __float_as_uint(b.hi) || __float_as_uint(a.lo) != __float_as_uint(b.lo);
}
__device__ bool differ(dfp p, df a, df b) { return differ(dfp_get(p, 0), a) || differ(dfp_get(p, 1), b); }
__device__ void check(unsigned long long* counts, int i, bool bad) {
    if (bad) atomicAdd(counts + i, 1ull);
}

// x: n double-floats (hi, lo), taken four at a time as (a, b) and (c, d)
__global__ void k_pairs(const float* x, long n, unsigned long long* counts) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (4 * i + 3 >= n) return;
    df v[4];
    for (int j = 0; j < 4; ++j) v[j] = df{x[8 * i + 2 * j], x[8 * i + 2 * j + 1]};
    const df a = v[0], b = v[1], c = v[2], d = v[3];
    const dfp p = dfp_of(a, b), q = dfp_of(c, d);
    check(counts, 0, differ(df_add(p, q), df_add(a, c), df_add(b, d)));
    check(counts, 1, differ(df_sub(p, q), df_sub(a, c), df_sub(b, d)));
    check(counts, 2, differ(df_mul(p, q), df_mul(a, c), df_mul(b, d)));
    check(counts, 3, differ(df_sqr(p), df_sqr(a), df_sqr(b)));
    check(counts, 4, differ(df_fma(p, q, p), df_fma(a, c, a), df_fma(b, d, b)));
    check(counts, 5, differ(df_fma_f(p.hi, q, p), df_fma_f(a.hi, c, a), df_fma_f(b.hi, d, b)));
    check(counts, 6, differ(df_add_f(p, q.hi * q.lo), df_add_f(a, c.hi * c.lo), df_add_f(b, d.hi * d.lo)));
    dfs::AccP s(p);
    dfs::Acc s0(a), s1(b);
    s.add(q, p);
    s.add(p, q);
    s0.add(c, a);
    s0.add(a, c);
    s1.add(d, b);
    s1.add(b, d);
    check(counts, 7, differ(s.get(), s0.get(), s1.get()));
    // exponents |a| r and |b| r, on both sides of the limit beyond which they are 0
    const df k1 = df_abs(a), k3 = df_abs(b), r = df_abs(c);
    const dfp e = dfs::sae_exp2(k1, k3, r, g_exp2);
    check(counts, 8, differ(e, dfs::sae_exp(k1, r, g_exp2), dfs::sae_exp(k3, r, g_exp2)));
}

extern "C" int df_pairs(const float* x, long n, unsigned long long* counts) {
    float* dx = nullptr;
    unsigned long long* dc = nullptr;
    if (cudaMalloc(&dx, 2 * n * sizeof(float)) || cudaMalloc(&dc, 9 * sizeof *dc)) return (int)cudaGetLastError();
    cudaMemcpy(dx, x, 2 * n * sizeof(float), cudaMemcpyHostToDevice);
    cudaMemset(dc, 0, 9 * sizeof *dc);
    k_pairs<<<(unsigned)((n / 4 + 255) / 256), 256>>>(dx, n, dc);
    const int rc = (int)cudaMemcpy(counts, dc, 9 * sizeof *dc, cudaMemcpyDeviceToHost);
    cudaFree(dx);
    cudaFree(dc);
    return rc;
}
