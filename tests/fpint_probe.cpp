// Host build of the integer-pipe FP64 operations (etraj.jl_gb300/csrc/fpint.h) and of
// detmath.h's functions on top of them, for tests/test_fpint.py.  `ulp` moves the
// approximate reciprocals by that many 2^-23, the device approximations' error bound.
static double g_ulp = 0.0;
#define FI_TEST_ERR g_ulp
#define ETRAJ_DM_INT 1
#include "detmath.h"

extern "C" {

void fp_set_ulp(double ulp) { g_ulp = ulp; }

void fp_op(int op, long n, const double* x, const double* y, double* out) {
    for (long i = 0; i < n; ++i) {
        double r = 0.0, s, c;
        int k;
        switch (op) {
            case 0: r = dm_exp(x[i]); break;
            case 1: r = dm_expm1(x[i]); break;
            case 2: r = dm_log(x[i]); break;
            case 3: r = dm_log1p(x[i]); break;
            case 4: dm_sincos(x[i], &s, &c); r = s; break;
            case 5: dm_sincos(x[i], &s, &c); r = c; break;
            case 6: r = dm_tanh(x[i]); break;
            case 7: r = dm_atan(x[i]); break;
            case 8: r = dm_atan2(x[i], y[i]); break;
            case 9: r = dm_asinh(x[i]); break;
            case 10: r = dm_pow_pos(x[i], y[i]); break;
            case 20: r = fi_div(x[i], y[i]); break;
            case 21: r = fi_sqrt(x[i]); break;
            case 22: r = fi_rint_small(x[i], &k); if ((double)k != r) r = dm_nan(); break;
            case 23: r = fi_from_int((int)x[i]); break;
            case 24: r = fi_half(x[i]); break;
            case 28: r = fi_one_minus(x[i], &s); if (s != (1.0 - r) - x[i]) r = dm_nan(); break;
            case 25: r = fi_lt(x[i], y[i]) ? 1.0 : 0.0; break;
            default: break;
        }
        out[i] = r;
    }
}
}
