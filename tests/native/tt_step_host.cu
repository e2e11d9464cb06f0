// tt_step_host.cu -- TEST HARNESS: the ten Tusscher source of the time steps
// (ucla_cmg_b200/csrc/tt_step.cuh, host+device code) beside the one in the
// reference's order of operations (tt.cuh), compiled for the host.  Not part of
// the library.
#include "../../ucla_cmg_b200/csrc/tt_step.cuh"

using namespace ep;

template <typename R>
static void run(int step, int n, double dt, const double *cd, double tol, const double *V, double *states, double *dvdt) {
    R c[64];
    for (int k = 0; k < 54; k++) c[k] = (R)cd[k];
    for (int i = 0; i < n; i++) {
        R s[18];
        double *st = states + 19 * i;
        for (int k = 0; k < 18; k++) s[k] = (R)st[k + 1];
        TTOpts o;
        o.newton_cap = 100;
        o.jac_true = 1;
        o.fp32_scaled_tol = sizeof(R) == 4 ? 1 : 0;
        o.newton_tol = tol;
        int it = 0;
        const R d = step ? tts::tt_compute_ion<R>(s, (R)V[i], R(0), (R)dt, c, R(1), o, it)
                         : tt_compute_ion<R>(s, (R)V[i], R(0), (R)dt, c, R(1), o, it);
        for (int k = 0; k < 18; k++) st[k + 1] = (double)s[k];
        dvdt[i] = (double)d;
    }
}

// step 1: tt_step.cuh, 0: tt.cuh, both with the true Jacobian
extern "C" void tt_step_host(int step, int fp32, int n, double dt, const double *consts, double tol, const double *V,
                             double *states, double *dvdt) {
    if (fp32) run<float>(step, n, dt, consts, tol, V, states, dvdt);
    else run<double>(step, n, dt, consts, tol, V, states, dvdt);
}
