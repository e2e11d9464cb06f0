// tt_step.cuh -- the ten Tusscher model as time steps run it (EP_TT_JAC_TRUE):
// the equations of tt.cuh with their fractions brought over one denominator
// and the Newton Jacobian written out.
//
// The kernel was bound by instructions: per sub-step some 46 exponentials and
// 70 divisions of the gates, and per Newton iteration 12 more evaluations of
// the rates for the differenced Jacobian, 36 divisions to form it and a pivoted
// 6x6 LU.  Here a gate takes one division, an iteration one evaluation with 19
// Jacobian entries that share its divisions and exponentials, and the solve is
// a band of five and one.  One ionic phase of the 263K-node shell (FP32, five
// sub-steps): 2024 -> 127 us; of a 24-slab batch of 446K nodes: 613 -> 58 us;
// of 14K nodes in FP64: 109 -> 24 us.  Against 64-bit values the FP32 form is
// the more accurate one (a differenced FP32 Jacobian has three digits).
#pragma once
#include "tt.cuh"

namespace ep {
namespace tts {

// Newton-state slots (reference State index): 0 Ki(1) 1 Nai(2) 2 Cai(3)
// 3 Cass(10) 4 CaSR(17) 5 R'(18)
template <typename R> struct TTFixed {          // voltage/gate-only terms, constants of the cell
    R V, rtf, rtf_half, ist;
    R nak, g_na, naca_n, naca_c;                // I_NaK factor; I_NaCa = naca_n Nai^3 - naca_c Cai
    R g_k1, g_to, g_kr, g_ks, g_pk;
    R cal_s, cal_0;                             // I_CaL = cal_s Cass - cal_0
    R eks_num;
    R cap, cap_ss, vsr_c, vsr_ss, vc_ss;        // C_m / (V_c F), C_m / (2 V_ss F), volume ratios
};

template <typename R> struct TTRev {            // concentration-dependent terms
    R ENa, EK, EKs, ECa, xk1;
};

// The 12 gates of one Compute_Ion call (kinetics Tusscher.cc:5-55): the
// semi-implicit (s + dt inf/tau) / (1 + dt/tau) at voltage V
// (UpdateStateVariables, Tusscher.cc:116-195).  With inf = I / A and tau = N /
// D the step is dt D (I - s A) / ((N + dt D) A): one division a gate in place of
// four to nine, and added to s its own rounding counts only as much as the gate
// moves (as one quotient, s N A + dt D I over the same, the new value's error was
// a quarter larger than the reference's order of operations gives; it is half of
// that: RMS over a wave's states 0.35-0.5 of 1e-16 in FP64, 0.8-0.95 there).
template <typename R>
EP_HD R tt_gate(R s, R dt, R N, R D, R A) {
    const R e = dt * D;
    return s + dv(e * (R(1) - s * A), (N + e) * A);
}
// the same for m, whose time constant may be far below dt: then the quotient,
// which keeps the digits of a small new value
template <typename R>
EP_HD R tt_gate_fast(R s, R dt, R N, R D, R A) {
    const R e = dt * D;
    const bool slow = e < N;
    const R q = dv(slow ? e * (R(1) - s * A) : s * N * A + e, (N + e) * A);
    return slow ? s + q : q;
}

template <typename R>
EP_HD void tt_gate_step(R s[TT_NS], R V, R dt, const R *__restrict__ c) {
    const R one = R(1);
    // Xr1, Xr2, Xs
    s[3] = tt_gate(s[3], dt, R(2700), (one + cexp(over(R(-45) - V, 10))) * (one + cexp(over(V + R(30), 11.5))),
                   one + cexp(over(R(-26) - V, 7)));
    s[4] = tt_gate(s[4], dt, R(3.36), (one + cexp(over(R(-60) - V, 20))) * (one + cexp(over(V - R(60), 20))),
                   one + cexp(over(V + R(88), 24)));
    {
        const R D = sqrt(one + cexp(over(R(5) - V, 6))) * (one + cexp(over(V - R(35), 15)));
        s[5] = tt_gate(s[5], dt, R(1400) + R(80) * D, D, one + cexp(over(R(-5) - V, 14)));
    }
    {   // m
        const R t = one + cexp(over(R(-56.86) - V, 9.03));
        const R b1 = one + cexp(over(V + R(35), 5)), b2 = one + cexp(over(V - R(50), 200));
        s[6] = tt_gate_fast(s[6], dt, R(0.1) * (b1 + b2), (one + cexp(over(R(-60) - V, 5))) * b1 * b2, t * t);
    }
    {   // h, j
        const R t = one + cexp(over(V + R(71.55), 7.43));
        R nh, dh, nj, dj;
        if (V < R(-40)) {
            nh = one;
            dh = R(0.057) * cexp(over(-(V + R(80)), 6.8)) + R(2.7) * exp(R(0.079) * V) + R(310000) * exp(R(0.3485) * V);
            const R p1 = one + exp(R(0.311) * (V + R(79.23))), p2 = one + cexp(R(-0.1378) * (V + R(40.14)));
            nj = p1 * p2;
            dj = (R(-25428) * exp(R(0.2444) * V) - R(6.948e-06) * cexp(R(-0.04391) * V)) * (V + R(37.78)) * p2
               + R(0.02424) * cexp(R(-0.01052) * V) * p1;
        } else {
            nh = R(0.13) * (one + cexp(over(-(V + R(10.66)), 11.1)));
            dh = R(0.77);
            nj = one + cexp(R(-0.1) * (V + R(32)));
            dj = R(0.6) * cexp(R(0.057) * V);
        }
        s[7] = tt_gate(s[7], dt, nh, dh, t * t);
        s[8] = tt_gate(s[8], dt, nj, dj, t * t);
    }
    {   // d
        const R b1 = one + cexp(over(R(-35) - V, 13)), b2 = one + cexp(over(V + R(5), 5)), b3 = one + cexp(over(R(50) - V, 20));
        s[10] = tt_gate(s[10], dt, (R(1.4) + R(0.25) * b1) * R(1.4) * b3 + b1 * b2, b1 * b2 * b3,
                        one + cexp(over(R(-8) - V, 7.5)));
    }
    const R v27 = (V + R(27)) * (V + R(27)), b30 = one + cexp(over(V + R(30), 10));
    {   // f
        const R b1 = one + cexp(over(R(13) - V, 10));
        s[11] = tt_gate(s[11], dt, (R(1102.5) * exp(over(-v27, 225)) + R(20)) * b1 * b30 + R(200) * b30 + R(180) * b1,
                        b1 * b30, one + cexp(over(V + R(20), 7)));
    }
    {   // f2: inf = 0.67 / A + 0.33
        const R b1 = one + cexp(over(R(25) - V, 10)), A = one + cexp(over(V + R(35), 7));
        const R N = R(562) * exp(over(-v27, 240)) * b1 * b30 + R(31) * b30 + R(80) * b1, D = b1 * b30;
        const R e = dt * D;
        s[12] += dv(e * (R(0.67) + (R(0.33) - s[12]) * A), (N + e) * A);
    }
    {   // fCass: inf = 0.6 / q + 0.4, tau = 80 / q + 2
        const R t = R(20) * s[9], q = one + t * t, N = R(80) + R(2) * q;
        s[13] += dv(dt * (R(0.6) + (R(0.4) - s[13]) * q), N + dt * q);
    }
    if (c[53] == R(0)) {   // s
        const R b = one + cexp(over(V - R(20), 5));
        s[14] = tt_gate(s[14], dt, (R(85) * exp(over(-((V + R(45)) * (V + R(45))), 320)) + R(3)) * b + R(5), b,
                        one + cexp(over(V + R(20), 5)));
    } else {               // TT2006 endocardial s gate (not in the reference)
        s[14] = tt_gate(s[14], dt, R(1000) * exp(over(-((V + R(67)) * (V + R(67))), 1000)) + R(8), one,
                        one + cexp(over(V + R(28), 5)));
    }
    s[15] = tt_gate(s[15], dt, R(9.5) * exp(over(-((V + R(40)) * (V + R(40))), 1800)) + R(0.8), one,
                    one + cexp(over(R(20) - V, 6)));
}

// s: the 18 stored states (s[k-1] = reference State[k]), after the gate update
template <typename R>
EP_HD TTFixed<R> tt_fixed(R V, const R *s, const R *__restrict__ c, R ist, R gks) {
    TTFixed<R> f;
    const R F = c[2], RT = c[0] * c[1], u = V * dv(F, RT);       // V F / RT
    f.V = V; f.ist = ist;
    f.rtf = dv(RT, F);
    f.rtf_half = R(0.5) * f.rtf;
    f.nak = dvc(c[21] * c[10],
               (c[10] + c[22]) * (R(1) + R(0.1245) * cexp(R(-0.1) * u) + R(0.0353) * cexp(-u)));
    f.g_na = c[16] * (s[6] * s[6] * s[6]) * s[7] * s[8];
    const R e_g = exp(c[27] * u), e_g1 = exp((c[27] - R(1)) * u);
    const R nao3 = c[11] * c[11] * c[11];
    const R naca = dvc(c[24], ((c[29] * c[29] * c[29]) + nao3) * (c[28] + c[12]) * (R(1) + c[25] * e_g1));
    f.naca_n = naca * e_g * c[12];
    f.naca_c = naca * e_g1 * nao3 * c[26];
    const R sq_ko = sqrt(over(c[10], 5.4));
    f.g_k1 = c[13] * sq_ko;
    f.g_to = c[20] * s[15] * s[14];                 // r (16), s (15)
    f.g_kr = c[14] * sq_ko * s[3] * s[4];           // Xr1, Xr2
    f.g_ks = (c[15] * gks) * (s[5] * s[5]);         // Xs (per-node G_Ks multiplier)
    // I_CaL = 2 F g x / (exp(x) - 1) (0.25 Cass exp(x) - Cao), x = 2 (V - 15) F
    // / RT.  The factor x / (exp(x) - 1) is 0/0 at V = 15 mV; FP32 lands on it
    // (V within an ulp of 15) often enough over millions of node-steps, so the
    // removable singularity takes its series 1 - x/2 + x^2/12 (next term
    // x^4/720) inside a band where that series is exact to the type's precision
    // and exp(x) - 1 would lose most of its digits to cancellation.
    const R xca = dv(R(2) * (V - R(15)) * F, RT), e_ca = exp(xca);
    const R band = sizeof(R) == 4 ? R(1e-2) : R(1e-6);
    const R ghk = fabs(xca) < band ? R(1) - xca * R(0.5) + over(xca * xca, 12) : dv(xca, e_ca - R(1));
    const R cal = c[18] * s[10] * s[11] * s[12] * s[13] * R(2) * F * ghk;
    f.cal_s = cal * R(0.25) * e_ca;
    f.cal_0 = cal * c[12];
    f.g_pk = dv(c[32], R(1) + cexp(over(R(25) - V, 5.98)));
    f.eks_num = c[10] + c[9] * c[11];
    f.cap = dv(c[3], c[4] * F);
    f.cap_ss = dv(c[3], R(2) * c[52] * F);
    f.vsr_c = dv(c[51], c[4]);
    f.vsr_ss = dv(c[51], c[52]);
    f.vc_ss = dv(c[4], c[52]);
    return f;
}

template <typename R>
EP_HD void tt_rev_na(TTRev<R> &e, R Nai, const R *c, const TTFixed<R> &f) {
    e.ENa = f.rtf * log(dv(c[11], Nai));
}
// the rectifier's two rates share one division: a / (a + b) = 1 / (1 + b / a)
template <typename R>
EP_HD void tt_rev_k(TTRev<R> &e, R Ki, const R *c, const TTFixed<R> &f) {
    e.EK = f.rtf * log(dv(c[10], Ki));
    const R vk = f.V - e.EK;
    const R a = R(1) + cexp(R(0.06) * (vk - R(200)));
    const R b = R(3) * exp(R(0.0002) * (vk + R(100))) + cexp(R(0.1) * (vk - R(10)));
    const R d = R(1) + cexp(R(-0.5) * vk);
    e.xk1 = dv(R(0.1) * d, R(0.1) * d + a * b);
}
template <typename R>
EP_HD void tt_rev_ks(TTRev<R> &e, R Ki, R Nai, const R *c, const TTFixed<R> &f) {
    e.EKs = f.rtf * log(dv(f.eks_num, Ki + c[9] * Nai));
}
template <typename R>
EP_HD void tt_rev_ca(TTRev<R> &e, R Cai, const R *c, const TTFixed<R> &f) {
    e.ECa = f.rtf_half * log(dv(c[12], Cai));
}
template <typename R>
EP_HD TTRev<R> tt_rev(const R x[6], const R *c, const TTFixed<R> &f) {
    TTRev<R> e;
    tt_rev_na(e, x[1], c, f);
    tt_rev_k(e, x[0], c, f);
    tt_rev_ks(e, x[0], x[1], c, f);
    tt_rev_ca(e, x[2], c, f);
    return e;
}

// Rates of the 6 Newton states and dV/dt (Tusscher.cc:56-95) at
// x = (Ki, Nai, Cai, Cass, CaSR, R').
template <typename R>
EP_HD void tt_nr_rates(const R x[6], const TTRev<R> &e, const TTFixed<R> &f,
                                            const R *c, R r[6], R &dvdt) {
    const R V = f.V;
    const R Nai = x[1], Cai = x[2], Cass = x[3], Casr = x[4], Rp = x[5];
    const R i_nak = f.nak * dvc(Nai, Nai + c[23]);
    const R i_na = f.g_na * (V - e.ENa);
    const R i_bna = c[17] * (V - e.ENa);
    const R i_naca = f.naca_n * (Nai * Nai * Nai) - f.naca_c * Cai;
    const R vk = V - e.EK;
    const R i_k1 = f.g_k1 * e.xk1 * vk;
    const R i_to = f.g_to * vk;
    const R i_kr = f.g_kr * vk;
    const R i_ks = f.g_ks * (V - e.EKs);
    const R i_cal = f.cal_s * Cass - f.cal_0;
    const R i_bca = c[19] * (V - e.ECa);
    const R i_pk = f.g_pk * vk;
    const R i_pca = dvc(c[30] * Cai, Cai + c[31]);
    dvdt = -(i_k1 + i_to + i_kr + i_ks + i_cal + i_nak + i_na + i_bna + i_naca + i_bca + i_pk + i_pca + f.ist);
    r[0] = -((i_k1 + i_to + i_kr + i_ks + i_pk + f.ist) - R(2) * i_nak) * f.cap;
    r[1] = -(i_na + i_bna + R(3) * i_nak + R(3) * i_naca) * f.cap;
    const R j_up = dv(c[44] * (Cai * Cai), Cai * Cai + c[42] * c[42]);
    const R j_leak = c[43] * (Casr - Cai);
    const R j_xfer = c[41] * (Cass - Cai);
    const R uc = (Cai + c[46]) * (Cai + c[46]);
    r[2] = dv(uc, uc + c[45] * c[46]) *
           (((j_leak - j_up) * f.vsr_c + j_xfer) - ((i_bca + i_pca) - R(2) * i_naca) * (R(0.5) * f.cap));
    const R kcasr = c[38] - (c[38] - c[39]) * dv(Casr * Casr, Casr * Casr + c[37] * c[37]);
    r[5] = -(c[34] * kcasr) * Cass * Rp + c[36] * (R(1) - Rp);
    const R k1s = dv(c[33] * (Cass * Cass), kcasr);
    const R j_rel = c[40] * dv(k1s * Rp, c[35] + k1s) * (Casr - Cass);
    const R usr = (Casr + c[48]) * (Casr + c[48]);
    r[4] = dv(usr, usr + c[47] * c[48]) * (j_up - (j_rel + j_leak));
    const R uss = (Cass + c[50]) * (Cass + c[50]);
    r[3] = dv(uss, uss + c[49] * c[50]) * ((j_rel * f.vsr_ss - i_cal * f.cap_ss) - j_xfer * f.vc_ss);
}

// dV/dt of the model at an arbitrary state (the current balance of
// ComputeRates, Tusscher.cc:56-78), s = the 18 stored states
template <typename R>
EP_HD R tt_dvdt(R V, const R *s, const R *__restrict__ c, R ist, R gks) {
    const TTFixed<R> f = tt_fixed<R>(V, s, c, ist, gks);
    const R x[6] = {s[0], s[1], s[2], s[9], s[16], s[17]};
    const TTRev<R> e = tt_rev(x, c, f);
    R r[6], dvdt;
    tt_nr_rates(x, e, f, c, r, dvdt);
    return dvdt;
}

// One Newton step of x - xn - dt f(x) = 0 with the Jacobian of the rates
// above, x <- x - B.  The Jacobian is written out: each rate depends on two to
// four of the six states, so it has 19 entries, which share their divisions
// and exponentials with the rates, where central differences take twelve more
// evaluations and, in FP32, resolve an entry to three digits only.  Ki appears
// in its own rate alone and is solved last; the other five, ordered Nai, Cai,
// Cass, CaSR, R', form a band that is eliminated in place (the diagonals are
// 1 + dt x decay, except where dt times Cass' buffered gain cancels its one and an
// exchange with CaSR's row would keep digits: over a wave's states the solutions
// equal a pivoted elimination's up to dt = 0.1 ms, and beyond, to 0.3 ms, Newton
// runs fail about equally often with and without).
template <typename R>
EP_HD void tt_newton_step(R x[6], const R xn[6], R dt, const TTFixed<R> &f, const R *__restrict__ c, R B[6]) {
    const R V = f.V;
    const R K = x[0], N = x[1], C = x[2], S = x[3], Q = x[4], P = x[5];
    // potassium: EK, EKs and the I_K1 rectifier
    const R iK = dv(R(1), K);
    const R vk = V - f.rtf * log(c[10] * iK);
    const R ks = dv(R(1), K + c[9] * N);
    const R vks = V - f.rtf * log(f.eks_num * ks);
    R xk1, dxk1;
    {
        const R e1 = cexp(R(0.06) * (vk - R(200))), e2 = R(3) * exp(R(0.0002) * (vk + R(100)));
        const R e3 = cexp(R(0.1) * (vk - R(10))), e4 = cexp(R(-0.5) * vk);
        // xk1 = n / (n + m), n = 0.1 (1 + e4), m = (1 + e1)(e2 + e3)
        const R n = R(0.1) * (R(1) + e4), m = (R(1) + e1) * (e2 + e3);
        const R dn = R(-0.05) * e4, dm = R(0.06) * e1 * (e2 + e3) + (R(1) + e1) * (R(0.0002) * e2 + R(0.1) * e3);
        const R q = dv(R(1), n + m);
        xk1 = n * q;
        dxk1 = (dn * m - n * dm) * q * q;
    }
    const R g_k = f.g_to + f.g_kr + f.g_pk;
    const R i_ks = f.g_ks * vks;
    // sodium
    const R nq = dv(R(1), N + c[23]);
    const R i_nak = f.nak * N * nq;
    const R d_nak = f.nak * c[23] * nq * nq;
    const R iN = dv(R(1), N);
    const R vna = V - f.rtf * log(c[11] * iN);
    const R i_naca = f.naca_n * (N * N * N) - f.naca_c * C;
    const R d_naca = R(3) * f.naca_n * (N * N);
    const R gna = f.g_na + c[17];
    const R dks = f.g_ks * f.rtf * ks;
    const R hcap = dt * f.cap;
    const R b0 = K - xn[0] + hcap * (vk * (f.g_k1 * xk1 + g_k) + i_ks + f.ist - R(2) * i_nak);
    const R a00 = R(1) + hcap * (f.rtf * iK * (f.g_k1 * (xk1 + vk * dxk1) + g_k) + dks);
    const R a01 = hcap * (c[9] * dks - R(2) * d_nak);
    R b1 = N - xn[1] + hcap * (gna * vna + R(3) * (i_nak + i_naca));
    const R a11 = R(1) + hcap * (gna * f.rtf * iN + R(3) * (d_nak + d_naca));
    const R a12 = R(-3) * hcap * f.naca_c;
    // cytosolic calcium
    const R iC = dv(R(1), C);
    const R pq = dv(R(1), C + c[31]);
    const R up = dv(R(1), C * C + c[42] * c[42]);
    const R j_up = c[44] * (C * C) * up, d_up = R(2) * c[44] * C * (c[42] * c[42]) * up * up;
    const R j_leak = c[43] * (Q - C), j_xfer = c[41] * (S - C);
    const R wc = C + c[46], bq = dv(R(1), wc * wc + c[45] * c[46]);
    const R bufc = wc * wc * bq, dbufc = R(2) * wc * (c[45] * c[46]) * bq * bq;
    const R hc = R(0.5) * f.cap;
    const R gc = ((j_leak - j_up) * f.vsr_c + j_xfer)
               - ((c[19] * (V - f.rtf_half * log(c[12] * iC)) + c[30] * C * pq) - R(2) * i_naca) * hc;
    R b2 = C - xn[2] - dt * bufc * gc;
    const R a21 = -dt * bufc * (R(2) * hc) * d_naca;
    R a22 = R(1) + dt * (bufc * ((c[43] + d_up) * f.vsr_c + c[41]
                                 + (c[19] * f.rtf_half * iC + c[30] * c[31] * pq * pq + R(2) * f.naca_c) * hc)
                         - dbufc * gc);
    const R a23 = -dt * bufc * c[41], a24 = -dt * bufc * c[43] * f.vsr_c;
    // release
    const R q2 = c[37] * c[37], kq = dv(R(1), Q * Q + q2);
    const R kcasr = c[38] - (c[38] - c[39]) * (Q * Q) * kq;
    const R d_kc = R(-2) * (c[38] - c[39]) * Q * q2 * kq * kq;
    const R ikc = dv(R(1), kcasr);
    const R k1 = c[33] * ikc, k1s = k1 * (S * S);
    const R oq = dv(R(1), c[35] + k1s);
    const R o_p = k1s * oq, O = o_p * P;
    const R dO = P * c[35] * oq * oq;                      // dO / d(k1 S^2)
    const R qs = Q - S;
    const R j_rel = c[40] * O * qs;
    const R rel_s = c[40] * (dO * R(2) * k1 * S * qs - O);
    const R rel_q = c[40] * (O - dO * k1s * ikc * d_kc * qs);
    const R rel_p = c[40] * o_p * qs;
    // subspace
    const R ws = S + c[50], sq = dv(R(1), ws * ws + c[49] * c[50]);
    const R bufs = ws * ws * sq, dbufs = R(2) * ws * (c[49] * c[50]) * sq * sq;
    const R gs = (j_rel * f.vsr_ss - (f.cal_s * S - f.cal_0) * f.cap_ss) - j_xfer * f.vc_ss;
    R b3 = S - xn[3] - dt * bufs * gs;
    const R a32 = -dt * bufs * c[41] * f.vc_ss;
    R a33 = R(1) - dt * (bufs * (rel_s * f.vsr_ss - f.cal_s * f.cap_ss - c[41] * f.vc_ss) + dbufs * gs);
    R a34 = -dt * bufs * rel_q * f.vsr_ss;
    const R a35 = -dt * bufs * rel_p * f.vsr_ss;
    // SR
    const R wr = Q + c[48], rq = dv(R(1), wr * wr + c[47] * c[48]);
    const R bufr = wr * wr * rq, dbufr = R(2) * wr * (c[47] * c[48]) * rq * rq;
    const R gr = j_up - (j_rel + j_leak);
    R b4 = Q - xn[4] - dt * bufr * gr;
    const R a42 = -dt * bufr * (d_up + c[43]);
    R a43 = dt * bufr * rel_s;
    R a44 = R(1) - dt * (dbufr * gr - bufr * (rel_q + c[43]));
    R a45 = dt * bufr * rel_p;
    // R'
    const R k2 = c[34] * kcasr;
    R b5 = P - xn[5] - dt * (-k2 * S * P + c[36] * (R(1) - P));
    const R a53 = dt * k2 * P;
    R a54 = dt * c[34] * d_kc * S * P;
    R a55 = R(1) + dt * (k2 * S + c[36]);
    // elimination; a zero pivot takes no step in its unknown
    auto inv = [](R p) { return p != R(0) ? dv(R(1), p) : R(0); };
    const R p1 = inv(a11);
    R l = a21 * p1;
    a22 -= l * a12; b2 -= l * b1;
    const R p2 = inv(a22);
    l = a32 * p2;
    a33 -= l * a23; a34 -= l * a24; b3 -= l * b2;
    l = a42 * p2;
    a43 -= l * a23; a44 -= l * a24; b4 -= l * b2;
    const R p3 = inv(a33);
    l = a43 * p3;
    a44 -= l * a34; a45 -= l * a35; b4 -= l * b3;
    l = a53 * p3;
    a54 -= l * a34; a55 -= l * a35; b5 -= l * b3;
    const R p4 = inv(a44);
    l = a54 * p4;
    a55 -= l * a45; b5 -= l * b4;
    B[5] = b5 * inv(a55);
    B[4] = (b4 - a45 * B[5]) * p4;
    B[3] = (b3 - a34 * B[4] - a35 * B[5]) * p3;
    B[2] = (b2 - a23 * B[3] - a24 * B[4]) * p2;
    B[1] = (b1 - a12 * B[2]) * p1;
    B[0] = (b0 - a01 * B[1]) * inv(a00);
#pragma unroll
    for (int i = 0; i < 6; i++) x[i] -= B[i];
}

// The size of a Newton correction B that the stop test looks at: the
// reference's absolute norm, or (FP32) relative to max(|x|, 1)
template <typename R>
EP_HD R tt_resid(const R B[6], const R x[6], int scaled) {
    R acc = R(0);
#pragma unroll
    for (int i = 0; i < 6; i++) {
        const R q = scaled ? dv(B[i], fmax(fabs(x[i]), R(1))) : B[i];
        acc += q * q;
    }
    return sqrt(acc);
}

// One Compute_Ion call with the Newton Jacobian the reference writes down but
// does not solve with (EP_TT_JAC_TRUE): s (18 stored states) advanced in place
// by dt at frozen voltage V; returns dV/dt at the final Newton iterate.
// *iters receives the Newton iteration count (capped by opt.newton_cap).
template <typename R>
EP_HD R tt_compute_ion(R s[TT_NS], R V, R ist, R dt, const R *__restrict__ c, R gks, const TTOpts &opt,
                            int &iters) {
    tt_gate_step(s, V, dt, c);
    const TTFixed<R> f = tt_fixed<R>(V, s, c, ist, gks);
    R x[6] = {s[0], s[1], s[2], s[9], s[16], s[17]};
    R xn[6];
#pragma unroll
    for (int i = 0; i < 6; i++) xn[i] = x[i];
    const R tol = R(opt.newton_tol);
    R resid = R(100);
    int it = 0;
#pragma unroll 1
    while (resid > tol && it < opt.newton_cap) {
        R B[6];
        tt_newton_step(x, xn, dt, f, c, B);
        resid = tt_resid(B, x, opt.fp32_scaled_tol);
        it++;
    }
    s[0] = x[0]; s[1] = x[1]; s[2] = x[2]; s[9] = x[3]; s[16] = x[4]; s[17] = x[5];
    iters = it;
    const TTRev<R> e = tt_rev(x, c, f);
    R r[6], dvdt;
    tt_nr_rates(x, e, f, c, r, dvdt);
    return dvdt;
}

}  // namespace tts
}  // namespace ep
