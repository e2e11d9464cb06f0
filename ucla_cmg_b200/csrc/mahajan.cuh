// mahajan.cuh -- Mahajan 2008 UCLA rabbit ventricular model, device side.
//
// Follows voomEP/src/IonicModel/Mahajan.cc: ucla_rhsfun (168-219) with the
// current routines (227-603), forward Euler with Rush-Larsen-type gate
// rates, and the adaptive update of UpdateStateVariables (607-621): if
// |dV/dt| > 20 the step is redone as 10 sub-steps of dt/10, and
// Compute_Ion (624-645) returns the rate of the LAST sub-step.
// Mahajan_fail.cc is the same code with other constants.
#pragma once
#include "common.cuh"

namespace ep {

constexpr int MH_NS = 25;   // stored states besides V: reference State[1..25]
constexpr int MH_NC = 35;

// The rates, in four parts of about equal length that need nothing of one
// another: one thread runs them in turn (mh_rhs), or four warps one each, for
// the same node (k_mahajan).  Then, with what the parts exchange, mh_finish
// completes part 3's rates and mh_totals the voltage and the sodium.
template <typename R> struct MhExchange {
    R xina, xik1, xito, xinak, xikr, xiks, jnaca, po, rxa;
};
template <typename R> struct MhOwn {      // part 3's, until mh_finish
    R jd, buf8, Qr, frac12, frac7;
};

// reference states whose rates part P computes (7, 8 and 12 in mh_finish; 0 and
// 19 are mh_totals')
EP_HD constexpr unsigned int mh_part_states(int P) {
    return P == 0 ? 0x0000000Eu : P == 1 ? 0x0007E010u : P == 2 ? 0x00F00000u : 0x03001FE0u;
}

// r[k] receives the rate of reference state k (k = 0..25); s[k] holds
// reference state k (s[0] = V).  The reference's expressions with their
// fractions brought over one denominator (some 110 divisions of one call
// become 40), 1 - x as the complementary fraction, exp(x) - 1 as expm1, and
// factors that cancel left out (fca in k4 and s2).
template <int P, typename R>
EP_HD void mh_part(const R s[26], const R *__restrict__ c, R h, R r[26], MhExchange<R> &ex, MhOwn<R> &own) {
    const R one = R(1);
    const R V = s[0], frt = c[24], vf = V * frt;
    const R rtf = dv(one, frt), inv_h = dv(one, h), csm = over(s[8], 1000);
    const R vk = V - rtf * log(dv(c[2], c[1]));
    // a gate's rate over the step, (inf - s)(1 - exp(-h k)) / h with k = 1 / tau
    auto relax = [&](R inf, R sk, R hk) { return (sk - inf) * expm1(-hk) * inv_h; };
    if constexpr (P == 0) {
        // I_Na; a = e / (1 + e) switches the h and j rates at -40 mV (over 4 mV):
        // each side's terms only where the other's weight does not leave them
        // under the type's last digit
        {
            const R x = V + R(47.13);
            R am = R(3.2);
            if (fabs(x) > R(0.001)) am = dv(R(-0.32) * x, cexpm1(R(-0.1) * x));
            const R bm = R(0.08) * cexp(over(-V, 11));
            const R u = over(V + R(40), 0.24), reach = sizeof(R) == 4 ? R(23) : R(46);
            R ah = R(0), bh = R(0), aj = R(0), bj = R(0);
            const R eu = exp(-fmin(fmax(u, -reach), reach));
            const R al = dv(eu, one + eu), ar = dv(one, one + eu);       // a and 1 - a
            if (u < reach) {
                ah = al * R(0.135) * cexp(over(R(80) + V, -6.8));
                bh = al * (R(3.56) * cexp(R(0.079) * V) + R(3.1e5) * cexp(R(0.35) * V));
                aj = al * dv((R(-1.2714e5) * cexp(R(0.2444) * V) - R(3.474e-5) * cexp(R(-0.04391) * V)) * (V + R(37.78)),
                             one + cexp(R(0.311) * (V + R(79.23))));
                bj = al * dv(R(0.1212) * cexp(R(-0.01052) * V), one + cexp(R(-0.1378) * (V + R(40.14))));
            }
            if (u > -reach) {
                bh += ar * dv(one, R(0.13) + R(0.13) * cexp(over(V + R(10.66), -11.1)));
                bj += ar * dv(R(0.3) * exp(R(-2.535e-7) * V), one + cexp(R(-0.1) * (V + R(32))));
            }
            const R gm = dv(s[1] + c[31], one + c[31]);
            const R gh = dv(s[2] + c[32], one + c[32]), gj = dv(s[3] + c[33], one + c[33]);
            ex.xina = c[15] * gh * gj * (gm * gm * gm) * (V - rtf * log(dv(c[0], s[19])));
            r[2] = relax(dv(ah, ah + bh), s[2], h * (ah + bh));
            const R ij = dv(one, aj + bj);
            r[3] = relax(aj * (c[34] * ij), s[3], dvc(h * (aj + bj), c[34]));
            r[1] = relax(dv(am, am + bm), s[1], h * (am + bm));
        }
    }
    if constexpr (P == 1) {
        // Markov L-type Ca channel
        {
            const R e8 = cexp(over(-V, 8));
            const R alpha = dv(one, one + e8), beta = e8 * alpha;
            const R r1 = R(0.30), r2 = R(3);
            const R cp3 = s[7] * s[7] * s[7], fca = dv(cp3, cp3 + R(27));
            const R s1 = R(0.0182688) * fca, s1t = R(0.00195);
            const R k1 = R(0.024168) * fca;
            const R k2 = R(1.03615e-4), k1t = R(0.00413), k2t = R(0.00224);
            const R s2 = R(0.0182688 * (0.30 / 3.0) * (1.03615e-4 / 0.024168)), s2t = R(0.00195 * (0.30 / 3.0) * (0.00224 / 0.00413));
            const R e3 = cexp(over(-(V + R(40)), 3));
            const R k3 = dv(e3, R(3) + R(3) * e3), k3t = k3;
            const R e4 = cexp(over(-(V + R(40)), 4));
            const R Pr = dv(e4, one + e4);
            const R recov = R(10) + R(4954) * cexp(over(V, 15.6));
            const R qc = over(s[7], 6.09365);
            const R qc2 = qc * qc;
            const R tau_ca = dv(R(78.0329), one + qc2 * qc2) + R(0.1);
            const R e11 = cexp(over(-(V + R(40)), 11.32));
            const R Ps = dv(one, one + e11), Qs = e11 * Ps;
            const R ica = dv(one, (recov - tau_ca) * Pr + tau_ca);
            const R iba = dv(one, (recov - R(450)) * Pr + R(450));
            const R k6 = fca * Ps * ica, k5 = Qs * ica;
            const R k6t = Ps * iba, k5t = Qs * iba;
            // alpha / beta = 1 / e8; k5 / k6 = e11 / fca, k5t / k6t = e11
            const R kab = k3 * dv(e11, e8);
            const R k4 = kab * R(0.024168 / 1.03615e-4);
            const R k4t = kab * R(0.00413 / 0.00224);
            const R po = ex.po = one - s[15] - s[17] - s[16] - s[18] - s[13] - s[14];
            r[14] = beta * s[13] + k5 * s[17] + k5t * s[18] - (k6 + k6t + alpha) * s[14];
            r[13] = alpha * s[14] + k2 * s[15] + k2t * s[16] + r2 * po - (beta + r1 + k1t + k1) * s[13];
            r[15] = k1 * s[13] + k4 * s[17] + s1 * po - (k3 + k2 + s2) * s[15];
            r[17] = k3 * s[15] + k6 * s[14] - (k5 + k4) * s[17];
            r[16] = k1t * s[13] + k4t * s[18] + s1t * po - (k3t + k2t + s2t) * s[16];
            r[18] = k3t * s[16] + k6t * s[14] - (k5t + k4t) * s[18];
        }
        // driving force of I_Ca
        {
            const R za = R(2) * vf;
            const R factor1 = dvc(R(4) * R(0.00054) * c[23] * c[23], c[22] * c[20]);
            const R em = cexpm1(za);
            const R num = factor1 * (csm * (em + one) - R(0.341) * c[3]);
            if (fabs(za) < R(0.001)) ex.rxa = dv(num, R(2) * frt);
            else ex.rxa = dv(V * num, em);
        }
        // I_Kr
        {
            const R x = V + R(7), y = V + R(10);
            R v1 = R(0.00138 / 0.123);
            if (fabs(x) > R(0.001)) v1 = dv(R(-0.00138) * x, cexpm1(R(-0.123) * x));
            R v2 = R(0.00061 / 0.145);
            if (fabs(y) > R(0.001)) v2 = dv(R(0.00061) * y, cexpm1(R(0.145) * y));
            ex.xikr = dv(c[9] * sqrt(over(c[2], 5.4)) * s[4] * vk, one + cexp(over(V + R(33), 22.4)));
            r[4] = relax(dv(one, one + cexp(over(V + R(50), -7.5))), s[4], h * (v1 + v2));
        }
    }
    if constexpr (P == 2) {
        // I_K1
        {
            const R w = V - rtf * log(dv(R(100) * c[2] + c[0], R(100) * c[1] + s[19]));
            const R e1 = one + cexp(R(0.2385) * (w - R(59.215)));
            const R n = R(0.49124) * cexp(R(0.08032) * (w + R(5.476))) + exp(R(0.061750) * (w - R(594.31)));
            const R d = R(1.02) * (one + cexp(R(-0.5143) * (w + R(4.753))));
            ex.xik1 = c[11] * sqrt(over(c[2], 5.4)) * dv(d, d + n * e1) * w;
        }
        // I_to (slow + fast)
        {
            const R e1 = cexp(over(-(V + R(3)), 15));
            const R xi = dv(one, one + e1);
            const R yi = dv(one, one + cexp(over(V + R(33.5), 10)));
            const R e3 = one + cexp(over(V + R(60), 10));
            ex.xito = (c[6] * s[22] * (s[23] + R(0.5) * yi) + c[7] * s[20] * s[21]) * vk;
            r[22] = relax(xi, s[22], dv(h, R(9) * (e1 * xi) + R(0.5)));
            r[23] = relax(yi, s[23], dv(h * e3, R(3000) + R(30) * e3));
            const R v30 = over(V, 30);
            r[20] = relax(xi, s[20], dv(h, R(3.5) * exp(-(v30 * v30)) + R(1.5)));
            r[21] = relax(yi, s[21], dv(h, R(20) * yi + R(20)));
        }
        // I_NaK
        const R sigma = over(exp(over(c[0], 67.3)) - one, 7);
        ex.xinak = dv(c[12] * c[2] * s[19], (c[2] + R(1.5)) * (s[19] + R(12)) *
                       (one + R(0.1245) * cexp(R(-0.1) * vf) + R(0.0365) * sigma * cexp(-vf)));
    }
    if constexpr (P == 3) {
        // I_Ks
        {
            const R eks = rtf * log(dv(c[2] + R(0.018330) * c[0], c[1] + R(0.018330) * s[19]));
            const R x = V + R(30);
            const R xs1ss = dv(one, one + cexp(over(V - R(1.5), -16.7)));
            R k = R(0.0000719 / 0.148 + 0.000131 / 0.0687);
            if (fabs(x) >= R(0.001 / 0.0687))
                k = dv(R(-0.0000719) * x, cexpm1(R(-0.148) * x)) + dv(R(0.000131) * x, cexpm1(R(0.0687) * x));
            const R c3 = s[9] * s[9] * s[9];
            ex.xiks = c[10] * (one + dv(R(0.8) * c3, c3 + R(0.125))) * s[5] * s[6] * (V - eks);
            r[5] = relax(xs1ss, s[5], h * k);
            r[6] = relax(xs1ss, s[6], R(0.25) * (h * k));
        }
        // Na-Ca exchange flux
        const R na3 = s[19] * s[19] * s[19], nao3 = c[0] * c[0] * c[0];
        {
            const R ez = cexp(R(-0.65) * vf);
            const R zw3 = na3 * c[3] * cexp(R(0.35) * vf) - nao3 * csm * ez;
            const R c3 = s[8] * s[8] * s[8];
            const R qn = over(s[19], 12.3);
            const R yz = R(1.3) * na3 + R(669921.875) * csm                                  // 87.5^3
                       + R(1860.867) * c[3] * (one + over(csm, 0.0036))                      // 12.3^3
                       + R(0.0036) * nao3 * (one + qn * qn * qn) + na3 * c[3] + nao3 * csm;
            ex.jnaca = dv(c[8] * c3 * zw3, (c3 + R(0.027)) * (one + R(0.2) * ez) * yz);
        }
        // Ca cycling
        const R jd = own.jd = dvc(c[28] * (s[8] - s[9]), c[14]);
        r[24] = c[29] * (R(0.0327) * s[9] * (R(70) - s[24]) - R(0.0196) * s[24]);
        r[25] = R(0.0327) * s[8] * (R(70) - s[25]) - R(0.0196) * s[25];
        const R jup = dv(c[30] * c[13] * (s[9] * s[9]), s[9] * s[9] + R(0.25));
        const R jleak = c[27] * dv(R(0.00002069) * (s[10] * s[10]), s[10] * s[10] + R(2500)) * (s[10] * R(16.667) - s[9]);
        // 1 / (1 + 168 / (7 + c)^2 + 28.2 / (0.6 + c)^2 + 4.5 / (0.3 + c)^2 + 546 / (13 + c)^2)
        auto buf = [](R cv) {
            const R a = (R(7) + cv) * (R(7) + cv), b = (R(0.6) + cv) * (R(0.6) + cv);
            const R d = (R(0.3) + cv) * (R(0.3) + cv), e = (R(13) + cv) * (R(13) + cv);
            const R bd = b * d, ae = a * e;
            return dv(ae * bd, ae * bd + R(168) * e * bd + R(546) * a * bd + ae * (R(28.2) * d + R(4.5) * b));
        };
        own.buf8 = buf(s[8]);
        r[9] = buf(s[9]) * (jd - jup + jleak - r[24]);
        r[10] = -s[12] + jup - jleak;
        r[11] = dvc(s[10] - s[11], c[17]);
        {
            const R bv = (c[19] - c[26]) - c[18] * c[19];
            R q = R(0);
            if (s[11] > c[26] && s[11] < c[19]) q = s[11] - c[26];
            else if (s[11] >= c[19]) q = c[18] * s[11] + bv;
            if (q >= c[25]) q = c[25];
            own.Qr = dvc(s[10] * q, c[19]);
        }
        const R e12 = cexp(R(-0.05) * (V + R(30))), e7 = cexp(R(-0.3576) * (V + R(30)));
        own.frac12 = dv(e12, one + e12);
        own.frac7 = dv(e7, one + e7);
        r[12] = s[12] * (dvc(one, c[16]) - dv(r[10], s[10]));
    }
}

// part 3's rates that need the L-type channel's opening and driving force
template <typename R>
EP_HD void mh_finish(const R s[26], const R *__restrict__ c, const MhExchange<R> &ex, const MhOwn<R> &own, R r[26]) {
    const R jca = c[4] * ex.po * ex.rxa, arxa = fabs(ex.rxa);
    r[8] = own.buf8 * (R(50) * (s[12] - own.jd - jca + ex.jnaca) - r[25]);
    r[12] = R(2.58079) * ex.po * arxa * own.frac12 * own.Qr - r[12];
    r[7] = ex.po * arxa * (own.Qr * R(26841.8) * own.frac7 + R(9000)) - R(2) * (s[7] - s[8]);
}

// the rates of the voltage and of the intracellular sodium
template <typename R>
EP_HD void mh_totals(const R *__restrict__ c, R istim, const MhExchange<R> &ex, R &r0, R &r19) {
    const R wca = R(8.0313), jca = c[4] * ex.po * ex.rxa;
    r19 = -over(ex.xina + R(3) * ex.xinak + R(3) * wca * ex.jnaca, 8.0313 * 1000.0);
    r0 = -(ex.xina + ex.xik1 + ex.xikr + ex.xiks + ex.xito + wca * ex.jnaca + R(2) * wca * jca + ex.xinak) + istim;
}

template <typename R>
EP_HD void mh_rhs(const R s[26], const R *__restrict__ c, R h, R istim, R r[26]) {
    MhExchange<R> ex;
    MhOwn<R> own;
    mh_part<0>(s, c, h, r, ex, own);
    mh_part<1>(s, c, h, r, ex, own);
    mh_part<2>(s, c, h, r, ex, own);
    mh_part<3>(s, c, h, r, ex, own);
    mh_finish(s, c, ex, own, r);
    mh_totals(c, istim, ex, r[0], r[19]);
}

// whether the rate asks for ten sub-steps
template <typename R> EP_HD bool mh_wants_substeps(R rate, int abs_mode) {
    return (abs_mode ? fabs(rate) : R(abs((int)rate))) > R(20);
}

// Compute_Ion; s[0..25] = reference State (s[0] overwritten with V).
template <typename R>
EP_HD R mh_compute_ion(R s[26], R V, R istim_pApF, R dt, const R *__restrict__ c,
                                            int abs_mode, int &substepped) {
    R r[26];
    s[0] = V;
    mh_rhs(s, c, dt, istim_pApF, r);
    if (mh_wants_substeps(r[0], abs_mode)) {
        const R h = dt / R(10);
#pragma unroll 1
        for (int k = 0; k < 10; k++) {
            mh_rhs(s, c, h, istim_pApF, r);
#pragma unroll
            for (int j = 0; j < 26; j++) s[j] += r[j] * h;
        }
        substepped = 1;
    } else {
#pragma unroll
        for (int j = 0; j < 26; j++) s[j] += r[j] * dt;
        substepped = 0;
    }
    return r[0];
}

}  // namespace ep
