// Polynomials of the pair factor for the FP64 pair kernel.
//
// A pair at separation r contributes F = g(x) / r^3 times its offset, x = r / (2 r_s),
// g(x) = erfc(x) + (2/sqrt(pi)) x exp(-x^2). With a cutoff, x is bounded, and F
// is formed from y = 1/r without erfc, a division or a library exp:
//   near (r^2 below `near2`, x below about 1): g = 1 - x^3 H(x^2), H entire:
//     F = y^3 + P(r^2), P = -H / (2 r_s)^3. g is above 0.55 there, so the
//     difference costs less than one bit;
//   far: g = exp(-x^2) K(x), K(x) = exp(x^2) erfc(x) + (2/sqrt(pi)) x, which lies
//     between 1.5 and x + 1 and is smooth: F = y^3 2^n Q(f) K(r), where
//     -x^2 log2(e) = n + f, n whole, |f| <= 1/2, Q = 2^f. Every factor keeps
//     its relative accuracy however small g is.
// P, K and Q are interpolated at Chebyshev nodes in long double and stored as
// monomials about the middle of their range; the coefficient counts keep the
// interpolation below kFit64Tol of the result.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

namespace p2p {

constexpr int kFit64Near = 12;     // coefficients of P
constexpr int kFit64Exp = 12;      // coefficients of Q
constexpr int kFit64MaxFar = 25;   // most coefficients of K
constexpr long double kFit64Tol = 4.0e-17L;  // about a third of half an ulp
constexpr long double kFit64Pi = 3.14159265358979323846264338327950288L;

// Passed by value with the kernel's arguments: no device copy to keep.
struct Fit64 {
    int nfar;  // coefficients of K; 0: no fit (no cutoff, or one out of range): the general kernel runs
    // high words of r^2: below hi_near a near pair; below hi_in surely inside
    // the cutoff; above hi_out (and finite) surely beyond it
    uint32_t hi_near, hi_in, hi_out;
    double near_mid, far_mid;  // centres: P in r^2 - near_mid, K in r - far_mid
    double e_hi, e_lo;         // -log2(e) / (2 r_s)^2 in two parts
    double near[kFit64Near], far[kFit64MaxFar], exp2[kFit64Exp];
};

inline uint32_t fit64_hi(double v) {
    uint64_t b;
    std::memcpy(&b, &v, 8);
    return (uint32_t)(b >> 32);
}
inline double fit64_from_hi(uint32_t hi) {
    const uint64_t b = (uint64_t)hi << 32;
    double v;
    std::memcpy(&v, &b, 8);
    return v;
}

// H(u) = (4/sqrt(pi)) sum (-u)^n / (n! (2n + 3)); u up to about 2.
inline long double fit64_h(long double u) {
    long double term = 1.0L, sum = 0.0L;
    for (int n = 0; n < 60; ++n) {
        sum += term / (2 * n + 3);
        term *= -u / (n + 1);
    }
    return 4.0L / std::sqrt(kFit64Pi) * sum;
}

inline long double fit64_k(long double x) {
    return std::exp(x * x) * std::erfc(x) + 2.0L / std::sqrt(kFit64Pi) * x;
}

// Interpolates f on [lo, hi] with n monomials in v - mid; returns the largest
// error relative to floor (absolute when floor is 0: relative to f itself).
template <class Fn>
long double fit64_poly(Fn f, long double lo, long double hi, long double mid, int n, long double floor, double *out) {
    long double node[kFit64MaxFar], val[kFit64MaxFar], mono[kFit64MaxFar];
    const long double half = 0.5L * (hi - lo), c = 0.5L * (hi + lo);
    for (int j = 0; j < n; ++j) {
        node[j] = std::cos(kFit64Pi * (j + 0.5L) / n);  // in [-1, 1]
        val[j] = f(c + half * node[j]);
    }
    // Newton's divided differences, then expanded into monomials about mid
    for (int j = 1; j < n; ++j)
        for (int i = n - 1; i >= j; --i) val[i] = (val[i] - val[i - 1]) / (node[i] - node[i - j]);
    const long double shift = (c - mid) / half;  // (v - mid) / half = node variable + shift
    for (int m = 0; m < n; ++m) mono[m] = 0.0L;
    mono[0] = val[n - 1];
    for (int i = n - 2; i >= 0; --i) {
        for (int m = n - 1; m > 0; --m) mono[m] = mono[m - 1] - (node[i] + shift) * mono[m];
        mono[0] = val[i] - (node[i] + shift) * mono[0];
    }
    long double err = 0.0L;
    for (int q = 0; q <= 48; ++q) {
        const long double v = lo + (hi - lo) * q / 48.0L, s = (v - mid) / half, want = f(v);
        long double p = mono[n - 1];
        for (int m = n - 2; m >= 0; --m) p = p * s + mono[m];
        const long double e = std::fabs(p - want) / (floor > 0.0L ? floor : std::fabs(want));
        if (!(e <= err)) err = e;
    }
    long double scale = 1.0L;
    for (int m = 0; m < n; ++m) {
        out[m] = (double)(mono[m] * scale);
        if (!std::isfinite(out[m]) || (out[m] != 0.0 && std::fabs(out[m]) < 1e-290)) err = 1.0L;
        scale /= half;
    }
    return err;
}

// The fit for a cutoff at x = x_cut, split radius r_s and softening (box units).
inline Fit64 fit64(double x_cut, double split_radius, double soften) {
    Fit64 F;
    std::memset(&F, 0, sizeof(F));
    // cutoffs with a far range to speak of; softenings whose squares and
    // inverse cubes are ordinary numbers
    if (!(x_cut >= 1.25 && x_cut <= 4.0) || !(split_radius > 1e-30 && split_radius < 1e30) || !(soften > 1e-60))
        return F;
    const long double kx = 0.5L / (long double)split_radius, k2 = kx * kx;
    const double rcut2 = (double)((long double)x_cut * x_cut / k2);
    F.hi_near = fit64_hi((double)(0.98L / k2));
    F.hi_in = fit64_hi(rcut2 * (1.0 - 1e-13));
    F.hi_out = fit64_hi(rcut2 * (1.0 + 1e-13));
    const double near2 = fit64_from_hi(F.hi_near), r_near = std::sqrt(near2), r_cut = std::sqrt(rcut2);
    F.near_mid = 0.5 * near2;
    F.far_mid = 0.5 * (r_near + r_cut);
    const long double e = -1.44269504088896340735992468100189214L * k2;
    F.e_hi = (double)e;
    F.e_lo = (double)(e - (long double)F.e_hi);
    // near: F is at least its value at the far end, 0.55 in units of 1 / (2 r_s)^3
    if (!(fit64_poly([&](long double v) { return -fit64_h(v * k2) * kx * k2; }, 0.0L, near2, F.near_mid, kFit64Near,
                     0.55L * kx * k2, F.near) <= kFit64Tol))
        return F;
    if (!(fit64_poly([](long double v) { return std::exp2(v); }, -0.5L, 0.5L, 0.0L, kFit64Exp, 0.0L, F.exp2) <= kFit64Tol))
        return F;
    const int counts[] = {17, 19, 22, kFit64MaxFar};
    for (int n : counts) {
        if (fit64_poly([&](long double v) { return fit64_k(v * kx); }, r_near * (1.0L - 1e-12L), r_cut * (1.0L + 1e-12L),
                       F.far_mid, n, 0.0L, F.far) <= kFit64Tol) {
            F.nfar = n;
            break;
        }
    }
    return F;
}

// The fit with the three numbers that it was made for. A fit takes 0.1 to 0.2 ms on
// the host, and a caller may set its parameters before every pass (PhotoNs' entry
// points do), mostly to the same numbers.
class Fit64For {
  public:
    // Makes the fit unless it is there; whether it was made.
    bool set(double x_cut, double split_radius, double soften) {
        if (made_ && x_cut == of_[0] && split_radius == of_[1] && soften == of_[2]) return false;
        fit_ = fit64(x_cut, split_radius, soften);
        of_[0] = x_cut;
        of_[1] = split_radius;
        of_[2] = soften;
        return made_ = true;
    }
    const Fit64 &fit() const { return fit_; }

  private:
    Fit64 fit_{};
    double of_[3] = {0.0, 0.0, 0.0};
    bool made_ = false;
};

}  // namespace p2p
