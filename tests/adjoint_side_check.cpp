// Which side's tangential velocity the HLLC flux carries, in the forward and in its reverse.
//
// The forward takes the L side's velocity for f1 >= 0, else the R side's, and the derivative of f3
// with respect to the tangential discharges shows which one its reverse took.  f1 is brought to where
// it changes sign, to the last bit of the left discharge, and the two are compared on both sides of
// that place.  With blending, f1 is a sum of two rounded quotients: its sign there is a matter of
// their last bits.
//
// Output: one line per topography, "name samples differing".
#include <cmath>
#include <cstdio>
#include <random>

#include "sp_adjoint.cuh"

using namespace sw2d;

static std::mt19937_64 rng(2024);
static double U(double a, double b) { return std::uniform_real_distribution<double>(a, b)(rng); }

struct Sample {
    bool blending;
    double phiL, phiR, zbL, zbR;
    SideState L, R;
    double f1(double q) const
    {
        SideState s = L;
        s.q = q;
        return hllc(blending, 1.0, 1.0, phiL, phiR, zbL, zbR, s, R, 1e-5, 1e-3).f1;
    }
    // the side the reverse takes: 0 L, 1 R
    int reverse_side(double q) const
    {
        SideState s = L;
        s.q = q;
        EdgeFlux fb{};
        fb.f3 = 1.0;
        SideBar Lb{0, 0, 0, 0, 0}, Rb{0, 0, 0, 0, 0};
        double zbLb = 0.0, zbRb = 0.0;
        hllc_rev(blending, 1.0, 1.0, phiL, phiR, zbL, zbR, s, R, 1e-5, 1e-3, fb, Lb, Rb, zbLb, zbRb);
        return Lb.r != 0.0 ? 0 : Rb.r != 0.0 ? 1 : -1;
    }
};

int main()
{
    for (int blending = 0; blending < 2; blending++) {
        int n = 0, differ = 0;
        for (int it = 0; it < 20000; it++) {
            Sample s;
            s.blending = blending != 0;
            s.phiL = U(0.5, 1.0);
            s.phiR = U(0.5, 1.0);
            s.zbL = U(0.0, 0.5);
            s.zbR = U(0.0, 0.5);
            const double hL = U(0.5, 1.5), hR = U(0.5, 1.5), c = std::sqrt(kGravity);
            s.L.z = hL + s.zbL;
            s.R.z = hR + s.zbR;
            s.L.r = U(0.5, 1.0);
            s.R.r = U(0.5, 1.0);
            s.R.q = U(-0.5, 0.5);
            s.L.lm = -c * std::sqrt(hL);
            s.L.lp = c * std::sqrt(hL);
            s.R.lm = -c * std::sqrt(hR);
            s.R.lp = c * std::sqrt(hR);
            double lo = -20.0, hi = 20.0;
            if (!(s.f1(lo) < 0.0 && s.f1(hi) > 0.0)) continue;
            for (int k = 0; k < 200 && std::nextafter(lo, hi) < hi; k++) {
                const double mid = lo + 0.5 * (hi - lo);
                if (s.f1(mid) < 0.0) lo = mid;
                else hi = mid;
            }
            double q = lo;
            for (int k = 0; k < 4; k++) q = std::nextafter(q, -1e9);
            for (int k = 0; k < 10; k++, q = std::nextafter(q, 1e9)) {
                const double f = s.f1(q);
                if (f == 0.0) continue;  // the reverse's derivative by r is zero on either side
                const int side = s.reverse_side(q);
                if (side < 0) continue;
                n++;
                if (side != (f >= 0.0 ? 0 : 1)) differ++;
            }
        }
        std::printf("%s %d %d\n", blending ? "blending" : "discontinuous", n, differ);
    }
    return 0;
}
