// The limiter's reverse under adjoints near the end of the range, on the host.
//
// Over still water a state adjoint can grow until it overflows (the gradient's entries there are counted
// and set to zero).  How far that spreads is a matter of the order of the products: where the limiter's
// factor is zero, because the cell itself holds the bound, its neighbours in the list get nothing, and
// 0 * inf must not arise.  The reverse written with plain divisions is the measure: an entry that is
// finite there has to be finite here.
//
// Output, one line per number of neighbours: "n entries nonfinite_there lost".
#include <cmath>
#include <cstdio>
#include <random>

#include "sp_adjoint.cuh"

using namespace sw2d;

static std::mt19937_64 rng(99);
static double U(double a, double b) { return std::uniform_real_distribution<double>(a, b)(rng); }

static void plain_reverse(double zc, int n, const SlopeNbr* nb, double sxb, double syb, double& zcb, double* zjb)
{
    double sx, sy, sxk[kMaxNbr], syk[kMaxNbr];
    slopes_fwd(zc, n, nb, sx, sy, sxk, syk);
    for (int k = 0; k < n; k++) zjb[k] = 0.0;
    for (int k = n - 1; k >= 0; k--) {
        const double zL = nb[k].c_is_r ? nb[k].zj : zc, zR = nb[k].c_is_r ? zc : nb[k].zj;
        const bool max_left = !(zL < zR), min_left = !(zR < zL);
        const double top = max_left ? zL : zR, low = min_left ? zL : zR;
        const double rec = zc + nb[k].ax * sxk[k] + nb[k].ay * syk[k];
        if (!(rec < low) && !(rec > top)) continue;
        const bool left = rec < low ? min_left : max_left;
        const double f = rec < low ? low : top, den = rec - zc, fac = (f - zc) / den;
        const double fac_bar = sxb * sxk[k] + syb * syk[k];
        const double num_bar = fac_bar / den, den_bar = -fac_bar * fac / den;
        if (left != nb[k].c_is_r) zcb += num_bar;
        else zjb[k] += num_bar;
        zcb -= num_bar;
        sxb = sxb * fac + den_bar * nb[k].ax;
        syb = syb * fac + den_bar * nb[k].ay;
    }
    double wsum = 0.0;
    for (int k = 0; k < n; k++) wsum += 1.0 / std::sqrt(nb[k].dx * nb[k].dx + nb[k].dy * nb[k].dy);
    for (int k = 0; k < n; k++) {
        const double d = std::sqrt(nb[k].dx * nb[k].dx + nb[k].dy * nb[k].dy), w = 1.0 / d;
        const double t = sxb / wsum * (nb[k].dx / d / d * w) + syb / wsum * (nb[k].dy / d / d * w);
        zjb[k] += t;
        zcb -= t;
    }
}

int main()
{
    for (int n = 2; n <= 6; n++) {
        int entries = 0, nonfinite = 0, lost = 0;
        for (int it = 0; it < 40000; it++) {
            SlopeNbr nb[kMaxNbr];
            const double zc = U(-1, 1);
            for (int k = 0; k < n; k++) {
                const double a = 6.283 * k / n + U(-0.3, 0.3), d = U(0.5, 1.5);
                nb[k].dx = d * std::cos(a);
                nb[k].dy = d * std::sin(a);
                nb[k].ax = 0.5 * nb[k].dx + U(-0.1, 0.1);
                nb[k].ay = 0.5 * nb[k].dy + U(-0.1, 0.1);
                nb[k].c_is_r = (it >> k) & 1;
                const double r = U(0, 1);  // levels far apart, nearly level (the still lake), level
                nb[k].zj = r < 0.4 ? zc + U(-1, 1) : r < 0.8 ? zc + U(-1, 1) * std::pow(10.0, -U(1, 16)) : zc;
            }
            const double mag = std::pow(10.0, U(280, 308));
            const double sxb = U(-1, 1) * mag, syb = U(-1, 1) * mag;
            double za = 0.0, zb = 0.0, ja[kMaxNbr + 1], jb[kMaxNbr + 1];
            plain_reverse(zc, n, nb, sxb, syb, za, ja);
            slopes_rev(zc, n, nb, sxb, syb, zb, jb);
            ja[n] = za;
            jb[n] = zb;
            for (int k = 0; k <= n; k++) {
                entries++;
                if (!std::isfinite(ja[k])) nonfinite++;
                else if (!std::isfinite(jb[k])) lost++;
            }
        }
        std::printf("%d %d %d %d\n", n, entries, nonfinite, lost);
    }
    return 0;
}
