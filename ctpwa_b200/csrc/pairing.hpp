// Which compact angular tables the samples allow, from maxima over their events.
#pragma once

#include <algorithm>

namespace ctpwa {

struct Pairing {
    bool pairs = false;   // SL_{c,npol-1-q} = conj(SL_{c,q}) in every plane
    bool reals = false;   // and the polarisation paired with itself is real, or imaginary, in all planes alike
    bool mid_im = false;  // imaginary
};

// maxima: per plane c and pair q |SL_{c,npol-1-q} - conj(SL_{c,q})| and the
// same with a plus sign, [nplane][npol / 2][2], then per plane |SL| and |Re SL|,
// |Im SL| of the polarisation paired with itself (npol odd), [nplane][3].
// Pairs are compared to 1e-12 of the largest |SL|. The component of the
// self-paired polarisation that the table of reals drops is compared plane by
// plane, to 1e-12 of the plane's own largest |SL|: a plane whose values are
// small against the others' would else lose digits of its own. (A component
// below four roundings of the largest |SL| of all planes counts as dropped too:
// planes whose terms cancel hold rounding errors of either kind only.)
inline Pairing pairingOf(int nplane, int npol, const double* maxima)
{
    Pairing r;
    const int npair = npol / 2;
    const double* plane = maxima + 2 * nplane * npair;
    double big = 0.0;
    for (int c = 0; c < nplane; ++c) big = std::max(big, plane[3 * c]);
    // the paired kernels rebuild conjugates with a plus sign
    r.pairs = npair > 0 && big > 0.0;
    for (int i = 0; i < nplane * npair; ++i) r.pairs = r.pairs && maxima[2 * i] <= 1e-12 * big;
    if (!r.pairs) return r;
    bool re = true, im = true;  // real, imaginary in all planes
    if (npol % 2)
        for (int c = 0; c < nplane; ++c) {
            const double tol = std::max(1e-12 * plane[3 * c], 4 * 2.2e-16 * big);
            re = re && plane[3 * c + 2] <= tol;
            im = im && plane[3 * c + 1] <= tol;
        }
    r.reals = re || im;
    r.mid_im = !re;
    return r;
}

}  // namespace ctpwa
