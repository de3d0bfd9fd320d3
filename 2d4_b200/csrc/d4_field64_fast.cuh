// d4_field64_fast.cuh: the wall field of d4_field64.cuh for the mixed form's
// FP64 sweeps, without the reference's operation order.
//
// Same images, blends and branches as d4::f64 (src/Fields/Field.cpp:172-346):
// images -3..3 summed exactly, the images +-4 and -+5 blended linearly in dx,
// the hyperbolic values of 2*pi*(dx +- i) from one e = exp(2*pi*dx) with the
// addition theorems.  Each image's quotients are formed from one reciprocal
// r = 1 / (ch - c) (f_l = dx2pi (ch c - 1) r^2 pi and its x-derivative from r^2
// and r^3), the field and its derivative share those reciprocals, and the
// translation unit that includes this file contracts product-adds.  The result
// is within a few ulps of the exact-order form: the mixed form's accuracy bar
// (positions per step against the FP64 form) has room for it, the plain form's
// bit parity does not, so only the mixed form's sweeps use it.  The Taylor
// branches near the pair's own origin stay those of d4::f64.
#pragma once

#include "d4_field64.cuh"

namespace d4 {
namespace f64fast {

using f64::cos2piy;
using f64::exp2pix;
using f64::kPi;
using f64::normalize;
using f64::weight;
using f64::weight_inv;

constexpr double k2Pi2 = 2 * f64::kPi * f64::kPi;

// cosh/sinh of 2*pi*(dx +- i) from e = exp(2*pi*dx) and one reciprocal.
struct Hyp {
    double ch0, sh0, chp1, chm1, shp1, shm1, chp2, chm2, shp2, shm2;
    double chp3, chm3, chp4, chm4, chp5, chm5;
    __device__ __forceinline__ explicit Hyp(double e) {
        const double inv = f64::recip(e);
        const double s = (e + inv) * 0.5, d = (e - inv) * 0.5;
        ch0 = s;
        sh0 = d;
        chp1 = s * f64::kCosh2Pi + d * f64::kSinh2Pi;
        chm1 = s * f64::kCosh2Pi - d * f64::kSinh2Pi;
        shp1 = d * f64::kCosh2Pi + s * f64::kSinh2Pi;
        shm1 = d * f64::kCosh2Pi - s * f64::kSinh2Pi;
        chp2 = s * f64::kCosh4Pi + d * f64::kSinh4Pi;
        chm2 = s * f64::kCosh4Pi - d * f64::kSinh4Pi;
        shp2 = d * f64::kCosh4Pi + s * f64::kSinh4Pi;
        shm2 = d * f64::kCosh4Pi - s * f64::kSinh4Pi;
        chp3 = f64::kCosh6Pi * e;
        chm3 = f64::kCosh6Pi * inv;
        chp4 = f64::kCosh8Pi * e;
        chm4 = f64::kCosh8Pi * inv;
        chp5 = f64::kCoshTPi * e;
        chm5 = f64::kCoshTPi * inv;
    }
};

// One image: f_l and, with kGrad, f_dx_l (sh = ch for |i| >= 3), from r = 1/q
// (within an ulp: Newton steps from the hardware's estimate).
template <bool kGrad>
__device__ __forceinline__ void image(double u, double c, double ch, double sh, double &f,
                                      double &g) {
    const double r = f64::recip(ch - c);
    const double n1 = ch * c - 1, w = n1 * (r * r);
    f = k2Pi2 * u * w;
    if (kGrad) g = (w + (2 * kPi) * u * (sh * c * (r * r) - 2 * sh * (w * r))) * k2Pi2;
}

// Field::xy and, with kGrad, Field::xy_diff_x over the same images and blends as
// d4::f64::pair.
template <bool kGrad>
__device__ __forceinline__ void pair(double dx, double dy, double &f, double &g) {
    const double c = cos2piy(dy);
    const Hyp h(exp2pix(dx));
    double t, u;
    image<kGrad>(dx + 3, c, h.chp3, h.chp3, f, g);
    auto add = [&](double v, double ch, double sh) {
        image<kGrad>(v, c, ch, sh, t, u);
        f += t;
        if (kGrad) g += u;
    };
    add(dx - 3, h.chm3, h.chm3);
    add(dx + 2, h.chp2, h.shp2);
    add(dx - 2, h.chm2, h.shm2);
    add(dx + 1, h.chp1, h.shp1);
    add(dx - 1, h.chm1, h.shm1);
    if (dx * dx + dy * dy > 1e-6) {
        add(dx, h.ch0, h.sh0);
    } else {
        f += f64::f_0(dx, c, dy, h.ch0);
        if (kGrad) g += f64::f_dx_0(dx, c, dy, h.ch0, h.sh0);
    }
    const bool neg = dx < 0;
    const double far = fabs(dx), sg = neg ? -1.0 : 1.0;
    const double ch5 = neg ? h.chp5 : h.chm5, ch4b = neg ? h.chm4 : h.chp4;
    add(dx - 4 * sg, neg ? h.chp4 : h.chm4, neg ? h.chp4 : h.chm4);
    image<kGrad>(dx - 5 * sg, c, ch5, ch5, t, u);
    f += t * far;
    if (kGrad) g += u * far + t * sg;
    image<kGrad>(dx + 4 * sg, c, ch4b, ch4b, t, u);
    f += t * (1 - far);
    if (kGrad) g += u * (1 - far) - t * sg;
}

}  // namespace f64fast
}  // namespace d4
