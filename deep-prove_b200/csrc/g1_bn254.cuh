// BN254 G1 (y^2 = x^3 + 3 over Fq): affine points and sums of points, the additions the bucket method needs.
// A sum is held as (X, Y, ZZ, ZZZ) with x = X / ZZ, y = Y / ZZZ and ZZ^3 = ZZZ^2 (the "XYZZ" coordinates of the
// Explicit-Formulas Database): adding an affine point takes 10 products where Jacobian coordinates take 11, adding
// two sums 14 instead of 16, and two of them share a reduction.  The point at infinity is ZZ = 0 in a sum (all words
// zero, as the functions here make it) and (0, 0) in affine coordinates ((0, 0) is not on the curve).
#pragma once
#include "fq_bn254.cuh"

namespace dpb {

struct G1Affine {
    Fq x, y;  // Montgomery form
};
struct G1Sum {
    Fq X, Y, ZZ, ZZZ;
};

DPB_HD G1Sum g1_infinity() {
    G1Sum p;
    p.X = p.Y = p.ZZ = p.ZZZ = fq_zero();
    return p;
}
DPB_HD bool g1_is_infinity(const G1Sum& p) { return fq_is_zero(p.ZZ); }
DPB_HD bool g1_affine_is_infinity(const G1Affine& p) { return fq_is_zero(p.x) && fq_is_zero(p.y); }
DPB_HD G1Sum g1_from_affine(const G1Affine& p) {
    if (g1_affine_is_infinity(p)) return g1_infinity();
    G1Sum r;
    r.X = p.x;
    r.Y = p.y;
    r.ZZ = r.ZZZ = fq_one();
    return r;
}
DPB_HD G1Affine g1_affine_neg(const G1Affine& p) {
    G1Affine r;
    r.x = p.x;
    r.y = fq_neg(p.y);
    return r;
}

// 2 P for a = 0 (dbl-2008-s-1: 6 products, 3 squarings)
DPB_HD G1Sum g1_double(const G1Sum& p) {
    if (g1_is_infinity(p)) return p;
    const Fq U = fq_dbl(p.Y), V = fq_sqr(U), W = fq_mul(U, V), S = fq_mul(p.X, V);
    const Fq XX = fq_sqr(p.X), M = fq_add(fq_dbl(XX), XX);
    G1Sum r;
    r.X = fq_sub(fq_sqr(M), fq_dbl(S));
    r.Y = fq_mul_sub_mul(M, fq_sub(S, r.X), W, p.Y);
    r.ZZ = fq_mul(V, p.ZZ);
    r.ZZZ = fq_mul(W, p.ZZZ);
    return r;
}

// The tail both additions share: P = U2 - U1, R = S2 - S1; the sum's X and Y from U1, S1, PP = P^2, PPP = P^3
DPB_HD void g1_add_xy(const Fq& U1, const Fq& S1, const Fq& R, const Fq& PP, const Fq& PPP, Fq& X, Fq& Y) {
    const Fq Q = fq_mul(U1, PP);
    X = fq_sub(fq_sub(fq_sqr(R), PPP), fq_dbl(Q));
    Y = fq_mul_sub_mul(R, fq_sub(Q, X), S1, PPP);
}

// P + Q, Q affine (madd-2008-s: 8 products, 2 squarings); every special case handled
DPB_HD G1Sum g1_add_mixed(const G1Sum& p, const G1Affine& q) {
    if (g1_affine_is_infinity(q)) return p;
    if (g1_is_infinity(p)) return g1_from_affine(q);
    const Fq P = fq_sub(fq_mul(q.x, p.ZZ), p.X), R = fq_sub(fq_mul(q.y, p.ZZZ), p.Y);
    if (fq_is_zero(P)) {
        if (fq_is_zero(R)) return g1_double(p);  // the same point
        return g1_infinity();                    // opposite points
    }
    const Fq PP = fq_sqr(P), PPP = fq_mul(P, PP);
    G1Sum r;
    g1_add_xy(p.X, p.Y, R, PP, PPP, r.X, r.Y);
    r.ZZ = fq_mul(p.ZZ, PP);
    r.ZZZ = fq_mul(p.ZZZ, PPP);
    return r;
}

// P + Q (add-2008-s: 12 products, 2 squarings)
DPB_HD G1Sum g1_add(const G1Sum& p, const G1Sum& q) {
    if (g1_is_infinity(p)) return q;
    if (g1_is_infinity(q)) return p;
    const Fq U1 = fq_mul(p.X, q.ZZ), S1 = fq_mul(p.Y, q.ZZZ);
    const Fq P = fq_sub(fq_mul(q.X, p.ZZ), U1), R = fq_sub(fq_mul(q.Y, p.ZZZ), S1);
    if (fq_is_zero(P)) {
        if (fq_is_zero(R)) return g1_double(p);
        return g1_infinity();
    }
    const Fq PP = fq_sqr(P), PPP = fq_mul(P, PP);
    G1Sum r;
    g1_add_xy(U1, S1, R, PP, PPP, r.X, r.Y);
    r.ZZ = fq_mul(fq_mul(p.ZZ, q.ZZ), PP);
    r.ZZZ = fq_mul(fq_mul(p.ZZZ, q.ZZZ), PPP);
    return r;
}

// k P for a small k, double-and-add from the top bit
DPB_HD G1Sum g1_mul_small(const G1Sum& p, uint32_t k) {
    G1Sum r = g1_infinity();
    int top = 31;
    while (top >= 0 && !((k >> top) & 1)) top--;
    for (int b = top; b >= 0; b--) {
        r = g1_double(r);
        if ((k >> b) & 1) r = g1_add(r, p);
    }
    return r;
}

// affine coordinates (one inversion)
DPB_HD G1Affine g1_to_affine(const G1Sum& p) {
    G1Affine r;
    if (g1_is_infinity(p)) {
        r.x = r.y = fq_zero();
        return r;
    }
    const Fq i = fq_inv(fq_mul(p.ZZ, p.ZZZ));
    r.x = fq_mul(p.X, fq_mul(i, p.ZZZ));
    r.y = fq_mul(p.Y, fq_mul(i, p.ZZ));
    return r;
}

DPB_HD bool g1_affine_on_curve(const G1Affine& p) {
    if (g1_affine_is_infinity(p)) return true;
    return fq_eq(fq_sqr(p.y), fq_add(fq_mul(fq_sqr(p.x), p.x), fq_three()));
}

}  // namespace dpb
