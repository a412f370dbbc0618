// nf_bodies.cuh -- the per-node and per-element arithmetic of the timestep, shared by the
// single-scene kernels (k_step.cu, k_mixed.cu) and the batched kernel (k_batch.cu). One copy
// of each body means a batched instance computes exactly what a single scene does.
#pragma once

#include "nf_internal.h"
#include "nf_fpconv.h"

namespace nf {

// A product on the integer units or on the FP64 pipe (with `bad`: nf_mul_try's convention).
template <bool INT> struct Product;
template <> struct Product<true> {
    static __device__ __forceinline__ double of(double a, double b, uint32_t *bad) {
        return nf_mul_try(a, b, bad);
    }
    static __device__ __forceinline__ double of(double a, double b) { return nf_mul(a, b); }
};
template <> struct Product<false> {
    static __device__ __forceinline__ double of(double a, double b, uint32_t *) { return a * b; }
    static __device__ __forceinline__ double of(double a, double b) { return a * b; }
};

// One node of nodalUpdate, ExplicitSolver.java:998-1062, with RigidWall.hold/crosses/arrive/
// slide (RigidWall.java:163-259): shared by the single-scene kernel and the batched one. Adds
// the node's wall terms to impulse/loss/fric. When geo.pMid is set (the mixed form) it also
// writes the FP32 geometry of the coming assembly: mid-step and current positions as float
// pairs (hi, lo) and v dt, at index geo.base + i.
struct NodalCoef {
    double decay, gain, dtAvg, dt;
};
struct WallRef {
    int present;
    double plane, friction;
    int *contact, *stuck;
};
struct MixedGeo {
    float4 *pMid, *pCur;
    float2 *vdt;
    int base;
};

// With INT (int_products) the products run on the integer units: the update is two dozen FP64
// instructions a node otherwise, which bound it. 1M nodes of the mixed form: 71 us with all of
// them on the FP64 pipe, 54 us so (76 and 59 us between events), bound by the dozen additions
// left and by the loads. A product by a decay of 1 (no damping) is its factor, and -0.5 dt v is
// -(v dt) / 2 exactly.
template <bool INT>
static __device__ __forceinline__ void nodal_node(const Dev &d, int i, const NodalCoef &co,
                                                  const WallRef &w, const MixedGeo &geo,
                                                  uint32_t *status, double &impulse,
                                                  double &loss, double &fric) {
    using P = Product<INT>;
    const double decay = co.decay, gain = co.gain, dtAvg = co.dtAvg, dt = co.dt;
    const bool undamped = __double_as_longlong(decay) == __double_as_longlong(1.0);
    uint8_t fl = d.flags[i];
    const bool fixedR = fl & 1, fixedZ = fl & 2;
    bool onWall = fl & 4;
    double2 u = d.U[i], v = d.V[i];
    const double2 f = d.F[i];
    const double m = d.mass[i];
    const double invM = d.invMass[i];
    const bool resting = w.present && onWall && f.y <= 0.0;
    uint8_t ws = 0;
    double stepR = 0.0, stepZ = 0.0;                     // v dt, where it moved the node
    if (fixedR) {
        v.x = 0.0;
    } else if (resting && w.friction > 0.0) {
        // RigidWall.slide, RigidWall.java:236-259
        const double normal = -f.y;
        const double trial = nf_div(-m * decay * v.x, gain) - f.x;
        const double limit = isinf(w.friction) ? INFINITY : w.friction * normal;
        if (fabs(trial) <= limit) {
            loss += 0.5 * m * v.x * v.x;
            atomicAdd(w.stuck, 1);
            ws |= NF_WALL_STUCK;
            v.x = 0.0;
        } else {
            const double tangential = copysign(limit, trial);
            const double slid = decay * v.x + nf_div(gain * (f.x + tangential), m);
            fric += -tangential * slid * dt;
            ws |= NF_WALL_SLID;
            v.x = slid;
        }
        stepR = v.x * dt;
        u.x += stepR;
    } else {
        v.x = (undamped ? v.x : P::of(decay, v.x)) + P::of(P::of(gain, f.x), invM);
        stepR = P::of(v.x, dt);
        u.x += stepR;
    }
    const double2 x0 = d.X0[i];
    if (fixedZ) {
        v.y = 0.0;
    } else if (resting) {
        impulse += -f.y * dtAvg;                         // RigidWall.hold :178-181
        atomicAdd(w.contact, 1);
        ws |= NF_WALL_HELD;
        stepZ = v.y * dt;                                // the geometry's v dt only
    } else {
        const double trial = (undamped ? v.y : P::of(decay, v.y)) + P::of(P::of(gain, f.y), invM);
        stepZ = P::of(trial, dt);
        if (w.present && less_bits(x0.y + u.y + stepZ, w.plane)) {
            impulse += -m * trial;                       // RigidWall.arrive :205-209
            loss += 0.5 * m * trial * trial;
            atomicAdd(w.contact, 1);
            u.y += w.plane - (x0.y + u.y);
            v.y = 0.0;
            stepZ = 0.0;
            onWall = true;
            ws |= NF_WALL_ARRIVED;
        } else {
            v.y = trial;
            u.y += stepZ;
            if (w.present) onWall = false;
        }
    }
    d.U[i] = u;
    d.V[i] = v;
    if (w.present) {
        d.flags[i] = (uint8_t)((fl & 3) | (onWall ? 4 : 0));
        d.wallState[i] = ws;
    }
    if (!(finite_bits(u.x) && finite_bits(u.y) && finite_bits(v.x) && finite_bits(v.y)))
        atomicOr(status, STATUS_NONFINITE);
    if (geo.pMid) {
        // the geometry of the coming assembly: mid-step and current positions as float
        // pairs, and v dt (see k_prepare_mixed)
        const double xr = x0.x + u.x, xz = x0.y + u.y;
        double pr = x0.x, pz = x0.y;
        if (d.finite) {
            pr = xr - nf_scale2(stepR, -1);
            pz = xz - nf_scale2(stepZ, -1);
        }
        const float2 sr = nf_split(pr), sz = nf_split(pz);
        geo.pMid[geo.base + i] = make_float4(sr.x, sr.y, sz.x, sz.y);
        if (geo.pCur) {
            const float2 qr = nf_split(xr), qz = nf_split(xz);
            geo.pCur[geo.base + i] = make_float4(qr.x, qr.y, qz.x, qz.y);
        }
        geo.vdt[geo.base + i] = make_float2(nf_narrow(stepR), nf_narrow(stepZ));
    }
}

// The mixed form's geometry of an assembly on its own (the initial one, and steps without the
// fused nodal update): node i's mid-step and current positions as float pairs and v sdt.
static __device__ __forceinline__ void prepare_node(const Dev &d, int i, double sdt,
                                                    const MixedGeo &geo) {
    const double mid = -0.5 * sdt;
    const double2 x = d.X0[i], u = d.U[i], v = d.V[i];
    double pr, pz;
    if (d.finite) {
        pr = x.x + u.x + mid * v.x;
        pz = x.y + u.y + mid * v.y;
    } else {
        pr = x.x;
        pz = x.y;
    }
    const float2 sr = nf_split(pr), sz = nf_split(pz);
    geo.pMid[geo.base + i] = make_float4(sr.x, sr.y, sz.x, sz.y);
    if (geo.pCur) {
        const float2 qr = nf_split(x.x + u.x), qz = nf_split(x.y + u.y);
        geo.pCur[geo.base + i] = make_float4(qr.x, qr.y, qz.x, qz.y);
    }
    geo.vdt[geo.base + i] = make_float2(nf_narrow(v.x * sdt), nf_narrow(v.y * sdt));
}

// The current positions x + u of element e's four nodes (the sums cr/cz and currentArea both
// start from).
static __device__ __forceinline__ void element_current(const Dev &d, int e, double2 *cur) {
    const int4 c = d.conn[e];
    const int n[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const double2 x = d.X0[n[k]], u = d.U[n[k]];
        cur[k] = make_double2(x.x + u.x, x.y + u.y);
    }
}

// The element's kinematics of one assembly in the machine's arithmetic: mid-step coordinates,
// displacement increments, shape derivatives (d2 = -d0, d3 = -d1), Jacobian and radius.
struct ElementKin {
    double r[4], z[4], a[4], c[4];
    double d0r, d1r, d0z, d1z, det, rg;
};
static __device__ void kinematics_machine(const Dev &d, int e, double strainDt, ElementKin &k) {
    const int4 c = d.conn[e];
    const int n[4] = {c.x, c.y, c.z, c.w};
    const double mid = -0.5 * strainDt;
    for (int i = 0; i < 4; i++) {
        const double2 v = d.V[n[i]], x = d.X0[n[i]];
        if (d.finite) {                                  // cr/cz, :1176-1182
            const double2 u = d.U[n[i]];
            k.r[i] = x.x + u.x + mid * v.x;
            k.z[i] = x.y + u.y + mid * v.y;
        } else {
            k.r[i] = x.x;
            k.z[i] = x.y;
        }
        k.a[i] = v.x * strainDt;
        k.c[i] = v.y * strainDt;
    }
    const double *r = k.r, *z = k.z;
    const double J00 = 0.25 * (-r[0] + r[1] + r[2] - r[3]);
    const double J01 = 0.25 * (-z[0] + z[1] + z[2] - z[3]);
    const double J10 = 0.25 * (-r[0] - r[1] + r[2] + r[3]);
    const double J11 = 0.25 * (-z[0] - z[1] + z[2] + z[3]);
    k.det = J00 * J11 - J01 * J10;
    const double inv = 1.0 / k.det;
    k.d0r = 0.25 * (J01 - J11) * inv;
    k.d1r = 0.25 * (J01 + J11) * inv;
    k.d0z = 0.25 * (J10 - J00) * inv;
    k.d1z = -0.25 * (J10 + J00) * inv;
    k.rg = d.axi ? 0.25 * (r[0] + r[1] + r[2] + r[3]) : 0.0;
}

// What the return map starts from: strain increments, rotated stress and back stress, and the
// element's shortest squared edge folded into minEdge. The machine's arithmetic, for the
// elements whose integer forms were not settled.
static __device__ __noinline__ void strain_machine(const Dev &d, int e, double strainDt,
                                                   double *strain, double *sg, double *bk,
                                                   double *minEdge) {
    ElementKin k;
    kinematics_machine(d, e, strainDt, k);
    const double *r = k.r, *z = k.z, *a = k.a, *c = k.c;
    if (d.finite)
        *minEdge = shortestEdge(*minEdge, r[0], r[1], r[2], r[3], z[0], z[1], z[2], z[3]);
    const double d2r = -k.d0r, d3r = -k.d1r, d2z = -k.d0z, d3z = -k.d1z;
    const double dRdZ = k.d0z * a[0] + k.d1z * a[1] + d2z * a[2] + d3z * a[3];
    const double dZdR = k.d0r * c[0] + k.d1r * c[1] + d2r * c[2] + d3r * c[3];
    strain[0] = k.d0r * a[0] + k.d1r * a[1] + d2r * a[2] + d3r * a[3];
    strain[1] = k.d0z * c[0] + k.d1z * c[1] + d2z * c[2] + d3z * c[3];
    strain[2] = d.axi ? 0.25 * (a[0] + a[1] + a[2] + a[3]) / k.rg : 0.0;
    strain[3] = dRdZ + dZdR;
    for (int i = 0; i < 4; i++) {
        sg[i] = d.sig[4 * (size_t)e + i];
        bk[i] = d.back[4 * (size_t)e + i];
    }
    if (d.finite) {
        const double spinDt = 0.5 * (dZdR - dRdZ);
        if (!is_zero(spinDt)) {
            const double h = 0.5 * spinDt;
            const double cs = (1.0 - h * h) / (1.0 + h * h), sn = 2.0 * h / (1.0 + h * h);
            corot_rotate(sg, cs, sn);
            corot_rotate(bk, cs, sn);
        }
    }
}

// The force terms and the hourglass update from the new stress sg, in the machine's arithmetic.
static __device__ __noinline__ void forces_machine(const Dev &d, int e, double strainDt,
                                                   double hourglass, const double *sg) {
    ElementKin k;
    kinematics_machine(d, e, strainDt, k);
    const double *r = k.r, *z = k.z, *a = k.a, *c = k.c;
    const double dr[4] = {k.d0r, k.d1r, -k.d0r, -k.d1r}, dz[4] = {k.d0z, k.d1z, -k.d0z, -k.d1z};
    const double sR = sg[0], sZ = sg[1], sT = sg[2], sRZ = sg[3];
    const double dV = 4.0 * (d.axi ? 2.0 * NF_PI * k.rg * k.det : d.thickness * k.det);
    const double hh = d.axi ? sT / k.rg * dV * 0.25 : 0.0;
    double gr[4], gz[4];
    for (int i = 0; i < 4; i++) {
        gr[i] = d.axi ? -((dr[i] * sR + dz[i] * sRZ) * dV + hh) : -(dr[i] * sR + dz[i] * sRZ) * dV;
        gz[i] = -(dz[i] * sZ + dr[i] * sRZ) * dV;
    }
    if (hourglass > 0.0) {
        const double hr = r[0] - r[1] + r[2] - r[3];
        const double hz = z[0] - z[1] + z[2] - z[3];
        const double one[4] = {1.0, -1.0, 1.0, -1.0};
        double y[4];
        for (int i = 0; i < 4; i++) y[i] = one[i] - hr * dr[i] - hz * dz[i];
        const double kk = hourglass * d.mats[d.emat[e]].mu * dV
                          * (dr[0] * dr[0] + dr[1] * dr[1] + dr[2] * dr[2] + dr[3] * dr[3]
                             + dz[0] * dz[0] + dz[1] * dz[1] + dz[2] * dz[2] + dz[3] * dz[3]);
        double2 hg = d.hg[e];
        hg.x += kk * (y[0] * a[0] + y[1] * a[1] + y[2] * a[2] + y[3] * a[3]);
        hg.y += kk * (y[0] * c[0] + y[1] * c[1] + y[2] * c[2] + y[3] * c[3]);
        d.hg[e] = hg;
        for (int i = 0; i < 4; i++) {
            gr[i] -= y[i] * hg.x;
            gz[i] -= y[i] * hg.y;
        }
        d.hgK[e] = kk;
    }
    double *ef = d.contribution + 8 * (size_t)e;
    for (int i = 0; i < 4; i++) {
        ef[i] = gr[i];
        ef[4 + i] = gz[i];
    }
}

// -(t + f) dV and its opposite corner's -(-t - f) dV, given the rounded products t and f of the
// corner (the opposite corner's are their negatives), s = t + f and g = s dV. Negating both
// terms negates the sum unless it is a zero: equal opposite terms give +0 both times.
static __device__ __forceinline__ double opposite_force(double t, double f, double s, double g,
                                                        double dV) {
    const bool mirrored = !is_zero(s) || __double_as_longlong(t) == __double_as_longlong(f);
    return mirrored ? g : copysign(0.0, -dV);
}

// reducedIntegration, ExplicitSolver.java:1373-1504, for element e: B at the centroid, strain
// increments, Cayley co-rotation, J2/Johnson-Cook return, FB hourglass, the eight force
// terms into the element's contribution slots; folds its shortest edge into minEdge.
// *cost (when given) receives the point's Johnson-Cook cost class (j2_update). cur (when given)
// holds element_current(d, e), already formed for the erosion test.
//
// The FP64 pipe issues one warp instruction per 64 to 76 cycles on a quarter SM, whatever the
// operation, and bounds this code. So the quotients, the scalings by powers of two and, with INT,
// the products run on the integer units (nf_ifp.h) beside the additions on the FP64 pipe, in
// straight-line code. A product is 53 integer instructions: with several warps on a quarter SM they
// fill the time between its FP64 instructions; a lone warp issues them in between and is faster
// without (int_products), and so are the FP64 batches' kernels (batch_int_products). An element with any operand outside their ranges (one
// test at the end of each half) is redone by strain_machine and forces_machine. Every value has
// the bits of the reference's sequence:
//  * -0.5 dt v is -(dt v) / 2 exactly, and 2 (0.5 spin) is spin;
//  * J = S / 4 with S the corner sums and det = D / 16 with D = S00 S11 - S01 S10, so
//    0.25 (J01 - J11) / det = (S01 - S11) / D: powers of two cancel while every scaled value
//    stays normal, which bounding the S and D exponents guarantees;
//  * the derivatives of opposite corners are negatives, so are their products, and 1 - hr d2r -
//    hz d2z is (1 + hr d0r) + hz d0z with the products of corner 0.
template <bool INT>
static __device__ __forceinline__ void element_reduced(const Dev &d, int e, double strainDt,
                                                       double hourglass, double &minEdge,
                                                       int *cost = nullptr,
                                                       const double2 *cur = nullptr) {
    double *ef = d.contribution + 8 * (size_t)e;
    if (d.gone != nullptr && d.gone[e]) {
        for (int k = 0; k < 8; k++) ef[k] = 0.0;
        return;
    }
    const MatDev &fl = d.mats[d.emat[e]];
    const double lambda = fl.lambda, mu = fl.mu;
    const int4 c = d.conn[e];
    const double2 v0 = d.V[c.x], v1 = d.V[c.y], v2 = d.V[c.z], v3 = d.V[c.w];
    uint32_t bad = 0;
    const double a0 = Product<INT>::of(v0.x, strainDt, &bad), a1 = Product<INT>::of(v1.x, strainDt, &bad);
    const double a2 = Product<INT>::of(v2.x, strainDt, &bad), a3 = Product<INT>::of(v3.x, strainDt, &bad);
    const double c0 = Product<INT>::of(v0.y, strainDt, &bad), c1 = Product<INT>::of(v1.y, strainDt, &bad);
    const double c2 = Product<INT>::of(v2.y, strainDt, &bad), c3 = Product<INT>::of(v3.y, strainDt, &bad);
    double r0, r1, r2, r3, z0, z1, z2, z3;
    if (d.finite) {                                  // cr/cz, :1176-1182
        double2 p[4];
        if (cur) {
            for (int k = 0; k < 4; k++) p[k] = cur[k];
        } else {
            element_current(d, e, p);
        }
        r0 = p[0].x - nf_scale_try(a0, -1, &bad); r1 = p[1].x - nf_scale_try(a1, -1, &bad);
        r2 = p[2].x - nf_scale_try(a2, -1, &bad); r3 = p[3].x - nf_scale_try(a3, -1, &bad);
        z0 = p[0].y - nf_scale_try(c0, -1, &bad); z1 = p[1].y - nf_scale_try(c1, -1, &bad);
        z2 = p[2].y - nf_scale_try(c2, -1, &bad); z3 = p[3].y - nf_scale_try(c3, -1, &bad);
    } else {
        const double2 x0 = d.X0[c.x], x1 = d.X0[c.y], x2 = d.X0[c.z], x3 = d.X0[c.w];
        r0 = x0.x; r1 = x1.x; r2 = x2.x; r3 = x3.x;
        z0 = x0.y; z1 = x1.y; z2 = x2.y; z3 = x3.y;
    }
    const double r10 = r1 - r0, z10 = z1 - z0;
    double edge = minEdge;
    if (d.finite) {                                  // shortestEdge, :1191-1197
        const double r21 = r2 - r1, z21 = z2 - z1, r32 = r3 - r2, z32 = z3 - z2;
        const double r03 = r0 - r3, z03 = z0 - z3;
        const double e0 = Product<INT>::of(r10, r10, &bad) + Product<INT>::of(z10, z10, &bad);
        const double e1 = Product<INT>::of(r21, r21, &bad) + Product<INT>::of(z21, z21, &bad);
        const double e2 = Product<INT>::of(r32, r32, &bad) + Product<INT>::of(z32, z32, &bad);
        const double e3 = Product<INT>::of(r03, r03, &bad) + Product<INT>::of(z03, z03, &bad);
        edge = jmin_nonneg(edge, jmin_nonneg(jmin_nonneg(e0, e1), jmin_nonneg(e2, e3)));
    }
    const double S00 = r10 + r2 - r3;
    const double S01 = z10 + z2 - z3;
    const double S10 = -r0 - r1 + r2 + r3;
    const double S11 = -z0 - z1 + z2 + z3;
    const double D = Product<INT>::of(S00, S11, &bad) - Product<INT>::of(S01, S10, &bad);
    bad |= !(moderate_or_zero(S00) & moderate_or_zero(S01) & moderate_or_zero(S10) &
             moderate_or_zero(S11) & moderate_or_zero(D));
    const double invD = nf_quot_try(1.0, nf_divisor_of(D), &bad);
    const double det = nf_scale_try(D, -4, &bad);
    const double d0r = Product<INT>::of(S01 - S11, invD, &bad);
    const double d1r = Product<INT>::of(S01 + S11, invD, &bad);
    const double d0z = Product<INT>::of(S10 - S00, invD, &bad);
    const double d1z = -Product<INT>::of(S10 + S00, invD, &bad);

    double strain[4];
    strain[0] = Product<INT>::of(d0r, a0, &bad) + Product<INT>::of(d1r, a1, &bad)
                - Product<INT>::of(d0r, a2, &bad) - Product<INT>::of(d1r, a3, &bad);
    strain[1] = Product<INT>::of(d0z, c0, &bad) + Product<INT>::of(d1z, c1, &bad)
                - Product<INT>::of(d0z, c2, &bad) - Product<INT>::of(d1z, c3, &bad);
    const double dRdZ = Product<INT>::of(d0z, a0, &bad) + Product<INT>::of(d1z, a1, &bad)
                        - Product<INT>::of(d0z, a2, &bad) - Product<INT>::of(d1z, a3, &bad);
    const double dZdR = Product<INT>::of(d0r, c0, &bad) + Product<INT>::of(d1r, c1, &bad)
                        - Product<INT>::of(d0r, c2, &bad) - Product<INT>::of(d1r, c3, &bad);
    strain[3] = dRdZ + dZdR;

    double rg = 0.0;
    nf_divisor byRg{};
    strain[2] = 0.0;
    if (d.axi) {
        rg = nf_scale_try(r0 + r1 + r2 + r3, -2, &bad);
        byRg = nf_divisor_of(rg);
        strain[2] = nf_quot_try(nf_scale_try(a0 + a1 + a2 + a3, -2, &bad), byRg, &bad);
    }
    double sg[4], bk[4];
    {
        const double2 *ps = reinterpret_cast<const double2 *>(d.sig + 4 * (size_t)e);
        const double2 *pb = reinterpret_cast<const double2 *>(d.back + 4 * (size_t)e);
        const double2 s01 = ps[0], s23 = ps[1], b01 = pb[0], b23 = pb[1];
        sg[0] = s01.x; sg[1] = s01.y; sg[2] = s23.x; sg[3] = s23.y;
        bk[0] = b01.x; bk[1] = b01.y; bk[2] = b23.x; bk[3] = b23.y;
    }
    if (d.finite) {
        const double w = dZdR - dRdZ;
        const double spinDt = nf_scale_try(w, -1, &bad);
        if (!is_zero(spinDt)) {
            const double h = nf_scale_try(w, -2, &bad);
            const double hh = Product<INT>::of(h, h, &bad);
            const nf_divisor by = nf_divisor_of(1.0 + hh);
            const double cs = nf_quot_try(1.0 - hh, by, &bad), sn = nf_quot_try(spinDt, by, &bad);
            // a back stress of +0s (no kinematic hardening) rotates to itself
            const bool still = all_plus_zero(bk[0], bk[1], bk[2], bk[3]) && corot_keeps_zero(cs, sn);
            const double ccc = Product<INT>::of(cs, cs, &bad), sss = Product<INT>::of(sn, sn, &bad);
            const double csn = Product<INT>::of(cs, sn, &bad), csn2 = nf_scale_try(csn, 1, &bad);
            const double diff = ccc - sss;
            auto rotate = [&](double *t) {           // corot_rotate
                const double rr = t[0], zz = t[1], rz = t[3];
                const double shear = Product<INT>::of(csn2, rz, &bad);
                t[0] = Product<INT>::of(ccc, rr, &bad) - shear + Product<INT>::of(sss, zz, &bad);
                t[1] = Product<INT>::of(sss, rr, &bad) + shear + Product<INT>::of(ccc, zz, &bad);
                t[3] = Product<INT>::of(csn, rr - zz, &bad) + Product<INT>::of(diff, rz, &bad);
            };
            rotate(sg);
            if (!still) rotate(bk);
        }
    }
    if (bad) strain_machine(d, e, strainDt, strain, sg, bk, &minEdge);
    else minEdge = edge;

    double epsP = d.epsP[e], work = d.wP[e];
    double2 *const jcYield = d.jcYield && fl.jc ? d.jcYield + e : nullptr;
    if (d.hasDamage) {
        DamageRef dr;
        dr.failureStrain = d.dFail[e];
        dr.strength = d.dStrength + e;
        dr.softening = d.dSoft + e;
        dr.width = d.dWidth + e;
        dr.geometry = d.dGeom + 5 * (size_t)e;
        dr.fractureEnergy = d.dGf[e];
        dr.youngs = fl.youngs;
        j2_update(sg, bk, epsP, work, strain[0], strain[1], strain[2], strain[3], lambda, mu, fl,
                  strainDt, &dr, d.dStrength[e], d.dSoft[e], cost, jcYield);
    } else {
        j2_update(sg, bk, epsP, work, strain[0], strain[1], strain[2], strain[3], lambda, mu, fl,
                  strainDt, (const DamageRef *)nullptr, 0.0, 0.0, cost, jcYield);
    }
    {
        double2 *ps = reinterpret_cast<double2 *>(d.sig + 4 * (size_t)e);
        double2 *pb = reinterpret_cast<double2 *>(d.back + 4 * (size_t)e);
        ps[0] = make_double2(sg[0], sg[1]); ps[1] = make_double2(sg[2], sg[3]);
        pb[0] = make_double2(bk[0], bk[1]); pb[1] = make_double2(bk[2], bk[3]);
        d.epsP[e] = epsP;
        d.wP[e] = work;
    }
    const double sR = sg[0], sZ = sg[1], sT = sg[2], sRZ = sg[3];
    const double dV = nf_scale_try(d.axi ? Product<INT>::of(Product<INT>::of(2.0 * NF_PI, rg, &bad), det, &bad)
                                         : Product<INT>::of(d.thickness, det, &bad), 2, &bad);
    double g0r, g1r, g2r, g3r, g0z, g1z, g2z, g3z;
    {
        const double t0 = Product<INT>::of(d0r, sR, &bad), f0 = Product<INT>::of(d0z, sRZ, &bad);
        const double t1 = Product<INT>::of(d1r, sR, &bad), f1 = Product<INT>::of(d1z, sRZ, &bad);
        const double w0 = t0 + f0, w1 = t1 + f1;
        const double G0 = Product<INT>::of(w0, dV, &bad), G1 = Product<INT>::of(w1, dV, &bad);
        const double H0 = opposite_force(t0, f0, w0, G0, dV);
        const double H1 = opposite_force(t1, f1, w1, G1, dV);
        if (d.axi) {
            const double hh = nf_scale_try(Product<INT>::of(nf_quot_try(sT, byRg, &bad), dV, &bad), -2, &bad);
            g0r = -(G0 + hh);
            g1r = -(G1 + hh);
            g2r = -(hh - H0);                        // -(-G0 + hh)
            g3r = -(hh - H1);
        } else {
            g0r = -G0; g1r = -G1; g2r = H0; g3r = H1;
        }
        const double p0 = Product<INT>::of(d0z, sZ, &bad), q0 = Product<INT>::of(d0r, sRZ, &bad);
        const double p1 = Product<INT>::of(d1z, sZ, &bad), q1 = Product<INT>::of(d1r, sRZ, &bad);
        const double s0 = p0 + q0, s1 = p1 + q1;
        const double K0 = Product<INT>::of(s0, dV, &bad), K1 = Product<INT>::of(s1, dV, &bad);
        g0z = -K0; g1z = -K1;
        g2z = opposite_force(p0, q0, s0, K0, dV);
        g3z = opposite_force(p1, q1, s1, K1, dV);
    }
    double2 hg;
    double kh = 0.0;
    if (hourglass > 0.0) {
        const double hr = -r10 + r2 - r3;
        const double hz = -z10 + z2 - z3;
        const double m0 = Product<INT>::of(hr, d0r, &bad), n0 = Product<INT>::of(hz, d0z, &bad);
        const double m1 = Product<INT>::of(hr, d1r, &bad), n1 = Product<INT>::of(hz, d1z, &bad);
        const double y0 = 1.0 - m0 - n0, y2 = 1.0 + m0 + n0;
        const double y1 = -1.0 - m1 - n1, y3 = -1.0 + m1 + n1;
        const double q0 = Product<INT>::of(d0r, d0r, &bad), q1 = Product<INT>::of(d1r, d1r, &bad);
        const double q2 = Product<INT>::of(d0z, d0z, &bad), q3 = Product<INT>::of(d1z, d1z, &bad);
        kh = Product<INT>::of(Product<INT>::of(Product<INT>::of(hourglass, mu, &bad), dV, &bad),
                        q0 + q1 + q0 + q1 + q2 + q3 + q2 + q3, &bad);
        hg = d.hg[e];
        hg.x += Product<INT>::of(kh, Product<INT>::of(y0, a0, &bad) + Product<INT>::of(y1, a1, &bad)
                               + Product<INT>::of(y2, a2, &bad) + Product<INT>::of(y3, a3, &bad), &bad);
        hg.y += Product<INT>::of(kh, Product<INT>::of(y0, c0, &bad) + Product<INT>::of(y1, c1, &bad)
                               + Product<INT>::of(y2, c2, &bad) + Product<INT>::of(y3, c3, &bad), &bad);
        const double qr = hg.x, qz = hg.y;
        g0r -= Product<INT>::of(y0, qr, &bad); g1r -= Product<INT>::of(y1, qr, &bad);
        g2r -= Product<INT>::of(y2, qr, &bad); g3r -= Product<INT>::of(y3, qr, &bad);
        g0z -= Product<INT>::of(y0, qz, &bad); g1z -= Product<INT>::of(y1, qz, &bad);
        g2z -= Product<INT>::of(y2, qz, &bad); g3z -= Product<INT>::of(y3, qz, &bad);
    }
    if (bad) {
        forces_machine(d, e, strainDt, hourglass, sg);
        return;
    }
    if (hourglass > 0.0) {
        d.hg[e] = hg;
        d.hgK[e] = kh;
    }
    double2 *ef2 = reinterpret_cast<double2 *>(ef);
    ef2[0] = make_double2(g0r, g1r);
    ef2[1] = make_double2(g2r, g3r);
    ef2[2] = make_double2(g0z, g1z);
    ef2[3] = make_double2(g2z, g3z);
}

static __device__ __forceinline__ float diff_hl(float4 a, float4 b, int comp) {
    // (a - b) for component comp (0: r, 1: z) of two hi/lo pairs
    return comp == 0 ? (a.x - b.x) + (a.y - b.y) : (a.z - b.z) + (a.w - b.w);
}

// One point's update in FP32; shared by the reduced and full kernels.
static __device__ __forceinline__ void point_update_mixed(const Dev &d, int e, int p, const MatF &fl,
                                                   float dEpsR, float dEpsZ, float dEpsT,
                                                   float dGamRZ, float spinDt, float strainDt,
                                                   float *sg) {
    float bk[4];
    {
        const float4 s = reinterpret_cast<const float4 *>(d.sigF)[p];
        const float4 b = reinterpret_cast<const float4 *>(d.backF)[p];
        sg[0] = s.x; sg[1] = s.y; sg[2] = s.z; sg[3] = s.w;
        bk[0] = b.x; bk[1] = b.y; bk[2] = b.z; bk[3] = b.w;
    }
    if (d.finite && spinDt != 0.0f) {
        float cs, sn;
        corot_angles(spinDt, cs, sn);
        corot_rotate(sg, cs, sn);
        corot_rotate(bk, cs, sn);
    }
    float epsP = d.epsPF[p], work = d.wPF[p];
    if (d.hasDamage) {
        DamageRefT<float> dr;
        dr.failureStrain = d.dFailF[e];
        dr.strength = d.dStrF + p;
        dr.softening = d.dSoftF + p;
        dr.width = d.dWidthF + p;
        dr.geometry = d.dGeomF + 5 * (size_t)e;
        dr.fractureEnergy = d.dGfF[e];
        dr.youngs = fl.youngs;
        j2_update(sg, bk, epsP, work, dEpsR, dEpsZ, dEpsT, dGamRZ, fl.lambda, fl.mu, fl,
                  strainDt, &dr, d.dStrF[p], d.dSoftF[p]);
    } else {
        j2_update(sg, bk, epsP, work, dEpsR, dEpsZ, dEpsT, dGamRZ, fl.lambda, fl.mu, fl,
                  strainDt, (const DamageRefT<float> *)nullptr, 0.0f, 0.0f);
    }
    reinterpret_cast<float4 *>(d.sigF)[p] = make_float4(sg[0], sg[1], sg[2], sg[3]);
    reinterpret_cast<float4 *>(d.backF)[p] = make_float4(bk[0], bk[1], bk[2], bk[3]);
    d.epsPF[p] = epsP;
    d.wPF[p] = work;
}

// reducedIntegration (ExplicitSolver.java:1373-1504) in FP32 for element e, on the float
// geometry pMid/vdt of its nodes (node n at index n - base). Shared by the single-scene and
// batched kernels.
static __device__ __forceinline__ void element_reduced_f32(const Dev &d, int e, float strainDt,
                                                           float hourglass, const float4 *pMid,
                                                           const float2 *vdt, int base,
                                                           float &minEdge) {
    float4 *ef = reinterpret_cast<float4 *>(d.contribF + 8 * (size_t)e);
    if (d.gone != nullptr && d.gone[e]) {
        ef[0] = make_float4(0.f, 0.f, 0.f, 0.f);
        ef[1] = make_float4(0.f, 0.f, 0.f, 0.f);
    } else {
        const MatF &fl = d.matsF[d.emat[e]];
        const float mu = fl.mu;
        const int4 c = d.conn[e];
        const float4 p0 = pMid[c.x - base], p1 = pMid[c.y - base], p2 = pMid[c.z - base],
                     p3 = pMid[c.w - base];
        const float2 w0 = vdt[c.x - base], w1 = vdt[c.y - base], w2 = vdt[c.z - base],
                     w3 = vdt[c.w - base];
        const float r0 = 0.0f, z0 = 0.0f;
        const float r1 = diff_hl(p1, p0, 0), r2 = diff_hl(p2, p0, 0), r3 = diff_hl(p3, p0, 0);
        const float z1 = diff_hl(p1, p0, 1), z2 = diff_hl(p2, p0, 1), z3 = diff_hl(p3, p0, 1);
        const float a0 = w0.x, a1 = w1.x, a2 = w2.x, a3 = w3.x;
        const float c0 = w0.y, c1 = w1.y, c2 = w2.y, c3 = w3.y;
        if (d.finite) minEdge = shortestEdge(minEdge, r0, r1, r2, r3, z0, z1, z2, z3);

        const float J00 = 0.25f * (-r0 + r1 + r2 - r3);
        const float J01 = 0.25f * (-z0 + z1 + z2 - z3);
        const float J10 = 0.25f * (-r0 - r1 + r2 + r3);
        const float J11 = 0.25f * (-z0 - z1 + z2 + z3);
        const float det = J00 * J11 - J01 * J10;
        const float inv = 1.0f / det;
        const float d0r = 0.25f * (J01 - J11) * inv;
        const float d1r = 0.25f * (J01 + J11) * inv;
        const float d2r = -d0r, d3r = -d1r;
        const float d0z = 0.25f * (J10 - J00) * inv;
        const float d1z = -0.25f * (J10 + J00) * inv;
        const float d2z = -d0z, d3z = -d1z;

        const float dEpsR = d0r * a0 + d1r * a1 + d2r * a2 + d3r * a3;
        const float dEpsZ = d0z * c0 + d1z * c1 + d2z * c2 + d3z * c3;
        const float dRdZ = d0z * a0 + d1z * a1 + d2z * a2 + d3z * a3;
        const float dZdR = d0r * c0 + d1r * c1 + d2r * c2 + d3r * c3;
        const float dGamRZ = dRdZ + dZdR;
        float rg = 0.0f, dEpsT = 0.0f;
        if (d.axi) {
            rg = 0.25f * (p0.x + p1.x + p2.x + p3.x);
            dEpsT = 0.25f * (a0 + a1 + a2 + a3) / rg;
        }
        float sg[4];
        point_update_mixed(d, e, e, fl, dEpsR, dEpsZ, dEpsT, dGamRZ,
                           0.5f * (dZdR - dRdZ), strainDt, sg);
        const float sR = sg[0], sZ = sg[1], sT = sg[2], sRZ = sg[3];
        const float dV = 4.0f * (d.axi ? 2.0f * 3.14159265358979f * rg * det
                                       : (float)d.thickness * det);
        float g0r, g1r, g2r, g3r;
        if (d.axi) {
            const float hh = sT / rg * dV * 0.25f;
            g0r = -((d0r * sR + d0z * sRZ) * dV + hh);
            g1r = -((d1r * sR + d1z * sRZ) * dV + hh);
            g2r = -((d2r * sR + d2z * sRZ) * dV + hh);
            g3r = -((d3r * sR + d3z * sRZ) * dV + hh);
        } else {
            g0r = -(d0r * sR + d0z * sRZ) * dV;
            g1r = -(d1r * sR + d1z * sRZ) * dV;
            g2r = -(d2r * sR + d2z * sRZ) * dV;
            g3r = -(d3r * sR + d3z * sRZ) * dV;
        }
        float g0z = -(d0z * sZ + d0r * sRZ) * dV;
        float g1z = -(d1z * sZ + d1r * sRZ) * dV;
        float g2z = -(d2z * sZ + d2r * sRZ) * dV;
        float g3z = -(d3z * sZ + d3r * sRZ) * dV;
        const float qhg = hourglass;
        if (qhg > 0.0f) {
            const float hr = r0 - r1 + r2 - r3;
            const float hz = z0 - z1 + z2 - z3;
            const float y0 = 1.0f - hr * d0r - hz * d0z;
            const float y1 = -1.0f - hr * d1r - hz * d1z;
            const float y2 = 1.0f - hr * d2r - hz * d2z;
            const float y3 = -1.0f - hr * d3r - hz * d3z;
            const float k = qhg * mu * dV
                            * (d0r * d0r + d1r * d1r + d2r * d2r + d3r * d3r
                               + d0z * d0z + d1z * d1z + d2z * d2z + d3z * d3z);
            float2 hg = d.hgF[e];
            hg.x += k * (y0 * a0 + y1 * a1 + y2 * a2 + y3 * a3);
            hg.y += k * (y0 * c0 + y1 * c1 + y2 * c2 + y3 * c3);
            d.hgF[e] = hg;
            g0r -= y0 * hg.x; g1r -= y1 * hg.x; g2r -= y2 * hg.x; g3r -= y3 * hg.x;
            g0z -= y0 * hg.y; g1z -= y1 * hg.y; g2z -= y2 * hg.y; g3z -= y3 * hg.y;
            d.hgKF[e] = k;
        }
        ef[0] = make_float4(g0r, g1r, g2r, g3r);
        ef[1] = make_float4(g0z, g1z, g2z, g3z);
    }
}

// applyPressure + pressureAt, ExplicitSolver.java:1203-1207, :1511-1556, for pressure edge e at
// time t (the ramp's target and duration given): writes the edge's contribution slots.
static __device__ __forceinline__ void pressure_edge(const Dev &d, int e, double t, double target,
                                                     double rampDuration) {
    double p = target;
    if (rampDuration > 0.0) {
        const double s = jmin(1.0, nf_div(t, rampDuration));
        p = target * s * s * (3.0 - 2.0 * s);
    }
    double *c = d.contribution + 8 * (size_t)(d.E + e);
    const int2 ed = d.pedges[e];
    const double2 xa = d.X0[ed.x], xb = d.X0[ed.y];
    double ra, rb, za, zb;
    if (d.finite) {
        const double2 ua = d.U[ed.x], ub = d.U[ed.y], va = d.V[ed.x], vb = d.V[ed.y];
        ra = xa.x + ua.x + 0.0 * va.x; rb = xb.x + ub.x + 0.0 * vb.x;
        za = xa.y + ua.y + 0.0 * va.y; zb = xb.y + ub.y + 0.0 * vb.y;
    } else {
        ra = xa.x; rb = xb.x; za = xa.y; zb = xb.y;
    }
    const double tr = rb - ra;
    const double tz = zb - za;
    const double len = nf_sqrt(tr * tr + tz * tz);
    if (len == 0.0) {
        c[0] = 0.0; c[1] = 0.0; c[4] = 0.0; c[5] = 0.0;
        return;
    }
    const nf_divisor byLen = nf_divisor_of(len);
    const double nr = nf_div_by(tz, len, byLen);
    const double nz = nf_div_by(-tr, len, byLen);
    double wa, wb;
    if (d.axi) {
        const double circumference = 2.0 * NF_PI * len;
        wa = circumference * (nf_div(ra, 3.0) + nf_div(rb, 6.0));
        wb = circumference * (nf_div(ra, 6.0) + nf_div(rb, 3.0));
    } else {
        wa = d.thickness * len * 0.5;
        wb = wa;
    }
    c[0] = p * nr * wa;
    c[1] = p * nr * wb;
    c[4] = p * nz * wa;
    c[5] = p * nz * wb;
}

// The same edge in the mixed form: FP64 geometry and load, float contribution slots.
static __device__ __forceinline__ void pressure_edge_f32(const Dev &d, int e, double t,
                                                         double target, double rampDuration) {
    double p = target;
    if (rampDuration > 0.0) {
        const double s = jmin(1.0, nf_div(t, rampDuration));
        p = target * s * s * (3.0 - 2.0 * s);
    }
    float *c = d.contribF + 8 * (size_t)(d.E + e);
    const int2 ed = d.pedges[e];
    const double2 xa = d.X0[ed.x], xb = d.X0[ed.y];
    double ra = xa.x, rb = xb.x, za = xa.y, zb = xb.y;
    if (d.finite) {
        const double2 ua = d.U[ed.x], ub = d.U[ed.y];
        ra += ua.x; rb += ub.x; za += ua.y; zb += ub.y;
    }
    const double tr = rb - ra, tz = zb - za;
    const double len = nf_sqrt(tr * tr + tz * tz);
    if (len == 0.0) {
        c[0] = 0.f; c[1] = 0.f; c[4] = 0.f; c[5] = 0.f;
        return;
    }
    const nf_divisor byLen = nf_divisor_of(len);
    const double nr = nf_div_by(tz, len, byLen), nz = nf_div_by(-tr, len, byLen);
    double wa, wb;
    if (d.axi) {
        const double circumference = 2.0 * NF_PI * len;
        wa = circumference * (nf_div(ra, 3.0) + nf_div(rb, 6.0));
        wb = circumference * (nf_div(ra, 6.0) + nf_div(rb, 3.0));
    } else {
        wa = d.thickness * len * 0.5;
        wb = wa;
    }
    c[0] = (float)(p * nr * wa);
    c[1] = (float)(p * nr * wb);
    c[4] = (float)(p * nz * wa);
    c[5] = (float)(p * nz * wb);
}

// ---------------------------------------------------------------- the compensated form
// FP32 nodal arithmetic with each displacement carried as an unevaluated float pair hi + lo
// (Kahan-style compensated accumulation, about 48 significant bits), FP32 velocities and an
// FP32 gather. The error-free transformations are additions only; the increment v dt that
// feeds one is rounded on its own (__fmul_rn), so a contracted multiply-add cannot change
// what the compensation sees.

// TwoSum (Knuth): s + e == a + b exactly.
static __device__ __forceinline__ float2 two_sum_f(float a, float b) {
    const float s = a + b;
    const float bb = s - a;
    return make_float2(s, (a - (s - bb)) + (b - bb));
}

// (hi, lo) += x, renormalised (|lo| <= ulp(hi) / 2).
static __device__ __forceinline__ void ff_add(float &hi, float &lo, float x) {
    const float2 s = two_sum_f(hi, x);
    const float l = s.y + lo;
    hi = s.x + l;
    lo = l - (hi - s.x);
}

// The pair nearest xh + xl + uh + ul + c for a small c (a node's position, mid-step or current).
static __device__ __forceinline__ float2 ff_point(float xh, float xl, float uh, float ul, float c) {
    const float2 s = two_sum_f(xh, uh);
    const float l = s.y + ((xl + ul) + c);
    const float hi = s.x + l;
    return make_float2(hi, l - (hi - s.x));
}

static __device__ __forceinline__ float2 ff_from(double x) {
    const float hi = (float)x;
    return make_float2(hi, (float)(x - (double)hi));
}

// nodalUpdate (:998-1062) with the rigid wall (RigidWall.java:163-259) for node i in the
// compensated form, the same branch structure as nodal_node; also writes the node's float
// geometry for the coming assembly. The audit terms are summed in FP64.
static __device__ __forceinline__ void nodal_node_comp(const Dev &d, int i, float decay,
                                                       float gain, float dtAvg, float dt,
                                                       float plane, float friction,
                                                       const WallRef &w, const MixedGeo &geo,
                                                       uint32_t *status, double &impulse,
                                                       double &loss, double &fric) {
    const uint8_t fl = d.flags[i];
    const bool fixedR = fl & 1, fixedZ = fl & 2;
    bool onWall = fl & 4;
    float4 u = d.uC[i];
    float2 v = d.vC[i];
    const float2 f = d.fC[i];
    const float2 mm = d.mC[i];
    const float m = mm.x, invM = mm.y;
    const float4 x0 = d.x0C[i];
    const bool resting = w.present && onWall && f.y <= 0.0f;
    uint8_t ws = 0;
    if (fixedR) {
        v.x = 0.0f;
    } else if (resting && friction > 0.0f) {
        const float normal = -f.y;
        const float trial = -m * decay * v.x / gain - f.x;
        const float limit = isinf(friction) ? INFINITY : friction * normal;
        if (fabsf(trial) <= limit) {
            loss += 0.5 * (double)m * (double)v.x * (double)v.x;
            atomicAdd(w.stuck, 1);
            ws |= NF_WALL_STUCK;
            v.x = 0.0f;
        } else {
            const float tangential = copysignf(limit, trial);
            const float slid = decay * v.x + gain * (f.x + tangential) / m;
            fric += -(double)tangential * (double)slid * (double)dt;
            ws |= NF_WALL_SLID;
            v.x = slid;
        }
        ff_add(u.x, u.y, __fmul_rn(v.x, dt));
    } else {
        v.x = decay * v.x + gain * f.x * invM;
        ff_add(u.x, u.y, __fmul_rn(v.x, dt));
    }
    if (fixedZ) {
        v.y = 0.0f;
    } else if (resting) {
        impulse += -(double)f.y * (double)dtAvg;
        atomicAdd(w.contact, 1);
        ws |= NF_WALL_HELD;
    } else {
        const float trial = decay * v.y + gain * f.y * invM;
        // z + trial dt < plane, with z = x0 + u as a pair
        const float2 s = two_sum_f(x0.z, u.z);
        const float below = (s.x - plane) + ((s.y + (x0.w + u.w)) + trial * dt);
        if (w.present && below < 0.0f) {
            impulse += -(double)m * (double)trial;
            loss += 0.5 * (double)m * (double)trial * (double)trial;
            atomicAdd(w.contact, 1);
            // u = plane - x0
            const float2 t = two_sum_f(plane, -x0.z);
            const float l = t.y - x0.w;
            u.z = t.x + l;
            u.w = l - (u.z - t.x);
            v.y = 0.0f;
            onWall = true;
            ws |= NF_WALL_ARRIVED;
        } else {
            v.y = trial;
            ff_add(u.z, u.w, __fmul_rn(v.y, dt));
            if (w.present) onWall = false;
        }
    }
    d.uC[i] = u;
    d.vC[i] = v;
    if (w.present) {
        d.flags[i] = (uint8_t)((fl & 3) | (onWall ? 4 : 0));
        d.wallState[i] = ws;
    }
    if (!(isfinite(u.x) && isfinite(u.z) && isfinite(v.x) && isfinite(v.y)))
        atomicOr(status, STATUS_NONFINITE);
    if (geo.pMid) {
        const float mid = -0.5f * dt;
        float2 pr, pz;
        if (d.finite) {
            pr = ff_point(x0.x, x0.y, u.x, u.y, mid * v.x);
            pz = ff_point(x0.z, x0.w, u.z, u.w, mid * v.y);
        } else {
            pr = make_float2(x0.x, x0.y);
            pz = make_float2(x0.z, x0.w);
        }
        geo.pMid[geo.base + i] = make_float4(pr.x, pr.y, pz.x, pz.y);
        geo.vdt[geo.base + i] = make_float2(v.x * dt, v.y * dt);
    }
}

// The pressure edge of the mixed form with the edge's current geometry read from the
// compensated pairs.
static __device__ __forceinline__ void pressure_edge_comp(const Dev &d, int e, double t,
                                                          double target, double rampDuration) {
    double p = target;
    if (rampDuration > 0.0) {
        const double s = jmin(1.0, nf_div(t, rampDuration));
        p = target * s * s * (3.0 - 2.0 * s);
    }
    float *c = d.contribF + 8 * (size_t)(d.E + e);
    const int2 ed = d.pedges[e];
    const float4 xa = d.x0C[ed.x], xb = d.x0C[ed.y];
    double ra = (double)xa.x + (double)xa.y, rb = (double)xb.x + (double)xb.y;
    double za = (double)xa.z + (double)xa.w, zb = (double)xb.z + (double)xb.w;
    if (d.finite) {
        const float4 ua = d.uC[ed.x], ub = d.uC[ed.y];
        ra += (double)ua.x + (double)ua.y; rb += (double)ub.x + (double)ub.y;
        za += (double)ua.z + (double)ua.w; zb += (double)ub.z + (double)ub.w;
    }
    const double tr = rb - ra, tz = zb - za;
    const double len = nf_sqrt(tr * tr + tz * tz);
    if (len == 0.0) {
        c[0] = 0.f; c[1] = 0.f; c[4] = 0.f; c[5] = 0.f;
        return;
    }
    const nf_divisor byLen = nf_divisor_of(len);
    const double nr = nf_div_by(tz, len, byLen), nz = nf_div_by(-tr, len, byLen);
    double wa, wb;
    if (d.axi) {
        const double circumference = 2.0 * NF_PI * len;
        wa = circumference * (nf_div(ra, 3.0) + nf_div(rb, 6.0));
        wb = circumference * (nf_div(ra, 6.0) + nf_div(rb, 3.0));
    } else {
        wa = d.thickness * len * 0.5;
        wb = wa;
    }
    c[0] = (float)(p * nr * wa);
    c[1] = (float)(p * nr * wb);
    c[4] = (float)(p * nz * wa);
    c[5] = (float)(p * nz * wb);
}

// The gather of float contributions into float sums, in CSR order, then m g.
static __device__ __forceinline__ float2 gather_node_comp(const Dev &d, int n, float gR,
                                                          float gZ) {
    float sr = 0.0f, sz = 0.0f;
    const int end = d.nodeSlotStart[n + 1];
    for (int k = d.nodeSlotStart[n]; k < end; k++) {
        const int slot = d.nodeSlot[k];
        sr += d.contribF[slot];
        sz += d.contribF[slot + 4];
    }
    const float m = d.mC[n].x;
    return make_float2(sr + m * gR, sz + m * gZ);
}

// The last addition of a gather, s + m g: s is never -0 (a sum that starts at +0 is not), so
// adding the +-0 that a zero g gives with a finite mass changes nothing.
template <bool INT>
static __device__ __forceinline__ double add_weight(double s, double m, double g) {
    const bool finite = (__double2hiint(m) & 0x7ff00000) != 0x7ff00000;
    if (!is_zero(g) || !finite) s += Product<INT>::of(m, g);
    return s;
}
// 0 + x: x, but +0 for -0.
static __device__ __forceinline__ double first_term(double x) {
    return is_zero(x) ? 0.0 : x;
}

// gather, ExplicitSolver.java:1147-1165: node n's sources in ascending order, then m g.
// The first slot, then three at a time (an interior node has four): their indices, then their
// values, are loaded before any is added, so the loads overlap; the sums still take the slots in
// order. The first sum, with 0, and the weight where there is no gravity are not formed: six FP64
// additions an interior node instead of ten and two products.
template <bool INT>
static __device__ __forceinline__ double2 gather_node(const Dev &d, int n) {
    double sr = 0.0, sz = 0.0;
    const int begin = d.nodeSlotStart[n], end = d.nodeSlotStart[n + 1];
    const double m = d.mass[n];
    if (begin < end) {
        const int slot = d.nodeSlot[begin];
        sr = first_term(d.contribution[slot]);
        sz = first_term(d.contribution[slot + 4]);
    }
    for (int k = begin + 1; k < end; k += 3) {
        const int cnt = end - k < 3 ? end - k : 3;
        int slot[3];
        double vr[3], vz[3];
#pragma unroll
        for (int j = 0; j < 3; j++) slot[j] = j < cnt ? d.nodeSlot[k + j] : 0;
#pragma unroll
        for (int j = 0; j < 3; j++) {
            vr[j] = j < cnt ? d.contribution[slot[j]] : 0.0;
            vz[j] = j < cnt ? d.contribution[slot[j] + 4] : 0.0;
        }
#pragma unroll
        for (int j = 0; j < 3; j++) {
            if (j < cnt) {
                sr += vr[j];
                sz += vz[j];
            }
        }
    }
    return make_double2(add_weight<INT>(sr, m, d.gravR), add_weight<INT>(sz, m, d.gravZ));
}

// The warp's smallest non-negative bit pattern into *best by the integer minimum of its halves
// (all 32 lanes call it). One address takes every warp's minimum, and most do not lower it any
// more, so a warp looks before it adds its atomic to the queue there.
__device__ __forceinline__ void commit_min_bits(unsigned long long bits, unsigned long long *best) {
    const unsigned hi = (unsigned)(bits >> 32);
    const unsigned h = __reduce_min_sync(0xffffffffu, hi);
    const unsigned l = __reduce_min_sync(0xffffffffu, hi == h ? (unsigned)bits : 0xffffffffu);
    const unsigned long long m = ((unsigned long long)h << 32) | l;
    if ((threadIdx.x & 31) == 0 && m < __ldcg(best)) atomicMin(best, m);
}

// The same gather of float contributions into FP64 sums (the mixed form). Each float is widened
// to double by integer arithmetic (exact, the value the conversion gives): only the sums use the
// FP64 pipe. 200k elements: 10.5 us in a profile, waiting for the contributions' loads.
template <bool INT>
static __device__ __forceinline__ double2 gather_node_f32(const Dev &d, int n) {
    double sr = 0.0, sz = 0.0;
    const int begin = d.nodeSlotStart[n], end = d.nodeSlotStart[n + 1];
    const double m = d.mass[n];
    if (begin < end) {
        const int slot = d.nodeSlot[begin];
        sr = first_term(nf_widen(d.contribF[slot]));
        sz = first_term(nf_widen(d.contribF[slot + 4]));
    }
    for (int k = begin + 1; k < end; k += 3) {
        const int cnt = end - k < 3 ? end - k : 3;
        int slot[3];
        float vr[3], vz[3];
#pragma unroll
        for (int j = 0; j < 3; j++) slot[j] = j < cnt ? d.nodeSlot[k + j] : 0;
#pragma unroll
        for (int j = 0; j < 3; j++) {
            vr[j] = j < cnt ? d.contribF[slot[j]] : 0.0f;
            vz[j] = j < cnt ? d.contribF[slot[j] + 4] : 0.0f;
        }
#pragma unroll
        for (int j = 0; j < 3; j++) {
            if (j < cnt) {
                sr += nf_widen(vr[j]);
                sz += nf_widen(vz[j]);
            }
        }
    }
    return make_double2(add_weight<INT>(sr, m, d.gravR), add_weight<INT>(sz, m, d.gravZ));
}

}  // namespace nf
