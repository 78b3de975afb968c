// Reverse-mode adjoint of the FP64 explicit USL step (no counterpart in the
// reference, which has no derivatives): gradients of a loss on the final
// particle positions with respect to the material parameters, through every
// step of a trajectory.
//
// Forward (mpmg_adj_forward_tape): the ordinary FP64 step, with the particle
// state saved every K steps (checkpoints).  Backward (mpmg_adj_backward):
// segment by segment from the last, the forward steps of the segment are run
// again from its checkpoint with each step's inputs recorded on the device
// (particle state at the step start, elements and activity after the keys
// phase, each element's ordered particle list from the step's rows, the nodal
// mass, acceleration and velocity, the step's time and gravity), then the
// segment's steps are reversed one by one:
//
//   adj_g2p    per particle: the material update (isolin, g_local_mu2 or
//              g_nonlocal_mu2), volume, strain rate, velocity and position
//              gathers, and the start-of-step shape functions, reversed;
//              writes the particle's share of the adjoint nodal velocity and
//              acceleration, and the parameter adjoint (block partial sums)
//   adj_node   per node: those shares summed over the particles of its four
//              elements, in colour order and list order (fixed order, no
//              atomics), then the boundary masks and the nodal update
//              (v = p/m, a = f/m, p += dt f) reversed -> adjoint nodal
//              momentum, force and mass
//   adj_p2g    per particle: the P2G of mass, momentum and internal force
//              reversed (a gather from the four nodes); one more block adds
//              the step's block partials to the parameter adjoint
//
// The particle kernels are bound by the FP64 pipe (64 cycles a warp
// instruction), so they work on each nodal field's bilinear coefficients on
// the element (value, gradient and mixed derivative from the four nodes)
// instead of on sums over shape functions, and on mat::root, mat::quot and
// register-operand FMAs.  65 536 particles with g_local_mu2: adj_g2p 76 -> 40 us
// (672 -> 150 FP64 instructions a warp), adj_p2g 28 -> 16 (248 -> 66), the
// element and node sums 32 -> 21, the parameter sum 23 -> none of its own, the
// recorded order 26 -> 2.
//
// The element of each particle is held fixed within a step (the map from
// positions to elements is piecewise constant), and the branches of the
// material law (elastic / plastic / stress-free) are those the forward step
// took.  Everything is FP64 and deterministic.
#include <math.h>
#include <string.h>

#include <vector>

#include "mpmg_fp64_common.cuh"
#include "mpmg_internal.cuh"
#include "mpmg_materials.cuh"

namespace {

using fp64::BcParams;
using fp64::GridGeom;
using fp64::ShapeFns;

constexpr int kAdjThreads = 128;
constexpr int kStateFields = 9;     // x y vx vy v sxx sxy syy Tzz
constexpr int kNodeFields = 5;      // m ax ay vx vy

// Parameter adjoint slots (mpmg_adj_backward's dtheta).
enum { TH_MU_S = 0, TH_MU_2 = 1, TH_I0 = 2, TH_E = 3, TH_COUNT = 4, TH_A = 4, TH_ALL = 5 };

struct MatParams {
    double G, K, lambda, dt, nu;
    double mu_s, mu_2, I0, grains_rho, grains_d, rho_critical;
    double A;               // nonlocal amplitude (g_nonlocal_mu2)
};

// ---------------------------------------------------------------------------
// Material laws reversed.  Inputs: the start-of-step stress T, the strain
// rate and spin (exx, exy, eyy, wxy), mass and updated volume; Tb the
// adjoint of the updated stress.  Outputs: the adjoint of T (overwrites Tb),
// of the strain rate and spin, and the parameter adjoint in terms of G, K
// (folded into E by the caller), mu_s, mu_2 and I0.

struct MatAdj {
    double exx, exy, eyy, wxy;
    double G, K, lambda, mu_s, mu_2, I0, A;
};

// isolin.c:75-116: s' = s + dt (lambda trD I + 2G D + W s - s W).
__device__ void isolin_adj(const MatParams &p, double exx, double exy, double eyy, double wxy, double sxx,
                           double sxy, double syy, double Tb[4], MatAdj &a)
{
    const double dt = p.dt, trD = exx + eyy;
    const double bxx = Tb[0], bxy = Tb[1], byy = Tb[2];
    a.exx += dt * (p.lambda * (bxx + byy) + 2.0 * p.G * bxx);
    a.eyy += dt * (p.lambda * (bxx + byy) + 2.0 * p.G * byy);
    a.exy += dt * 2.0 * p.G * bxy;
    a.wxy += dt * (2.0 * sxy * bxx - (sxx - syy) * bxy - 2.0 * sxy * byy);
    a.lambda += dt * trD * (bxx + byy);
    a.G += dt * 2.0 * (exx * bxx + exy * bxy + eyy * byy);
    Tb[0] = bxx - dt * wxy * bxy;
    Tb[2] = byy + dt * wxy * bxy;
    Tb[1] = bxy + dt * 2.0 * wxy * (bxx - byy);
    Tb[3] = 0.0;
}

// The constants of the particle kernels, staged in shared memory (mat::Unit).
struct AdjConst {
    mat::Elastic el;
    MatParams mp;
    mat::Known krho;                // grains_rho as a divisor
    double ca, caG, caI0;           // G I0 dt / d and its derivatives by G and I0
    double twodt, twoGdt, ldt;      // 2 dt, 2 G dt, lambda dt
    double inv_h, half_inv_h;
};

AdjConst make_adj_const(const MatParams &p, double inv_h)
{
    AdjConst c;
    c.el = mat::make_elastic(p.G, p.K, p.lambda, p.dt);
    c.mp = p;
    c.krho = mat::make_known(p.grains_rho);
    c.caG = p.I0 * p.dt / p.grains_d;
    c.caI0 = p.G * p.dt / p.grains_d;
    c.ca = p.G * c.caG;
    c.twodt = 2.0 * p.dt;
    c.twoGdt = 2.0 * p.G * p.dt;
    c.ldt = p.lambda * p.dt;
    c.inv_h = inv_h;
    c.half_inv_h = 0.5 * inv_h;
    return c;
}

// g_local_mu2.c:165-310 (plane strain, T = [[Txx, Txy, 0], [Txy, Tyy, 0],
// [0, 0, Tzz]]): trial Jaumann stress, deviatoric split, mu(I) return map, with
// d2 = 2 Dxy and w2 = 2 Wxy.  The return's tau' is a root of
// t^2 + B t + H = 0 with 2 tau' + B = -disc, so d tau' / dB = tau' / disc and
// d tau' / dH = 1 / disc.  Adds to a.exx, a.eyy, a.exy, a.wxy as the other laws
// do (exy and wxy the halves of d2 and w2).
__device__ __forceinline__ void g_local_mu2_adj(const AdjConst &C, double m, double v, double exx, double eyy,
                                                double d2, double w2, double Txx, double Txy, double Tyy,
                                                double Tzz, double Tb[4], MatAdj &a)
{
    const mat::Elastic &u = C.el;
    const MatParams &p = C.mp;
    const double dt = u.dt;
    const double trD = u.add(exx, eyy), wxy = u.mul(u.half, w2);
    const double lt = u.mul(u.lambda, trD), dT = u.sub(Tyy, Txx);
    const double Ttr_xx = fma(dt, fma(w2, Txy, fma(u.twoG, exx, lt)), Txx);
    const double Ttr_xy = fma(dt, fma(u.G, d2, u.mul(wxy, dT)), Txy);
    const double Ttr_yy = fma(dt, fma(-w2, Txy, fma(u.twoG, eyy, lt)), Tyy);
    const double Ttr_zz = fma(dt, lt, Tzz);
    const double pm = mat::dvd_const(u.add(u.add(Ttr_xx, Ttr_yy), Ttr_zz), u.k3);
    const double T0xx = u.sub(Ttr_xx, pm), T0yy = u.sub(Ttr_yy, pm), T0zz = u.sub(Ttr_zz, pm), T0xy = Ttr_xy;
    const double dev = fma(T0xx, T0xx, fma(T0yy, T0yy, u.mul(T0zz, T0zz)));
    const double tau = mat::root(fma(u.half, dev, u.mul(T0xy, T0xy)));
    const double pr = -pm;

    // adjoint of the trial stress
    double bxx = 0, bxy = 0, byy = 0, bzz = 0;
    if (mat::quot(m, v) < p.rho_critical || !(pr > 0)) {
        // stress-free (or undefined) branch: T' = 0 does not depend on anything
    } else {
        const double S0 = u.mul(p.mu_s, pr);
        if (tau <= S0) {
            // elastic: T' = T0 - p I = T_trial
            bxx = Tb[0];
            bxy = Tb[1];
            byy = Tb[2];
            bzz = Tb[3];
        } else {
            const double S2 = u.mul(p.mu_2, pr);
            const double sq = mat::root(mat::dvd_const(pr, C.krho));
            const double alpha = u.mul(C.ca, sq);
            const double nB = u.add(u.add(S2, tau), alpha);       // -B
            const double H = fma(S2, tau, u.mul(S0, alpha));
            const double disc = mat::root(fma(u.mfour, H, u.mul(nB, nB)));
            const double taup = nB < 0 ? u.mul(u.half, u.sub(nB, disc)) : mat::quot<1>(H, u.add(nB, disc));
            const double idisc = mat::quot(u.one, disc), itau = mat::quot(u.one, tau);
            const double s = u.mul(taup, itau);
            // T'_ii = T0_ii s + pm (ii = xx, yy, zz), T'_xy = T0xy s
            const double sb = fma(Tb[0], T0xx, fma(Tb[1], T0xy, fma(Tb[2], T0yy, u.mul(Tb[3], T0zz))));
            double pmb = u.add(u.add(Tb[0], Tb[2]), Tb[3]);
            const double taupb = u.mul(sb, itau);
            const double Hb = u.mul(taupb, idisc), Bb = u.mul(Hb, taup);
            // H = S2 tau + S0 alpha; B = -(S2 + tau + alpha)
            const double S2b = fma(Hb, tau, -Bb), S0b = u.mul(Hb, alpha), alphab = fma(Hb, S0, -Bb);
            const double taub = fma(-taupb, s, fma(Hb, S2, -Bb));
            // alpha = ca sqrt(p / rho_g), ca = G I0 dt / d
            const double cab = u.mul(alphab, sq);
            a.G = fma(cab, C.caG, a.G);
            a.I0 = fma(cab, C.caI0, a.I0);
            a.mu_2 = fma(S2b, pr, a.mu_2);
            a.mu_s = fma(S0b, pr, a.mu_s);
            const double prb = fma(S0b, p.mu_s, fma(S2b, p.mu_2, u.mul(u.half, mat::quot(u.mul(alphab, alpha), pr))));
            pmb = u.sub(pmb, prb);
            // tau = sqrt(tt / 2), tt = T0xx^2 + 2 T0xy^2 + T0yy^2 + T0zz^2
            const double kxy = u.mul(taub, itau), k = u.mul(u.half, kxy);
            const double b0xx = fma(T0xx, k, u.mul(Tb[0], s)), b0yy = fma(T0yy, k, u.mul(Tb[2], s));
            const double b0zz = fma(T0zz, k, u.mul(Tb[3], s));
            bxy = fma(T0xy, kxy, u.mul(Tb[1], s));
            // T0_ii = Ttr_ii - pm, pm = (Ttr_xx + Ttr_yy + Ttr_zz) / 3
            const double pm3 = mat::dvd_const(u.sub(u.sub(u.sub(pmb, b0xx), b0yy), b0zz), u.k3);
            bxx = u.add(b0xx, pm3);
            byy = u.add(b0yy, pm3);
            bzz = u.add(b0zz, pm3);
        }
    }
    // trial stress reversed
    const double trb = u.add(u.add(bxx, byy), bzz), lb = u.mul(C.ldt, trb), db = u.sub(bxx, byy), db2 = u.add(db, db);
    a.exx = fma(C.twoGdt, bxx, lb);
    a.eyy = fma(C.twoGdt, byy, lb);
    a.exy = u.mul(C.twoGdt, bxy);
    a.wxy = u.mul(dt, fma(Txy, db2, u.mul(dT, bxy)));
    a.G = fma(C.twodt, fma(exx, bxx, u.mul(eyy, byy)), fma(dt, u.mul(d2, bxy), a.G));
    a.lambda = u.mul(u.mul(dt, trD), trb);
    const double wdt = u.mul(dt, wxy);
    Tb[0] = fma(-wdt, bxy, bxx);
    Tb[1] = fma(wdt, db2, bxy);
    Tb[2] = fma(wdt, bxy, byy);
    Tb[3] = bzz;
}

// Upper-triangle index of (a, b), a <= b, in an element's 10-entry symmetric
// block (the layout of the fluidity assembly).
__device__ __forceinline__ int sym10(int a, int b)
{
    const int row_start[4] = {0, 4, 7, 9};
    return row_start[a] + (b - a);
}

// g_nonlocal_mu2 reversed for one particle: the stress update after the
// fluidity solve (g_nonlocal_mu2.c:160-218), the bulk fluidity
// (calculate_bulk_granular_fluidity, :238-321) and the particle's share of
// the assembled system (:418-507: K_ab += v (xi^-2 N_a N_b + grad N_a .
// grad N_b), f_a += v gf_local xi^-2 N_a over dense particles).  gf is the
// fluidity interpolated at the particle; kb and fb are the adjoints of its
// element's block and right-hand side.  Returns, besides Tb and a as
// g_local_mu2_adj does, the adjoint of the updated volume (vb) and adds the
// adjoints of the shape values and gradients to sb, gxb, gyb.  (The
// adjoint of gf itself is formed by adj_nl_pre_kernel.)
__device__ void g_nonlocal_mu2_adj(const MatParams &p, double m, double v, double exx, double exy, double eyy,
                                   double wxy, double Txx, double Txy, double Tyy, const ShapeFns &f, double gf,
                                   const double kb[10], const double fb[4], double Tb[4], MatAdj &a, double &vb,
                                   double sb[4], double gxb[4], double gyb[4])
{
    const double G = p.G, dt = p.dt, lambda = p.K - 2.0 * G / 3.0;
    const double trD = exx + eyy;
    const double sxx_tr = Txx + dt * (lambda * trD + 2.0 * G * exx + 2.0 * wxy * Txy);
    const double sxy_tr = Txy + dt * (2.0 * G * exy - wxy * (Txx - Tyy));
    const double syy_tr = Tyy + dt * (lambda * trD + 2.0 * G * eyy - 2.0 * wxy * Txy);
    const double pr = -0.5 * (sxx_tr + syy_tr);
    const double t0xx = sxx_tr + pr, t0xy = sxy_tr, t0yy = syy_tr + pr;
    const double tau = sqrt(0.5 * (t0xx * t0xx + 2.0 * t0xy * t0xy + t0yy * t0yy));
    const bool dense = !(m / v < p.rho_critical || pr < 0);
    double t0xxb = 0, t0xyb = 0, t0yyb = 0, prb = 0, taub = 0;
    vb = 0;
    if (dense && pr > 0) {
        // stress update: s = pr / (G dt gf + pr), T' = s t0 - pr I
        const double den = G * dt * gf + pr;
        const double sc = pr / den;
        const double sbar = Tb[0] * t0xx + Tb[1] * t0xy + Tb[2] * t0yy;
        t0xxb += sc * Tb[0];
        t0xyb += sc * Tb[1];
        t0yyb += sc * Tb[2];
        prb -= Tb[0] + Tb[2];
        prb += sbar * (G * dt * gf) / (den * den);
        a.G -= sbar * pr * dt * gf / (den * den);

        // bulk fluidity: tau' from the mu(I) return (tau itself below yield)
        const double S0 = p.mu_s * pr;
        const bool plastic = tau > S0;
        double taup = tau, dB = 0, dH = 0, S2 = 0, alpha = 0, sq = 0, ca = 0;
        if (plastic) {
            S2 = p.mu_2 * pr;
            sq = sqrt(pr / p.grains_rho);
            ca = G * p.I0 * dt / p.grains_d;
            alpha = ca * sq;
            const double B = -(S2 + tau + alpha);
            const double H = S2 * tau + S0 * alpha;
            const double disc = sqrt(B * B - 4.0 * H);
            if (B > 0) {
                taup = 0.5 * (-B - disc);
                dB = 0.5 * (-1.0 - B / disc);
                dH = 1.0 / disc;
            } else {
                const double q = -B + disc;
                taup = 2.0 * H / q;
                const double dqB = -1.0 + B / disc, dqH = -2.0 / disc;
                dB = -2.0 * H / (q * q) * dqB;
                dH = 2.0 / q - 2.0 * H / (q * q) * dqH;
            }
        }
        const double gfl = plastic ? pr / (G * dt) * (tau / taup - 1.0) : 0.0;
        const double D = p.A * p.A * p.grains_d * p.grains_d;
        const double r = taup / pr - p.mu_s;
        const double xisq = fabs(r) / D;

        // the particle's share of the element block and right-hand side
        double xisqb = 0, gflb = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) {
#pragma unroll
            for (int j = i; j < 4; j++) {
                const double k = kb[sym10(i, j)];
                vb += k * (xisq * f.s[i] * f.s[j] + f.gx[i] * f.gx[j] + f.gy[i] * f.gy[j]);
                xisqb += k * v * f.s[i] * f.s[j];
                sb[i] += k * v * xisq * f.s[j];
                sb[j] += k * v * xisq * f.s[i];
                gxb[i] += k * v * f.gx[j];
                gxb[j] += k * v * f.gx[i];
                gyb[i] += k * v * f.gy[j];
                gyb[j] += k * v * f.gy[i];
            }
            vb += fb[i] * gfl * xisq * f.s[i];
            gflb += fb[i] * v * xisq * f.s[i];
            xisqb += fb[i] * v * gfl * f.s[i];
            sb[i] += fb[i] * v * gfl * xisq;
        }
        // xi^-2 = |tau' / pr - mu_s| / (A^2 d^2)
        const double rb = xisqb * (r >= 0 ? 1.0 : -1.0) / D;
        a.A -= xisqb * 2.0 * xisq / p.A;
        double taupb = rb / pr;
        prb -= rb * taup / (pr * pr);
        a.mu_s -= rb;
        if (plastic) {
            // gf_local = pr / (G dt) (tau / tau' - 1)
            const double c = pr / (G * dt);
            prb += gflb * (tau / taup - 1.0) / (G * dt);
            a.G -= gflb * gfl / G;
            taub += gflb * c / taup;
            taupb -= gflb * c * tau / (taup * taup);
            // the return's root reversed (as in g_local_mu2_adj)
            const double Bb = taupb * dB, Hb = taupb * dH;
            const double S2b = Hb * tau - Bb;
            taub += Hb * S2 - Bb;
            const double S0b = Hb * alpha;
            const double alphab = Hb * S0 - Bb;
            prb += alphab * ca * 0.5 / (sq * p.grains_rho);
            const double cab = alphab * sq;
            a.G += cab * p.I0 * dt / p.grains_d;
            a.I0 += cab * G * dt / p.grains_d;
            a.mu_2 += S2b * pr;
            prb += S2b * p.mu_2;
            a.mu_s += S0b * pr;
            prb += S0b * p.mu_s;
        } else {
            taub += taupb;
        }
    }
    // tau = sqrt((t0xx^2 + 2 t0xy^2 + t0yy^2) / 2)
    if (tau > 0) {
        t0xxb += taub * t0xx / (2.0 * tau);
        t0xyb += taub * t0xy / tau;
        t0yyb += taub * t0yy / (2.0 * tau);
    }
    // t0 = T_trial + pr I (xx, yy), pr = -(T_trial,xx + T_trial,yy) / 2
    const double P = prb + t0xxb + t0yyb;
    const double bxx = t0xxb - 0.5 * P, byy = t0yyb - 0.5 * P, bxy = t0xyb;
    // the trial Jaumann stress reversed, lambda = K - 2G/3
    a.exx += dt * (lambda * (bxx + byy) + 2.0 * G * bxx);
    a.eyy += dt * (lambda * (bxx + byy) + 2.0 * G * byy);
    a.exy += dt * 2.0 * G * bxy;
    a.wxy += dt * (2.0 * Txy * bxx - (Txx - Tyy) * bxy - 2.0 * Txy * byy);
    a.lambda += dt * trD * (bxx + byy);
    a.G += dt * 2.0 * (exx * bxx + exy * bxy + eyy * byy);
    Tb[0] = bxx - dt * wxy * bxy;
    Tb[2] = byy + dt * wxy * bxy;
    Tb[1] = bxy + dt * 2.0 * wxy * (bxx - byy);
}

// Mixed second derivative of the shape functions, d2 N_a / dx dy (tent
// products): +1, -1, +1, -1 over h^2 for BL, BR, TR, TL.
__device__ __forceinline__ double shape_xy(int a, double inv_h)
{
    return ((a & 1) ? -1.0 : 1.0) * inv_h * inv_h;
}

struct AdjStep {
    GridGeom g;
    BcParams bc;
    MatParams mp;
    int material;
    int n, ne, nn;
    double dt;
    // recorded forward inputs of the step
    const double *state;        // kStateFields x n, start of step
    const double *mass;         // n (constant)
    const int *elem;            // n
    const int *active;          // n
    const uint32_t *perm;       // n: the elements' particle lists
    const int *start;           // ne: where an element's list begins
    const uint32_t *count;      // ne: and its length
    const double *nodes;        // kNodeFields x nn
    const StepParams *params;   // after the step (t used by the BCs, the step's gravity)
    // adjoints
    const double *adj_in;       // kStateFields x n, of the state after the step
    double *adj_out;            // kStateFields x n, of the state at the step start
    double *contrib;            // n x 16: per particle and corner (Ux, Uy, Ax, Ay) adjoint shares
    double *node_adj;           // nn x 6: pb_x, pb_y, fb_x, fb_y, mb, unused
    double *theta_part;         // per adj_g2p block: the slots' partials
    double *theta_acc;          // their sums over the steps
    AdjConst k;
    // g_nonlocal_mu2
    const double *gf_nodes;     // nn: the step's nodal fluidity (solution of the solve)
    double *gfb;                // n: adjoint of the fluidity interpolated at each particle
    double *rhs;                // 4 x ne: its gather to the nodes, as element corner sums
    const double *lam;          // nn: adjoint of the nodal fluidity (the adjoint solve)
};

constexpr int kThetaSlots = 7;   // mu_s mu_2 I0 (direct) G K lambda, E folded later; A (nonlocal)

// Copies the constants to shared memory (the caller synchronises).
__device__ __forceinline__ void stage_const(AdjConst &C, const AdjConst &param)
{
    static_assert(sizeof(AdjConst) % 8 == 0, "copied as 64-bit words");
    const unsigned long long *src = reinterpret_cast<const unsigned long long *>(&param);
    unsigned long long *dst = reinterpret_cast<unsigned long long *>(&C);
    for (int k = threadIdx.x; k < (int)(sizeof(AdjConst) / 8); k += blockDim.x) dst[k] = src[k];
}

// A nodal field's bilinear coefficients on an element, q0 + c1 x + c2 y + c3 xy
// from the corners BL, BR, TR, TL, and h times its gradient at (x, y).
struct Coef {
    double q0, c1, c2, c3, gx, gy;
};
__device__ __forceinline__ Coef coef_at(const mat::Unit &u, double q0, double q1, double q2, double q3, double x,
                                        double y)
{
    Coef f;
    f.q0 = q0;
    f.c1 = u.sub(q1, q0);
    f.c2 = u.sub(q3, q0);
    f.c3 = u.sub(u.sub(q2, q3), f.c1);
    f.gx = fma(y, f.c3, f.c1);
    f.gy = fma(x, f.c3, f.c2);
    return f;
}
__device__ __forceinline__ double value_at(const Coef &f, double x, double y)
{
    return fma(y, f.gy, fma(x, f.c1, f.q0));
}

// Adds each of eight values over the warp, the sum of value q to lanes with
// lane / 4 == q: three exchanges that halve the values, then two of one value,
// nine additions instead of forty.
__device__ __forceinline__ double warp_sum8(const mat::Unit &u, const double v[8])
{
    const int lane = threadIdx.x & 31;
    double a[4], b[2];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const double keep = lane & 16 ? v[4 + k] : v[k], send = lane & 16 ? v[k] : v[4 + k];
        a[k] = u.add(keep, __shfl_xor_sync(0xffffffffu, send, 16));
    }
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const double keep = lane & 8 ? a[2 + k] : a[k], send = lane & 8 ? a[k] : a[2 + k];
        b[k] = u.add(keep, __shfl_xor_sync(0xffffffffu, send, 8));
    }
    const double keep = lane & 4 ? b[1] : b[0], send = lane & 4 ? b[0] : b[1];
    double c = u.add(keep, __shfl_xor_sync(0xffffffffu, send, 4));
    c = u.add(c, __shfl_xor_sync(0xffffffffu, c, 2));
    return u.add(c, __shfl_xor_sync(0xffffffffu, c, 1));
}

// One particle's corner shares of a field's adjoint where the field enters
// through its value (adjoint R) and h times its gradient (P, Q): with
// t1 = P + R x and t2 = Q + R y the corners TR, BR, TL, BL are t1 y + Q x,
// t1 - TR, t2 - TR and R - t1 - TL.
__device__ __forceinline__ void corner_shares(const mat::Unit &u, double R, double t1, double t2, double tr,
                                              double out[4])
{
    out[2] = tr;
    out[1] = u.sub(t1, tr);
    out[3] = u.sub(t2, tr);
    out[0] = u.sub(u.sub(R, t1), out[3]);
}

template <int MATERIAL>
__global__ void __launch_bounds__(kAdjThreads) adj_g2p_kernel(const __grid_constant__ AdjStep S)
{
    __shared__ AdjConst C;
    __shared__ double red[kAdjThreads / 32][8];
    stage_const(C, S.k);
    __syncthreads();
    const mat::Elastic &u = C.el;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double th[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (i < S.n) {
        const size_t n = (size_t)S.n;
        double in[kStateFields];
#pragma unroll
        for (int f = 0; f < kStateFields; f++) in[f] = S.adj_in[f * n + i];
        const int e = S.elem[i];
        if (!S.active[i] || e < 0) {
            // inactive: the state is carried unchanged (and no list holds it)
#pragma unroll
            for (int f = 0; f < kStateFields; f++) S.adj_out[f * n + i] = in[f];
        } else {
            const GridGeom &g = S.g;
            const double px = S.state[0 * n + i], py = S.state[1 * n + i];
            const double V = S.state[4 * n + i];
            const double Txx = S.state[5 * n + i], Txy = S.state[6 * n + i], Tyy = S.state[7 * n + i],
                         Tzz = S.state[8 * n + i];
            const int cj = e / g.Ex, ci = e - cj * g.Ex;
            const int n0 = cj * g.Nx + ci;
            const int nd[4] = {n0, n0 + 1, n0 + 1 + g.Nx, n0 + g.Nx};
            const double inv_h = C.inv_h, dt = u.dt;
            const double x = mpmg_local_coord_fma(px, mat::small_int(ci), inv_h);
            const double y = mpmg_local_coord_fma(py, mat::small_int(cj), inv_h);
            const size_t nn = (size_t)S.nn;
            Coef q[4];          // ax, ay, ux, uy
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const double *v = S.nodes + (size_t)(1 + k) * nn;
                q[k] = coef_at(u, v[nd[0]], v[nd[1]], v[nd[2]], v[nd[3]], x, y);
            }
            const Coef &qax = q[0], &qay = q[1], &qux = q[2], &quy = q[3];
            const double exx = u.mul(qux.gx, inv_h), eyy = u.mul(quy.gy, inv_h);
            const double gsum = u.add(qux.gy, quy.gx), gdiff = u.sub(qux.gy, quy.gx);
            const double ex = mat::exp_small(u.mul(dt, u.add(exx, eyy)));
            const double Vn = u.mul(V, ex);

            // material
            double Tb[4] = {in[5], in[6], in[7], in[8]};
            MatAdj ma = {};
            double vnb = in[4], xb = in[0], yb = in[1];
            if (MATERIAL == MPMG_ISOLIN) {
                isolin_adj(C.mp, exx, C.half_inv_h * gsum, eyy, C.half_inv_h * gdiff, Txx, Txy, Tyy, Tb, ma);
                Tb[3] = in[8];      // isolin leaves Tzz alone
            } else if (MATERIAL == MPMG_G_NONLOCAL_MU2) {
                // the element's nodal fluidity g and its adjoint lam: the block's
                // adjoint is -(lam g^T) symmetrised, the right-hand side's lam
                const ShapeFns f = fp64::shape(x, y, inv_h);
                double vnl = 0, snl[4] = {0, 0, 0, 0}, gxnl[4] = {0, 0, 0, 0}, gynl[4] = {0, 0, 0, 0};
                double gn[4], ln[4], gf = 0;
#pragma unroll
                for (int a = 0; a < 4; a++) {
                    gn[a] = S.gf_nodes[nd[a]];
                    ln[a] = S.lam[nd[a]];
                    gf += gn[a] * f.s[a];
                }
                double kb[10], fb[4];
#pragma unroll
                for (int a = 0; a < 4; a++) {
                    fb[a] = ln[a];
#pragma unroll
                    for (int b = a; b < 4; b++)
                        kb[sym10(a, b)] = a == b ? -ln[a] * gn[a] : -(ln[a] * gn[b] + ln[b] * gn[a]);
                }
                g_nonlocal_mu2_adj(C.mp, S.mass[i], Vn, exx, C.half_inv_h * gsum, eyy, C.half_inv_h * gdiff, Txx, Txy,
                                   Tyy, f, gf, kb, fb, Tb, ma, vnl, snl, gxnl, gynl);
                // the fluidity gather gf = sum N_a g_a, shape values reversed
                const double gfb = S.gfb[i];
#pragma unroll
                for (int a = 0; a < 4; a++) {
                    const double sa = fma(gfb, gn[a], snl[a]), hxy = shape_xy(a, inv_h);
                    xb += sa * f.gx[a] + gynl[a] * hxy;
                    yb += sa * f.gy[a] + gxnl[a] * hxy;
                }
                vnb += vnl;         // the nonlocal assembly also reads V'
                Tb[3] = in[8];      // plane stress state: Tzz is carried
            } else {
                g_local_mu2_adj(C, S.mass[i], Vn, exx, eyy, u.mul(gsum, inv_h), u.mul(gdiff, inv_h), Txx, Txy, Tyy,
                                Tzz, Tb, ma);
            }
            // volume V' = V exp(dt trD)
            const double Vb = u.mul(vnb, ex);
            const double trb = u.mul(u.mul(vnb, Vn), dt);
            // adjoints of the gathers: h times the gradients of ux (Pu, Qu) and
            // uy (Pv, Qv), and the values of the four fields (R)
            const double Pu = u.mul(u.add(ma.exx, trb), inv_h), Qv = u.mul(u.add(ma.eyy, trb), inv_h);
            const double Qu = u.mul(u.add(ma.exy, ma.wxy), C.half_inv_h), Pv = u.mul(u.sub(ma.exy, ma.wxy), C.half_inv_h);
            double R[4], sh[4][4];      // ux, uy, ax, ay
#pragma unroll
            for (int k = 0; k < 4; k++) {
                R[k] = u.mul(dt, in[k]);
                double t1, t2, tr;
                if (k < 2) {
                    const double P = k == 0 ? Pu : Pv, Q = k == 0 ? Qu : Qv;
                    t1 = fma(R[k], x, P);
                    t2 = fma(R[k], y, Q);
                    tr = fma(t1, y, u.mul(Q, x));
                } else {
                    t1 = u.mul(R[k], x);
                    t2 = u.mul(R[k], y);
                    tr = u.mul(t1, y);
                }
                corner_shares(u, R[k], t1, t2, tr, sh[k]);
            }
            double2 *out = reinterpret_cast<double2 *>(S.contrib + (size_t)i * 16);
#pragma unroll
            for (int a = 0; a < 4; a++) {
                out[2 * a] = make_double2(sh[0][a], sh[1][a]);
                out[2 * a + 1] = make_double2(sh[2][a], sh[3][a]);
            }
            // the start-of-step position: the fields' gradients and mixed derivatives
            double tx = fma(Qv, quy.c3, u.mul(Qu, qux.c3)), ty = fma(Pv, quy.c3, u.mul(Pu, qux.c3));
            tx = fma(R[0], qux.gx, fma(R[1], quy.gx, fma(R[2], qax.gx, fma(R[3], qay.gx, tx))));
            ty = fma(R[0], qux.gy, fma(R[1], quy.gy, fma(R[2], qax.gy, fma(R[3], qay.gy, ty))));
            S.adj_out[0 * n + i] = fma(inv_h, tx, xb);
            S.adj_out[1 * n + i] = fma(inv_h, ty, yb);
            S.adj_out[2 * n + i] = in[2];
            S.adj_out[3 * n + i] = in[3];
            S.adj_out[4 * n + i] = Vb;
            S.adj_out[5 * n + i] = Tb[0];
            S.adj_out[6 * n + i] = Tb[1];
            S.adj_out[7 * n + i] = Tb[2];
            S.adj_out[8 * n + i] = Tb[3];
            th[0] = ma.mu_s;
            th[1] = ma.mu_2;
            th[2] = ma.I0;
            th[3] = ma.G;
            th[4] = ma.K;
            th[5] = ma.lambda;
            th[6] = ma.A;
        }
    }
    // block partials of the parameter adjoint (fixed tree order)
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const double sum = warp_sum8(u, th);
    if ((lane & 3) == 0) red[w][lane >> 2] = sum;
    __syncthreads();
    if (threadIdx.x < kThetaSlots) {
        double v = red[0][threadIdx.x];
        for (int k = 1; k < kAdjThreads / 32; k++) v = u.add(v, red[k][threadIdx.x]);
        S.theta_part[(size_t)blockIdx.x * kThetaSlots + threadIdx.x] = v;
    }
}

// g_nonlocal_mu2, before adj_g2p: per particle, the adjoint of the fluidity
// interpolated at it, through the stress update s = pr / (G dt gf + pr),
// T' = s t0 - pr I (g_nonlocal_mu2.c:160-218).
__global__ void __launch_bounds__(kAdjThreads) adj_nl_pre_kernel(AdjStep S)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S.n) return;
    const int e = S.elem[i];
    double gfb = 0;
    if (S.active[i] && e >= 0) {
        const GridGeom &g = S.g;
        const size_t n = (size_t)S.n, nn = (size_t)S.nn;
        const double x = S.state[0 * n + i], y = S.state[1 * n + i], V = S.state[4 * n + i];
        const double Txx = S.state[5 * n + i], Txy = S.state[6 * n + i], Tyy = S.state[7 * n + i];
        const int ci = e % g.Ex, cj = e / g.Ex;
        const int n0 = cj * g.Nx + ci;
        const int nd[4] = {n0, n0 + 1, n0 + 1 + g.Nx, n0 + g.Nx};
        const double xl = (x - ci * g.h) * g.inv_h, yl = (y - cj * g.h) * g.inv_h;
        const ShapeFns f = fp64::shape(xl, yl, g.inv_h);
        double exx = 0, eyy = 0, dxdy = 0, dydx = 0, gf = 0;
#pragma unroll
        for (int a = 0; a < 4; a++) {
            const double ux = S.nodes[3 * nn + nd[a]], uy = S.nodes[4 * nn + nd[a]];
            exx += f.gx[a] * ux;
            eyy += f.gy[a] * uy;
            dxdy += f.gy[a] * ux;
            dydx += f.gx[a] * uy;
            gf += S.gf_nodes[nd[a]] * f.s[a];
        }
        const MatParams &p = S.mp;
        const double dt = S.dt, G = p.G, lambda = p.K - 2.0 * G / 3.0;
        const double exy = 0.5 * (dxdy + dydx), wxy = 0.5 * (dxdy - dydx);
        const double Vn = V * mat::exp_small(dt * (exx + eyy));
        const double trD = exx + eyy;
        const double sxx_tr = Txx + dt * (lambda * trD + 2.0 * G * exx + 2.0 * wxy * Txy);
        const double sxy_tr = Txy + dt * (2.0 * G * exy - wxy * (Txx - Tyy));
        const double syy_tr = Tyy + dt * (lambda * trD + 2.0 * G * eyy - 2.0 * wxy * Txy);
        const double pr = -0.5 * (sxx_tr + syy_tr);
        const bool dense = !(S.mass[i] / Vn < p.rho_critical || pr < 0);
        if (dense && pr > 0) {
            const double den = G * dt * gf + pr;
            const double sbar = S.adj_in[5 * n + i] * (sxx_tr + pr) + S.adj_in[6 * n + i] * sxy_tr +
                                S.adj_in[7 * n + i] * (syy_tr + pr);
            gfb = -sbar * pr * G * dt / (den * den);
        }
    }
    S.gfb[i] = gfb;
}

// g_nonlocal_mu2: per element, the gather gf_p = sum N_a g_a reversed as
// corner sums N_a gfb_p over the element's particles in the binned order
// (the right-hand-side layout of the assembly, so that the solver sums the
// corners to the nodes).
__global__ void __launch_bounds__(128) adj_nl_rhs_kernel(AdjStep S)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= S.ne) return;
    const GridGeom &g = S.g;
    const size_t n = (size_t)S.n;
    const int ci = e % g.Ex, cj = e / g.Ex;
    double F[4] = {0, 0, 0, 0};
    const int k0 = S.start[e], k1 = k0 + (int)S.count[e];
    for (int k = k0; k < k1; k++) {
        const int i = (int)S.perm[k];
        const double xl = (S.state[0 * n + i] - ci * g.h) * g.inv_h, yl = (S.state[1 * n + i] - cj * g.h) * g.inv_h;
        const ShapeFns f = fp64::shape(xl, yl, g.inv_h);
        const double gfb = S.gfb[i];
#pragma unroll
        for (int a = 0; a < 4; a++) F[a] += f.s[a] * gfb;
    }
#pragma unroll
    for (int a = 0; a < 4; a++) S.rhs[(size_t)a * S.ne + e] = F[a];
}

// Per node: the corner shares of the particles around it summed, then the
// nodal update reversed (grid_kernel of mpmg_step.cu).  Four lanes a node, one
// for each of Ux, Uy, Ax, Ay (a particle's share of a node is one 32-byte
// sector): a warp's chain of additions is the particles around its eight nodes.
__global__ void __launch_bounds__(256) adj_node_kernel(const __grid_constant__ AdjStep S)
{
    __shared__ AdjConst C;
    stage_const(C, S.k);
    __syncthreads();
    const mat::Unit &u = C.el;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = t >> 2, q = t & 3;
    const bool inside = n < S.nn;
    const GridGeom &g = S.g;
    const size_t nn = (size_t)S.nn;
    const double m = inside ? S.nodes[n] : 0.0;
    const int i = n % g.Nx, j = n / g.Nx;
    const bool live = m > MPMG_TOL;
    double ub = 0;
    if (live) {
        int k0[4], cnt[4], corner[4];
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const int ci = ((i & 1) == (c & 1)) ? i : i - 1;
            const int cj = ((j & 1) == (c >> 1)) ? j : j - 1;
            const bool have = ci >= 0 && cj >= 0 && ci < g.Ex && cj < g.Ey;
            const int e = have ? cj * g.Ex + ci : 0;
            cnt[c] = have ? (int)S.count[e] : 0;
            k0[c] = S.start[e];
            corner[c] = (ci == i) ? ((cj == j) ? 0 : 3) : ((cj == j) ? 1 : 2);
        }
        // the first four particles of every element in flight together
        double v[4][4];
        uint32_t at[4][4];
#pragma unroll
        for (int c = 0; c < 4; c++) {
#pragma unroll
            for (int k = 0; k < 4; k++) at[c][k] = k < cnt[c] ? S.perm[k0[c] + k] : 0u;
        }
#pragma unroll
        for (int c = 0; c < 4; c++) {
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (k < cnt[c]) v[c][k] = S.contrib[(size_t)at[c][k] * 16 + corner[c] * 4 + q];
        }
#pragma unroll
        for (int c = 0; c < 4; c++) {
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (k < cnt[c]) ub = u.add(ub, v[c][k]);
            for (int k = 4; k < cnt[c]; k++)
                ub = u.add(ub, S.contrib[(size_t)S.perm[k0[c] + k] * 16 + corner[c] * 4 + q]);
        }
    }
    // U = (P + dt F) / m, A = F / m on unmasked components: lanes 0 and 1 (2 and
    // 3 alike) reverse x and y
    const double other = __shfl_xor_sync(0xffffffffu, ub, 2);
    const double uc = q < 2 ? ub : other, ac = q < 2 ? other : ub;
    double pb = 0, fb = 0, mb = 0;
    if (live) {
        bool bx, by;
        fp64::bc_mask(S.bc, g, i, j, S.params->t, bx, by);
        if (!((q & 1) ? by : bx)) {
            const double a = S.nodes[(size_t)(1 + (q & 1)) * nn + n], v = S.nodes[(size_t)(3 + (q & 1)) * nn + n];
            const double inv_m = mat::quot(u.one, m);
            pb = u.mul(uc, inv_m);
            fb = u.mul(fma(C.el.dt, uc, ac), inv_m);
            mb = -u.mul(fma(uc, v, u.mul(ac, a)), inv_m);
        }
    }
    mb = u.add(mb, __shfl_xor_sync(0xffffffffu, mb, 1));
    if (inside && q < 2) {
        double *out = S.node_adj + (size_t)n * 6;
        out[q] = pb;
        out[2 + q] = fb;
        if (q == 0) out[4] = mb;
    }
}

// Per particle: P2G (p2g_cells_kernel of mpmg_step.cu) reversed.  With the
// nodal adjoints as fields: v' = m pb, V' = -T : grad fb, T' = -V sym grad fb,
// and the position's from grad (m (mb + v pb + g fb_y)) and fb's mixed
// derivative (the gradients of the shape functions).  The last block adds the
// step's block partials to the parameter adjoint, a warp a slot.
__global__ void __launch_bounds__(kAdjThreads) adj_p2g_kernel(const __grid_constant__ AdjStep S)
{
    __shared__ AdjConst C;
    stage_const(C, S.k);
    __syncthreads();
    const mat::Elastic &u = C.el;
    const int blocks = gridDim.x - 1;
    if ((int)blockIdx.x == blocks) {
        const int lane = threadIdx.x & 31;
        for (int slot = threadIdx.x >> 5; slot < kThetaSlots; slot += kAdjThreads / 32) {
            double v = 0;
            for (int b = lane; b < blocks; b += 32) v = u.add(v, S.theta_part[(size_t)b * kThetaSlots + slot]);
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) v = u.add(v, __shfl_down_sync(0xffffffffu, v, off));
            if (lane == 0) S.theta_acc[slot] = u.add(S.theta_acc[slot], v);
        }
        return;
    }
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S.n) return;
    const int e = S.elem[i];
    if (!S.active[i] || e < 0) return;
    const GridGeom &g = S.g;
    const size_t n = (size_t)S.n;
    const double px = S.state[0 * n + i], py = S.state[1 * n + i];
    const double vx = S.state[2 * n + i], vy = S.state[3 * n + i];
    const double V = S.state[4 * n + i];
    const double Txx = S.state[5 * n + i], Txy = S.state[6 * n + i], Tyy = S.state[7 * n + i];
    const double mp = S.mass[i];
    const double grav = S.params->gravity;
    const int cj = e / g.Ex, ci = e - cj * g.Ex;
    const int n0 = cj * g.Nx + ci;
    const int nd[4] = {n0, n0 + 1, n0 + 1 + g.Nx, n0 + g.Nx};
    const double inv_h = C.inv_h;
    const double x = mpmg_local_coord_fma(px, mat::small_int(ci), inv_h);
    const double y = mpmg_local_coord_fma(py, mat::small_int(cj), inv_h);
    double2 p[4], f[4];
    double mb[4];
#pragma unroll
    for (int a = 0; a < 4; a++) {
        const double *v = S.node_adj + (size_t)nd[a] * 6;
        p[a] = *reinterpret_cast<const double2 *>(v);
        f[a] = *reinterpret_cast<const double2 *>(v + 2);
        mb[a] = v[4];
    }
    const Coef pbx = coef_at(u, p[0].x, p[1].x, p[2].x, p[3].x, x, y);
    const Coef pby = coef_at(u, p[0].y, p[1].y, p[2].y, p[3].y, x, y);
    const Coef fbx = coef_at(u, f[0].x, f[1].x, f[2].x, f[3].x, x, y);
    const Coef fby = coef_at(u, f[0].y, f[1].y, f[2].y, f[3].y, x, y);
    const Coef mbc = coef_at(u, mb[0], mb[1], mb[2], mb[3], x, y);
    // m_a += N m; P_a += N m v; F_a += N m b - V T grad N (b = (0, g))
    const double gxy = u.add(fbx.gy, fby.gx);
    const double Vh = -u.mul(V, inv_h);
    const double Vb = u.mul(fma(Txx, fbx.gx, fma(Txy, gxy, u.mul(Tyy, fby.gy))), -inv_h);
    const double wx = fma(vx, pbx.gx, fma(vy, pby.gx, fma(grav, fby.gx, mbc.gx)));
    const double wy = fma(vx, pbx.gy, fma(vy, pby.gy, fma(grav, fby.gy, mbc.gy)));
    const double mh = u.mul(mp, inv_h), Vhh = u.mul(Vh, inv_h);
    const double hx = fma(Txy, fbx.c3, u.mul(Tyy, fby.c3)), hy = fma(Txx, fbx.c3, u.mul(Txy, fby.c3));
    double *out = S.adj_out + i;
    out[0 * n] = fma(mh, wx, fma(Vhh, hx, out[0 * n]));
    out[1 * n] = fma(mh, wy, fma(Vhh, hy, out[1 * n]));
    out[2 * n] = fma(mp, value_at(pbx, x, y), out[2 * n]);
    out[3 * n] = fma(mp, value_at(pby, x, y), out[3 * n]);
    out[4 * n] = u.add(out[4 * n], Vb);
    out[5 * n] = fma(Vh, fbx.gx, out[5 * n]);
    out[6 * n] = fma(Vh, gxy, out[6 * n]);
    out[7 * n] = fma(Vh, fby.gy, out[7 * n]);
}

// The particle state's arrays.
struct StatePtrs {
    const double *x, *y, *vx, *vy, *v, *sxx, *sxy, *syy, *Tzz;
};

__device__ __forceinline__ void copy_state(const StatePtrs &p, int n, int i, double *__restrict__ out)
{
    const size_t N = (size_t)n;
    out[0 * N + i] = p.x[i];
    out[1 * N + i] = p.y[i];
    out[2 * N + i] = p.vx[i];
    out[3 * N + i] = p.vy[i];
    out[4 * N + i] = p.v[i];
    out[5 * N + i] = p.sxx[i];
    out[6 * N + i] = p.sxy[i];
    out[7 * N + i] = p.syy[i];
    out[8 * N + i] = p.Tzz ? p.Tzz[i] : 0.0;
}

// Copies the step-start particle state into a tape slot (one launch).
__global__ void save_state_kernel(int n, StatePtrs p, double *__restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) copy_state(p, n, i, out);
}

__global__ void load_state_kernel(int n, const double *__restrict__ in, double *x, double *y, double *vx,
                                  double *vy, double *v, double *sxx, double *sxy, double *syy, double *Tzz)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const size_t N = (size_t)n;
    x[i] = in[0 * N + i];
    y[i] = in[1 * N + i];
    vx[i] = in[2 * N + i];
    vy[i] = in[3 * N + i];
    v[i] = in[4 * N + i];
    sxx[i] = in[5 * N + i];
    sxy[i] = in[6 * N + i];
    syy[i] = in[7 * N + i];
    if (Tzz) Tzz[i] = in[8 * N + i];
}

// Records the step's outputs the reverse pass needs: elements and activity
// after the keys phase, the ordered list of each element's particles (from the
// rows the P2G ordered; lists follow one another in the order in which warps
// take their space, which nothing depends on), the nodal fields, the step
// record; and the state after the step where the next step is recorded too.
__global__ void __launch_bounds__(256) save_step_kernel(
    int n, int ne, int nn, const int *in_element, const int *active, RowView rv, const double *node_m,
    const double *node_ax, const double *node_ay, const double *node_vx, const double *node_vy, const StepParams *sp,
    StatePtrs next, int *__restrict__ elem_out, int *__restrict__ active_out, uint32_t *__restrict__ perm_out,
    int *__restrict__ start_out, uint32_t *__restrict__ count_out, uint32_t *__restrict__ cursor,
    double *__restrict__ nodes_out, StepParams *__restrict__ sp_out, double *__restrict__ next_out)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k == 0) *sp_out = *sp;
    if (k < n) {
        elem_out[k] = active[k] ? in_element[k] : -1;
        active_out[k] = active[k];
        if (next_out != nullptr) copy_state(next, n, k, next_out);
    }
    const int lane = threadIdx.x & 31;
    const int cnt = k < ne ? (int)rv.count[k] : 0;
    int incl = cnt;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int w = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += w;
    }
    uint32_t base = 0;
    if (lane == 31 && incl > 0) base = atomicAdd(cursor, (uint32_t)incl);
    base = __shfl_sync(0xffffffffu, base, 31) + (uint32_t)(incl - cnt);
    if (k < ne) {
        start_out[k] = (int)base;
        count_out[k] = (uint32_t)cnt;
        if (cnt > 0) {
            const uint32_t *list = rv.list(k, cnt);
            for (int q = 0; q < cnt; q++) perm_out[base + q] = list[q];
        }
    }
    if (k < nn) {
        const size_t N = (size_t)nn;
        nodes_out[0 * N + k] = node_m[k];
        nodes_out[1 * N + k] = node_ax[k];
        nodes_out[2 * N + k] = node_ay[k];
        nodes_out[3 * N + k] = node_vx[k];
        nodes_out[4 * N + k] = node_vy[k];
    }
}

inline int blocks_for(size_t n, int threads)
{
    size_t b = (n + (size_t)threads - 1) / (size_t)threads;
    return (int)(b > 0 ? b : 1);
}

template <typename T>
int dalloc(T **p, size_t count)
{
    cudaError_t e = cudaMalloc((void **)p, (count ? count : 1) * sizeof(T));
    if (e != cudaSuccess) {
        *p = nullptr;
        return mpmg_cuda_status(e, "cudaMalloc (adjoint tape)");
    }
    return MPMG_OK;
}

}  // namespace

// Tape of a forward run (checkpoints) and the scratch of the reverse pass.
struct AdjTape {
    int K = 0;                      // checkpoint interval
    int nsteps = 0;                 // steps of the taped run
    int nck = 0;                    // checkpoints (steps 0, K, 2K, ... < nsteps)
    double *ck_state = nullptr;     // nck x kStateFields x n
    int *ck_active = nullptr;       // nck x n
    int *ck_elem = nullptr;         // nck x n (in_element)
    StepParams *ck_params = nullptr;   // nck (device)
    double *final_state = nullptr;  // kStateFields x n, the state after the run
    int *final_active = nullptr, *final_elem = nullptr;
    StepParams *final_params = nullptr;
    // one segment of recorded steps
    double *seg_state = nullptr;    // K x kStateFields x n
    int *seg_elem = nullptr, *seg_active = nullptr;   // K x n
    uint32_t *seg_perm = nullptr;   // K x n
    int *seg_start = nullptr;       // K x ne
    uint32_t *seg_count = nullptr;  // K x ne
    uint32_t *seg_cursor = nullptr; // K
    double *seg_nodes = nullptr;    // K x kNodeFields x nn
    StepParams *seg_params = nullptr;   // K
    // g_nonlocal_mu2: each recorded step's nodal fluidity and element blocks
    double *seg_gf = nullptr;       // K x nn
    double *seg_ek = nullptr;       // K x 10 x ne
    // reverse pass
    double *adj[2] = {nullptr, nullptr};   // kStateFields x n
    double *contrib = nullptr, *node_adj = nullptr;
    double *theta_part = nullptr, *theta_acc = nullptr;
    double *gfb = nullptr, *rhs = nullptr, *lam = nullptr;   // g_nonlocal_mu2
    double grad[TH_ALL] = {0, 0, 0, 0, 0};   // the last backward pass's parameter gradient
    int cur = 0;                    // adj[cur] holds the latest adjoint state
};

void mpmg_adj_free(mpmg_ctx *ctx)
{
    AdjTape *t = ctx->adj;
    if (t == nullptr) return;
    void *ptrs[] = {t->ck_state, t->ck_active, t->ck_elem, t->ck_params, t->final_state, t->final_active,
                    t->final_elem, t->final_params, t->seg_state, t->seg_elem, t->seg_active, t->seg_perm,
                    t->seg_start, t->seg_count, t->seg_cursor, t->seg_nodes, t->seg_params, t->adj[0], t->adj[1],
                    t->contrib, t->node_adj, t->theta_part, t->theta_acc, t->seg_gf, t->seg_ek, t->gfb, t->rhs, t->lam};
    for (void *p : ptrs) cudaFree(p);
    delete t;
    ctx->adj = nullptr;
}

namespace {

StatePtrs state_ptrs(const mpmg_ctx *ctx)
{
    return StatePtrs{ctx->x, ctx->y, ctx->vx, ctx->vy, ctx->v, ctx->sxx, ctx->sxy, ctx->syy, ctx->Tzz};
}

int save_state(mpmg_ctx *ctx, double *out)
{
    const int n = (int)ctx->np;
    if (n == 0) return MPMG_OK;
    save_state_kernel<<<blocks_for(n, 256), 256, 0, ctx->stream>>>(n, state_ptrs(ctx), out);
    ctx->launches += 1;
    MPMG_CHECK(cudaGetLastError());
    return MPMG_OK;
}

int load_state(mpmg_ctx *ctx, const double *in, const int *active, const int *elem, const StepParams *params)
{
    const int n = (int)ctx->np;
    cudaStream_t s = ctx->stream;
    if (n > 0) {
        load_state_kernel<<<blocks_for(n, 256), 256, 0, s>>>(n, in, ctx->x, ctx->y, ctx->vx, ctx->vy, ctx->v,
                                                            ctx->sxx, ctx->sxy, ctx->syy, ctx->Tzz);
        ctx->launches += 1;
        MPMG_CHECK(cudaMemcpyAsync(ctx->active, active, (size_t)n * sizeof(int), cudaMemcpyDeviceToDevice, s));
        MPMG_CHECK(cudaMemcpyAsync(ctx->in_element, elem, (size_t)n * sizeof(int), cudaMemcpyDeviceToDevice, s));
    }
    MPMG_CHECK(cudaMemcpyAsync(ctx->d_params, params, sizeof(StepParams), cudaMemcpyDeviceToDevice, s));
    MPMG_CHECK(cudaGetLastError());
    ctx->row.ready = false;   // the positions and the element map changed
    return MPMG_OK;
}

int snapshot(mpmg_ctx *ctx, double *state, int *active, int *elem, StepParams *params)
{
    int rc = save_state(ctx, state);
    if (rc != MPMG_OK) return rc;
    cudaStream_t s = ctx->stream;
    const size_t n = ctx->np;
    if (n > 0) {
        MPMG_CHECK(cudaMemcpyAsync(active, ctx->active, n * sizeof(int), cudaMemcpyDeviceToDevice, s));
        MPMG_CHECK(cudaMemcpyAsync(elem, ctx->in_element, n * sizeof(int), cudaMemcpyDeviceToDevice, s));
    }
    MPMG_CHECK(cudaMemcpyAsync(params, ctx->d_params, sizeof(StepParams), cudaMemcpyDeviceToDevice, s));
    return MPMG_OK;
}

MatParams make_params(const mpmg_ctx *ctx)
{
    MatParams p;
    const mpmg_config &c = ctx->cfg;
    p.G = ctx->G;
    p.K = ctx->K;
    p.lambda = ctx->lambda;
    p.dt = c.dt;
    p.nu = c.mp[MPMG_MP_NU];
    p.mu_s = c.mp[MPMG_MP_MU_S];
    p.mu_2 = c.mp[MPMG_MP_MU_2];
    p.I0 = c.mp[MPMG_MP_I0];
    p.grains_rho = c.mp[MPMG_MP_GRAINS_RHO];
    p.grains_d = c.mp[MPMG_MP_GRAINS_D];
    p.rho_critical = c.mp[MPMG_MP_RHO_CRITICAL];
    p.A = c.mp[MPMG_MP_A];
    return p;
}

int check_adjoint_ctx(const mpmg_ctx *ctx)
{
    if (ctx->mixed || ctx->batch) {
        mpmg_set_error("the adjoint runs on the FP64 form of a single simulation");
        return MPMG_ERR_UNSUPPORTED;
    }
    if (ctx->cfg.material != MPMG_ISOLIN && ctx->cfg.material != MPMG_G_LOCAL_MU2 &&
        ctx->cfg.material != MPMG_G_NONLOCAL_MU2) {
        mpmg_set_error("the adjoint supports isolin, g_local_mu2 and g_nonlocal_mu2");
        return MPMG_ERR_UNSUPPORTED;
    }
    return MPMG_OK;
}

int alloc_tape(mpmg_ctx *ctx, AdjTape *t)
{
    const size_t n = ctx->np, ne = ctx->ne, nn = ctx->nn;
    const int K = t->K;
    int rc;
    const size_t nck = (size_t)t->nck;
    if ((rc = dalloc(&t->ck_state, nck * kStateFields * n)) != MPMG_OK ||
        (rc = dalloc(&t->ck_active, nck * n)) != MPMG_OK || (rc = dalloc(&t->ck_elem, nck * n)) != MPMG_OK ||
        (rc = dalloc(&t->ck_params, nck)) != MPMG_OK || (rc = dalloc(&t->final_state, kStateFields * n)) != MPMG_OK ||
        (rc = dalloc(&t->final_active, n)) != MPMG_OK || (rc = dalloc(&t->final_elem, n)) != MPMG_OK ||
        (rc = dalloc(&t->final_params, 1)) != MPMG_OK ||
        (rc = dalloc(&t->seg_state, (size_t)K * kStateFields * n)) != MPMG_OK ||
        (rc = dalloc(&t->seg_elem, (size_t)K * n)) != MPMG_OK ||
        (rc = dalloc(&t->seg_active, (size_t)K * n)) != MPMG_OK ||
        (rc = dalloc(&t->seg_perm, (size_t)K * n)) != MPMG_OK ||
        (rc = dalloc(&t->seg_start, (size_t)K * ne)) != MPMG_OK ||
        (rc = dalloc(&t->seg_count, (size_t)K * ne)) != MPMG_OK ||
        (rc = dalloc(&t->seg_cursor, (size_t)K)) != MPMG_OK ||
        (rc = dalloc(&t->seg_nodes, (size_t)K * kNodeFields * nn)) != MPMG_OK ||
        (rc = dalloc(&t->seg_params, (size_t)K)) != MPMG_OK ||
        (rc = dalloc(&t->adj[0], kStateFields * n)) != MPMG_OK ||
        (rc = dalloc(&t->adj[1], kStateFields * n)) != MPMG_OK || (rc = dalloc(&t->contrib, 16 * n)) != MPMG_OK ||
        (rc = dalloc(&t->node_adj, 6 * nn)) != MPMG_OK ||
        (rc = dalloc(&t->theta_part, (size_t)blocks_for(n, kAdjThreads) * kThetaSlots)) != MPMG_OK ||
        (rc = dalloc(&t->theta_acc, kThetaSlots)) != MPMG_OK) {
        return rc;
    }
    if (ctx->cfg.material == MPMG_G_NONLOCAL_MU2 &&
        ((rc = dalloc(&t->seg_gf, (size_t)K * nn)) != MPMG_OK ||
         (rc = dalloc(&t->seg_ek, (size_t)K * 10 * ne)) != MPMG_OK || (rc = dalloc(&t->gfb, n)) != MPMG_OK ||
         (rc = dalloc(&t->rhs, 4 * ne)) != MPMG_OK || (rc = dalloc(&t->lam, nn)) != MPMG_OK)) {
        return rc;
    }
    return MPMG_OK;
}

}  // namespace

extern "C" {

int mpmg_adj_forward_tape(mpmg_ctx *ctx, int nsteps, int checkpoint_every)
{
    if (ctx == nullptr || nsteps < 1 || checkpoint_every < 1) return MPMG_ERR_INVALID;
    int rc = check_adjoint_ctx(ctx);
    if (rc != MPMG_OK) return rc;
    MPMG_CHECK(cudaSetDevice(ctx->dev));
    const size_t n = ctx->np;
    const int K = checkpoint_every < nsteps ? checkpoint_every : nsteps, checkpoints = (nsteps + K - 1) / K;
    // the last run's tape where its buffers have this one's sizes (27
    // allocations and as many frees took as long as 20 steps of 65k particles)
    AdjTape *t = ctx->adj;
    if (t == nullptr || t->K != K || t->nck != checkpoints) {
        mpmg_adj_free(ctx);
        t = new (std::nothrow) AdjTape();
        if (t == nullptr) return MPMG_ERR_NOMEM;
        ctx->adj = t;
        t->K = K;
        t->nck = checkpoints;
        if ((rc = alloc_tape(ctx, t)) != MPMG_OK) {
            mpmg_adj_free(ctx);
            return rc;
        }
    }
    t->nsteps = nsteps;
    t->cur = 0;
    for (double &v : t->grad) v = 0;
    // The forward run: checkpoint, then K ordinary steps (CUDA graphs).
    for (int c = 0; c < t->nck; c++) {
        rc = snapshot(ctx, t->ck_state + (size_t)c * kStateFields * n, t->ck_active + (size_t)c * n,
                      t->ck_elem + (size_t)c * n, t->ck_params + c);
        if (rc != MPMG_OK) return rc;
        const int steps = (c + 1) * K <= nsteps ? K : nsteps - c * K;
        rc = mpmg_step(ctx, steps);
        if (rc != MPMG_OK) return rc;
    }
    rc = snapshot(ctx, t->final_state, t->final_active, t->final_elem, t->final_params);
    if (rc != MPMG_OK) return rc;
    return mpmg_synchronize(ctx);
}

int mpmg_adj_backward(mpmg_ctx *ctx, const double *dl_dx, const double *dl_dy, double *dl_dtheta)
{
    if (ctx == nullptr || dl_dx == nullptr || dl_dy == nullptr || dl_dtheta == nullptr) return MPMG_ERR_INVALID;
    AdjTape *t = ctx->adj;
    if (t == nullptr) {
        mpmg_set_error("no taped forward run (mpmg_adj_forward_tape)");
        return MPMG_ERR_INVALID;
    }
    MPMG_CHECK(cudaSetDevice(ctx->dev));
    cudaStream_t s = ctx->stream;
    const size_t n = ctx->np, ne = ctx->ne, nn = ctx->nn;
    // adjoint of the final state: the loss gradient with respect to x and y
    t->cur = 0;
    MPMG_CHECK(cudaMemsetAsync(t->adj[0], 0, kStateFields * n * sizeof(double), s));
    if (n > 0) {
        MPMG_CHECK(cudaMemcpyAsync(t->adj[0], dl_dx, n * sizeof(double), cudaMemcpyHostToDevice, s));
        MPMG_CHECK(cudaMemcpyAsync(t->adj[0] + n, dl_dy, n * sizeof(double), cudaMemcpyHostToDevice, s));
    }
    MPMG_CHECK(cudaMemsetAsync(t->theta_acc, 0, kThetaSlots * sizeof(double), s));

    AdjStep S = {};
    S.g = fp64::make_geom(ctx);
    S.bc = fp64::make_bc(ctx);
    S.mp = make_params(ctx);
    S.material = ctx->cfg.material;
    S.n = (int)n;
    S.ne = (int)ne;
    S.nn = (int)nn;
    S.dt = ctx->cfg.dt;
    S.mass = ctx->m;
    S.contrib = t->contrib;
    S.node_adj = t->node_adj;
    S.theta_part = t->theta_part;
    S.theta_acc = t->theta_acc;
    S.k = make_adj_const(S.mp, ctx->inv_h);
    S.gfb = t->gfb;
    S.rhs = t->rhs;
    S.lam = t->lam;
    const bool nonlocal = ctx->cfg.material == MPMG_G_NONLOCAL_MU2;
    const int pblocks = blocks_for(n, kAdjThreads);
    int rc;
    for (int c = t->nck - 1; c >= 0; c--) {
        const int len = (c + 1) * t->K <= t->nsteps ? t->K : t->nsteps - c * t->K;
        // run the segment again from its checkpoint, recording each step
        rc = load_state(ctx, t->ck_state + (size_t)c * kStateFields * n, t->ck_active + (size_t)c * n,
                        t->ck_elem + (size_t)c * n, t->ck_params + c);
        if (rc != MPMG_OK) return rc;
        MPMG_CHECK(cudaMemsetAsync(t->seg_cursor, 0, (size_t)len * sizeof(uint32_t), s));
        if ((rc = save_state(ctx, t->seg_state)) != MPMG_OK) return rc;
        for (int k = 0; k < len; k++) {
            if ((rc = mpmg_fp64_ready(ctx)) != MPMG_OK) return rc;
            ctx->row.record = true;
            rc = mpmg_launch_step(ctx);
            ctx->row.record = false;
            if (rc != MPMG_OK) return rc;
            const size_t m = n > ne ? (n > nn ? n : nn) : (ne > nn ? ne : nn);
            const RowBins &r = ctx->row;
            const int b = 1 - r.cur;        // the step's rows
            save_step_kernel<<<blocks_for(m, 256), 256, 0, s>>>(
                (int)n, (int)ne, (int)nn, ctx->in_element, ctx->active, RowView{r.count[b], r.rows[b], r.over_list, r.cap},
                ctx->node_m, ctx->node_ax, ctx->node_ay, ctx->node_vx, ctx->node_vy, ctx->d_params, state_ptrs(ctx),
                t->seg_elem + (size_t)k * n, t->seg_active + (size_t)k * n, t->seg_perm + (size_t)k * n,
                t->seg_start + (size_t)k * ne, t->seg_count + (size_t)k * ne, t->seg_cursor + k,
                t->seg_nodes + (size_t)k * kNodeFields * nn, t->seg_params + k,
                k + 1 < len ? t->seg_state + (size_t)(k + 1) * kStateFields * n : nullptr);
            ctx->launches += 1;
            if (nonlocal) {
                MPMG_CHECK(cudaMemcpyAsync(t->seg_gf + (size_t)k * nn, ctx->node_gf, nn * sizeof(double),
                                           cudaMemcpyDeviceToDevice, s));
                MPMG_CHECK(cudaMemcpyAsync(t->seg_ek + (size_t)k * 10 * ne, ctx->elem_k, 10 * ne * sizeof(double),
                                           cudaMemcpyDeviceToDevice, s));
            }
        }
        // reverse the segment's steps
        for (int k = len - 1; k >= 0; k--) {
            S.state = t->seg_state + (size_t)k * kStateFields * n;
            S.elem = t->seg_elem + (size_t)k * n;
            S.active = t->seg_active + (size_t)k * n;
            S.perm = t->seg_perm + (size_t)k * n;
            S.start = t->seg_start + (size_t)k * ne;
            S.count = t->seg_count + (size_t)k * ne;
            S.nodes = t->seg_nodes + (size_t)k * kNodeFields * nn;
            S.params = t->seg_params + k;
            S.adj_in = t->adj[t->cur];
            S.adj_out = t->adj[1 - t->cur];
            if (n > 0 && nonlocal) {
                // the fluidity's adjoint: gathered to the nodes, then the same
                // symmetric system solved for it (zero start, same tolerance)
                S.gf_nodes = t->seg_gf + (size_t)k * nn;
                adj_nl_pre_kernel<<<pblocks, kAdjThreads, 0, s>>>(S);
                adj_nl_rhs_kernel<<<blocks_for(ne, 128), 128, 0, s>>>(S);
                ctx->launches += 2;
                MPMG_CHECK(cudaGetLastError());
                rc = mpmg_solve_fluidity_system(ctx, t->seg_ek + (size_t)k * 10 * ne, t->rhs, S.nodes, S.count, nullptr,
                                                t->lam, true);
                if (rc != MPMG_OK) return rc;
            }
            if (n > 0) {
                switch (S.material) {
                case MPMG_ISOLIN: adj_g2p_kernel<MPMG_ISOLIN><<<pblocks, kAdjThreads, 0, s>>>(S); break;
                case MPMG_G_NONLOCAL_MU2:
                    adj_g2p_kernel<MPMG_G_NONLOCAL_MU2><<<pblocks, kAdjThreads, 0, s>>>(S);
                    break;
                default: adj_g2p_kernel<MPMG_G_LOCAL_MU2><<<pblocks, kAdjThreads, 0, s>>>(S); break;
                }
                adj_node_kernel<<<blocks_for(4 * nn, 256), 256, 0, s>>>(S);
                adj_p2g_kernel<<<pblocks + 1, kAdjThreads, 0, s>>>(S);
                ctx->launches += 3;
            }
            MPMG_CHECK(cudaGetLastError());
            t->cur = 1 - t->cur;
        }
    }
    // the run's final state again, so that stepping can go on
    if ((rc = load_state(ctx, t->final_state, t->final_active, t->final_elem, t->final_params)) != MPMG_OK)
        return rc;
    double th[kThetaSlots];
    MPMG_CHECK(cudaMemcpyAsync(th, t->theta_acc, sizeof(th), cudaMemcpyDeviceToHost, s));
    MPMG_CHECK(cudaStreamSynchronize(s));
    // fold the elastic constants into E: G = E / (2 (1 + nu)), K = E / (3 (1 - 2 nu)),
    // lambda = K - 2 G / 3
    const double nu = ctx->cfg.mp[MPMG_MP_NU];
    const double dG = 1.0 / (2.0 * (1.0 + nu)), dK = 1.0 / (3.0 * (1.0 - 2.0 * nu));
    t->grad[TH_MU_S] = th[0];
    t->grad[TH_MU_2] = th[1];
    t->grad[TH_I0] = th[2];
    t->grad[TH_E] = th[3] * dG + th[4] * dK + th[5] * (dK - 2.0 / 3.0 * dG);
    t->grad[TH_A] = th[6];
    for (int k = 0; k < TH_COUNT; k++) dl_dtheta[k] = t->grad[k];
    return mpmg_synchronize(ctx);
}

// One parameter's gradient from the last mpmg_adj_backward: 0 mu_s, 1 mu_2,
// 2 I0, 3 E, 4 the nonlocal amplitude A (zero for the local materials).
int mpmg_adj_gradient(mpmg_ctx *ctx, int index, double *out)
{
    if (ctx == nullptr || out == nullptr || index < 0 || index >= TH_ALL) return MPMG_ERR_INVALID;
    if (ctx->adj == nullptr) return MPMG_ERR_INVALID;
    *out = ctx->adj->grad[index];
    return MPMG_OK;
}

// Adjoint of one field of the taped run's initial state (after
// mpmg_adj_backward): x y vx vy v sxx sxy syy Tzz, in particle order.
int mpmg_adj_state(mpmg_ctx *ctx, const char *name, double *host_out)
{
    if (ctx == nullptr || name == nullptr || host_out == nullptr) return MPMG_ERR_INVALID;
    if (ctx->adj == nullptr) return MPMG_ERR_INVALID;
    static const char *names[kStateFields] = {"x", "y", "vx", "vy", "v", "sxx", "sxy", "syy", "Tzz"};
    for (int f = 0; f < kStateFields; f++) {
        if (strcmp(name, names[f]) == 0) {
            MPMG_CHECK(cudaSetDevice(ctx->dev));
            return mpmg_copy_out(ctx, host_out, ctx->adj->adj[ctx->adj->cur] + (size_t)f * ctx->np,
                                 ctx->np * sizeof(double));
        }
    }
    return MPMG_ERR_UNKNOWN_FIELD;
}

}  // extern "C"
