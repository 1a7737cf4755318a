// Two-component dwarf initial conditions on the GPU, one warp per body.
//
// Restates the sampler of nbGenerateMixedDwarfCore (nbody/src/nbody_mixeddwarf.c:765-1026)
// for the reference's dwarf profiles (Dwarf.plummer, nfw, general_hernquist and cored,
// nbody/src/nbody_dwarf_potential.c:36-175; Einasto has no case in the reference's
// get_density/get_potential): radii by rejection from r^2 rho(r) of the body's own component
// (r_mag, :538-574), speeds by rejection from the Eddington distribution function of that
// component in the combined potential (vel_mag, :576-618, dist_fun :471-535), the DF evaluated
// as the reference does -- five-point stencil derivatives (:63-95), the d^2rho/dpsi^2 integrand
// (fun, :368-445), a bisection root finder for the integration limit (:247-366) and its
// composite three-point Gauss quadrature (:97-209), the DF maximum by golden-section search
// (:211-245) -- then isotropic directions by rejection in the unit cube (get_components,
// :620-647), and each component recentred on its own centre of mass and velocity and shifted
// onto the orbit (cm_correction_by_comp, :649-694).  The per-component constants -- r200, the
// NFW/cored normalisations (set_vars, :696-726), the NFW/cored mass reset to the mass inside
// the sampling bound (get_extra_nfw_mass, :728-762), the bounds and the r^2 rho maxima
// (:797-903) -- are computed once on the host in the reference's order.
//
// The random numbers are not the reference's dSFMT stream: every body draws from its own
// counter-based stream (splitmix64 of the seed and the body index), so the samples agree with
// the reference's in distribution, not body for body.  The per-body work (tens of DF
// evaluations of ~330 integrand points each) is what makes the reference's sampler take ~12 min
// per 10^6 bodies on one core; here the bodies are independent warps.
#include "nb_common.cuh"
#include "nb_crmath.cuh"
#include "nb_rdiv.cuh"
#include <vector>

namespace {

// pcrit and vol_pcrit = 200 pcrit 4 pi / 3 (milkyway/include/milkyway_math_supplemental.h:224-225)
constexpr double kPcrit = 0.000679087369829744220469326744094105320596648627735869652;
constexpr double kVolPcrit = 0.568910904587397184785763397846734505212216314432372653620;

// One component of the dwarf with the constants its density and potential need.
struct NbIcComp {
    int type;                    // NBCUDA_DWARF_*
    double M, a;                 // mass (after the NFW/cored reset) and scale length
    double p0, ps, r1, rc;       // NFW/cored normalisations, cored radii
    double C2, C3;               // cored potential constants (cored_pot)
    double bound, rhoMax;        // r_mag's sampling bound and maximum of r^2 rho

    // get_density (nbody_dwarf_potential.c:207-236); the Plummer case inline, the others out of
    // line, so that the DF integrand's many evaluations keep the Plummer sampler's registers
    NB_HD double den(double r) const
    {
        if (type == NBCUDA_DWARF_PLUMMER) {
            const double x = 1.0 + (r / a) * (r / a);
            return (3.0 / (4.0 * M_PI)) * (M / (a * a * a)) * (1.0 / sqrt(x * x * x * x * x));
        }
        return den_profile(r);
    }
    // get_potential (nbody_dwarf_potential.c:176-205), the positive psi
    NB_HD double pot(double r) const
    {
        if (type == NBCUDA_DWARF_PLUMMER) return M / sqrt(r * r + a * a);
        return pot_profile(r);
    }
    __host__ __device__ __noinline__ double den_profile(double r) const
    {
        switch (type) {
        case NBCUDA_DWARF_NFW: {
            const double R = r / a;
            return p0 * (1.0 / R) * (1.0 / ((1.0 + R) * (1.0 + R)));
        }
        case NBCUDA_DWARF_GEN_HERNQUIST:
            return (1.0 / (2.0 * M_PI)) * M * a / (r * ((r + a) * (r + a) * (r + a)));
        default:                                     // cored
            if (r <= r1) return p0 / (1.0 + (r / rc) * (r / rc));
            return ps / ((r / a) * ((1.0 + r / a) * (1.0 + r / a)));
        }
    }
    // log and atan are the CUDA library's here (the samples match the reference's in
    // distribution only, and psi is evaluated ~10^5 times per body); the set-up's below are
    // correctly rounded as the reference's
    __host__ __device__ __noinline__ double pot_profile(double r) const
    {
        switch (type) {
        case NBCUDA_DWARF_NFW: {
            const double R = r / a;
            return 4.0 * M_PI * (a * a) * p0 * (1.0 / R) * log(1.0 + R);
        }
        case NBCUDA_DWARF_GEN_HERNQUIST:
            return M / (r + a);
        default:                                     // cored
            if (r <= r1)
                return -1.0 * (4.0 * M_PI * p0 * ((rc * rc) / 2.0 * log(r * r + rc * rc) +
                                                  (rc * rc * rc) / r * atan(r / rc)) + C2);
            return -1.0 * (-4.0 * M_PI * ps * (a * a * a) / r * log(1.0 + r / a) + C3 / r);
        }
    }
};

struct NbIcDwarf {
    int first, count, nBaryon;
    NbIcComp L, D;
    double pos[3], vel[3];
    unsigned long long seed;
};

// ---- random numbers: splitmix64 (Steele, Lea & Flood 2014) per body ----
struct NbRng {
    unsigned long long s;
    __device__ double uniform()                      // [0, 1)
    {
        s += 0x9E3779B97F4A7C15ull;
        unsigned long long z = s;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        return (double) (z >> 11) * 0x1.0p-53;
    }
};

// The two components of the body's dwarf as the DF evaluation sees them: potL/potD/psi/den
// and the masses and scale lengths.  Two forms: both components Plummer, held in
// registers (the common case; the potential is evaluated ~10^5 times per body), and any
// profiles, read from the device table.
struct NbIcPlummerModel {
    double ML, aL, MD, aD;
    // of the body's own component: the density's constant, the scale length and its reciprocal
    double rho, a, ra;
    bool shared;                // masses and scales in the ranges of the shared reciprocals
    __device__ NbIcPlummerModel(double ML_, double aL_, double MD_, double aD_, bool dark)
        : ML(ML_), aL(aL_), MD(MD_), aD(aD_)
    {
        const double M = dark ? MD : ML;
        a = dark ? aD : aL;
        ra = 1.0 / a;
        rho = (3.0 / (4.0 * M_PI)) * (M / (a * a * a));
        shared = nb_exp_in<-700, 700>(ML) && nb_exp_in<-700, 700>(MD) &&
                 nb_pos_exp_in<-49, 49>(aL) && nb_pos_exp_in<-49, 49>(aD) && !nb_near_ones(a);
    }
    __device__ double potL(double r) const { return ML / sqrt(r * r + aL * aL); }
    __device__ double potD(double r) const { return MD / sqrt(r * r + aD * aD); }
    __device__ double psi(double r) const { return potL(r) + potD(r); }
    __device__ double den(bool, double r) const
    {
        const double x = 1.0 + (r / a) * (r / a);
        return rho * (1.0 / sqrt(x * x * x * x * x));
    }
    __device__ double massL() const { return ML; }
    __device__ double massD() const { return MD; }
    __device__ double scaleL() const { return aL; }
    __device__ double scaleD() const { return aD; }
    // M / sqrt(s) with a shared reciprocal (nb_rdiv.cuh); ok falls outside its range
    __device__ __forceinline__ static double over_root(double M, double s, bool& ok)
    {
        double y;
        const double root = nb_sqrt_recip(s, nb_rsqrt_estimate(s), y);
        ok &= nb_pos_exp_in<-100, 100>(s) && !nb_near_ones(s);
        return nb_quot(M, root, y);
    }
    // potL, potD and den at the five stencil points of x, rounded as the functions above: the
    // divisions and roots share their reciprocals, and no branch keeps the fifteen chains from
    // overlapping
    __device__ __forceinline__ void stencils(bool dark, double x, double (&L)[5], double (&D)[5],
                                             double (&R)[5]) const
    {
        const double h = 0.001;
        const double r[5] = {x - 2.0 * h, x - h, x, x + h, x + 2.0 * h};
        bool ok = shared;
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            L[k] = over_root(ML, r[k] * r[k] + aL * aL, ok);
            D[k] = over_root(MD, r[k] * r[k] + aD * aD, ok);
            const double q = nb_quot(r[k], a, ra);
            const double w = 1.0 + q * q;
            const double w5 = w * w * w * w * w;
            double y;
            const double root = nb_sqrt_recip(w5, nb_rsqrt_estimate(w5), y);
            ok &= nb_pos_exp_in<-1, 400>(w5) && !nb_near_ones(w5);
            R[k] = rho * nb_recip_step(root, y);
        }
        if (!ok) {
#pragma unroll 1
            for (int k = 0; k < 5; ++k) {
                const double rk = k == 0 ? r[0] : k == 1 ? r[1] : k == 2 ? r[2] : k == 3 ? r[3] : r[4];
                const double l = potL(rk), d = potD(rk), e = den(dark, rk);
#pragma unroll
                for (int q = 0; q < 5; ++q)
                    if (q == k) { L[q] = l; D[q] = d; R[q] = e; }
            }
        }
    }
};
struct NbIcModel {
    const NbIcComp* __restrict__ L;
    const NbIcComp* __restrict__ D;
    __device__ double potL(double r) const { return L->pot(r); }
    __device__ double potD(double r) const { return D->pot(r); }
    __device__ double psi(double r) const { return L->pot(r) + D->pot(r); }
    __device__ double den(bool dark, double r) const { return dark ? D->den(r) : L->den(r); }
    __device__ double massL() const { return L->M; }
    __device__ double massD() const { return D->M; }
    __device__ double scaleL() const { return L->a; }
    __device__ double scaleD() const { return D->a; }
    __device__ __forceinline__ void stencils(bool dark, double x, double (&vL)[5], double (&vD)[5],
                                             double (&vR)[5]) const
    {
        const double h = 0.001;
        const double r[5] = {x - 2.0 * h, x - h, x, x + h, x + 2.0 * h};
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            vL[k] = potL(r[k]);
            vD[k] = potD(r[k]);
            vR[k] = den(dark, r[k]);
        }
    }
};

// The five-point stencils take their values at x - 2h, x - h, x, x + h, x + 2h (h = 0.001).
// first_derivative / second_derivative from those values
__device__ __forceinline__ double ic_d1(const double (&v)[5])
{
    const double h = 0.001;
    const double p1 = 1.0 * v[0], p2 = -8.0 * v[1], p3 = -1.0 * v[4], p4 = 8.0 * v[3];
    return (p1 + p2 + p3 + p4) * (1.0 / (12.0 * h));
}
__device__ __forceinline__ double ic_d2(const double (&v)[5])
{
    const double h = 0.001;
    const double p1 = -1.0 * v[4], p2 = 16.0 * v[3], p3 = -30.0 * v[2];
    const double p4 = 16.0 * v[1], p5 = -1.0 * v[0];
    return (p1 + p2 + p3 + p4 + p5) * (1.0 / (12.0 * h * h));
}

// the DF integrand d^2 rho / d psi^2 / sqrt(|E - psi|) at radius ri (fun)
template <typename Model>
__device__ __forceinline__ double ic_integrand(const Model& m, double ri, double energy, bool dark)
{
    double L[5], D[5], R[5];
    m.stencils(dark, ri, L, D, R);
    double dpsi = ic_d1(L) + ic_d1(D);
    const double d2psi = ic_d2(L) + ic_d2(D);
    const double dden = ic_d1(R), d2den = ic_d2(R);
    if (dpsi == 0.0) dpsi = 1.0e-6;
    const double dsq = d2den * (1.0 / dpsi) - dden * d2psi * (1.0 / (dpsi * dpsi));
    const double diff = fabs(energy - (L[2] + D[2]));
    const double denom = diff != 0.0 ? 1.0 / sqrt(diff)
                                     : 1.0 / sqrt(fabs(energy - m.psi(ri + 0.0001)));
    return dsq * denom;
}

// A warp samples one body.  Its lanes follow the body's rejections and searches together and
// share out what a step evaluates many of: the quadrature's 330 integrand points (ten panels of
// three points at a time) and the bisection's midpoints (the 31 of its next five steps).  Sums
// and decisions keep the order of the one-thread form, so the samples are the same bit for bit.
// A body takes 10 to 60 evaluations of the distribution function of 330 x ~450 FP64 operations
// each: with a thread a body the warps waited for their longest body and a few long ones set
// the time (eight dwarfs of 4,096 to 65,536 bodies: 185 -> 83 ms, and 62 with the shared
// reciprocals of NbIcPlummerModel::stencils).  FP64 issue and its dependences bound it now; five
// resident blocks (96 registers; 300 bytes of spill stores with two Plummer components, 644 with
// others) beat four by 2 % and three by 10 %.
struct NbIcWarp {
    int lane;
    double* terms;              // 32 doubles of shared memory
};

// composite three-point Gauss quadrature: 100 panels over [a, 1.5 a], then 10 up to b
template <typename Model>
__device__ double ic_gauss_quad(const NbIcWarp& w, const Model& m, double lower, double upper,
                                double energy, bool dark)
{
    const double a = lower > upper ? upper : lower, b = lower > upper ? lower : upper;
    const double benchmark = 1.5 * a;
    double hg = (benchmark - a) / 100.0;
    double lowerg = a, upperg = lowerg + hg;
    double coef2 = (lowerg + upperg) / 2.0, coef1 = (upperg - lowerg) / 2.0;
    const double c1 = 0.55555555555, c2 = 0.88888888888, c3 = 0.55555555555;
    const double x1 = -0.77459666924, x3 = 0.77459666924;
    const int panel = w.lane / 3, point = w.lane % 3;       // of the ten panels at a time
    double intv = 0.0;
    int counter = 0;
    for (bool done = false; !done;) {
        double my1 = 0.0, my2 = 0.0;
        int panels = 0;
        for (; panels < 10 && !done; ++panels) {
            if (panel == panels) { my1 = coef1; my2 = coef2; }
            lowerg = upperg;
            upperg = upperg + hg;
            coef2 = (lowerg + upperg) / 2.0;
            coef1 = (upperg - lowerg) / 2.0;
            if (lowerg > benchmark) hg = (b - benchmark) / 10.0;
            if (upper > lower) { if (lowerg >= upper) done = true; }
            else if (lower > upper) { if (lowerg >= lower) done = true; }
            if (++counter > 100000) done = true;
        }
        double term = 0.0;
        if (panel < panels) {
            const double x = point == 0 ? my1 * x1 + my2 : point == 1 ? my2 : my1 * x3 + my2;
            const double c = point == 0 ? c1 : point == 1 ? c2 : c3;
            term = c * ic_integrand(m, x, energy, dark) * my1;
        }
        __syncwarp();
        w.terms[w.lane] = term;
        __syncwarp();
        for (int t = 0; t < 3 * panels; ++t) intv = intv + w.terms[t];
    }
    return lower > upper ? -intv : intv;
}

// bisection for psi(r) = value on [lo, hi] split in 4 intervals (root_finder); 0 if none
template <typename Model>
__device__ double ic_root(const NbIcWarp& w, const Model& m, double value, double lo, double hi)
{
    double x = ((hi - lo) * (double) min(w.lane, 4)) / 4.0 + lo;
    double v = m.psi(x) - value;
    if (isnan(v)) { x += 0.0001; v = m.psi(x) - value; }
    for (int q = 0; q < 4; ++q) {
        const double v0 = __shfl_sync(NB_FULL_MASK, v, q), v1 = __shfl_sync(NB_FULL_MASK, v, q + 1);
        const double b0 = __shfl_sync(NB_FULL_MASK, x, q), b1 = __shfl_sync(NB_FULL_MASK, x, q + 1);
        double nlo, nhi;
        if (v0 < 0 && v1 > 0) { nlo = b0; nhi = b1; }
        else if (v0 > 0 && v1 < 0) { nlo = b1; nhi = b0; }
        else continue;
        double mid = 0.0, f = 1.0;
        int counter = 0;
        while (fabs(f) > .0001 && counter <= 10000) {
            // lane h (1 .. 31) holds the midpoint reached from here by the steps that the bits of
            // h after its first one spell: a one where psi - value was negative
            double l = nlo, r = nhi;
            const int h0 = max(w.lane, 1);
            for (int d = 30 - __clz(h0); d >= 0; --d) {
                const double c = (l + r) / 2.0;
                if ((h0 >> d) & 1) l = c; else r = c;
            }
            const double myMid = (l + r) / 2.0;
            const double myF = m.psi(myMid) - value;
            for (int h = 1; h < 32 && fabs(f) > .0001 && counter <= 10000; ++counter) {
                mid = __shfl_sync(NB_FULL_MASK, myMid, h);
                f = __shfl_sync(NB_FULL_MASK, myF, h);
                if (f < 0.0) { nlo = mid; h = 2 * h + 1; }
                else { nhi = mid; h = 2 * h; }
            }
        }
        return mid;
    }
    return 0.0;
}

// the Eddington DF at speed v and radius r (dist_fun)
template <typename Model>
__device__ double ic_df(const NbIcWarp& w, const Model& m, double v, double r, bool dark)
{
    const double cons = 0.03582244801567226;
    const double energy = m.psi(r) - 0.5 * v * v;
    const double ML = m.massL(), MD = m.massD(), aL = m.scaleL(), aD = m.scaleD();
    double range = MD == 0 ? 20.0 * sqrt(fabs((ML / energy) * (ML / energy) - aL * aL))
                           : 20.0 * sqrt(fabs((MD / energy) * (MD / energy) - aD * aD));
    for (int counter = 0; m.psi(range) > energy; ++counter) {
        range = 100.0 * range;
        if (counter > 100) { range = 100.0 * (aL + aD); break; }
    }
    double up = ic_root(w, m, energy, 0.0, range);
    if (isinf(up) || up == 0.0 || isnan(up)) up = r;        // find_upperlimit_r's fallback
    up = fabs(up);
    const double lo = 10.0 * up;
    return v * v * cons * ic_gauss_quad(w, m, lo, up, energy, dark);
}

// golden-section search for the DF maximum over speeds (max_finder)
template <typename Model>
__device__ double ic_df_max(const NbIcWarp& w, const Model& m, double r, bool dark, double a,
                            double b, double c, int limit, double tol)
{
    const double R = 0.61803399, C = 1.0 - R;
    double x0 = a, x3 = c, x1, x2;
    if (fabs(b - c) > fabs(b - a)) { x1 = b; x2 = b + (C * (c - b)); }
    else { x2 = b; x1 = b - (C * (b - a)); }
    double f1 = 0.0, f2 = 0.0;
    // one call of ic_df in the code (its quadrature is inlined): first at x1, then x2, then the
    // point each step replaces
    int counter = -2;
    bool second = false;
    for (;;) {
        const double f = -ic_df(w, m, second ? x2 : x1, r, dark);
        if (second) f2 = f; else f1 = f;
        if (++counter == -1) { second = true; continue; }
        if (counter > limit) break;                 // counter: the steps taken
        if (!(fabs(x3 - x0) > (tol * (fabs(x1) + fabs(x2))))) break;
        second = f2 < f1;
        if (second) { x0 = x1; x1 = x2; x2 = R * x2 + C * x3; f1 = f2; }
        else { x3 = x2; x2 = x1; x1 = R * x1 + C * x0; f2 = f1; }
    }
    return f1 < f2 ? -f1 : -f2;
}

__device__ void ic_direction(NbRng& rng, double rad, double out[3])
{
    double x, y, z, rsq;
    int guard = 0;
    do {
        x = 2.0 * rng.uniform() - 1.0;
        y = 2.0 * rng.uniform() - 1.0;
        z = 2.0 * rng.uniform() - 1.0;
        rsq = x * x + y * y + z * z;
    } while ((rsq > 1.0 || rsq == 0.0) && ++guard < 1000);
    const double s = rad / sqrt(rsq);
    out[0] = x * s; out[1] = y * s; out[2] = z * s;
}

__device__ __forceinline__ unsigned long long ic_mix(unsigned long long z)
{
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__device__ int ic_dwarf_of(const NbIcDwarf* dw, int nD, int i)
{
    int lo = 0, hi = nD - 1;
    while (lo < hi) {                                 // last dwarf with first <= i
        const int mid = (lo + hi + 1) >> 1;
        if (dw[mid].first <= i) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// The radius and speed of one body by rejection (r_mag, vel_mag); r = v = 0 when either fails.
template <typename Model>
__device__ void ic_sample_rv(const NbIcWarp& w, const Model& m, const NbIcComp& comp, bool dark, NbRng& rng,
                             double& rOut, double& vOut)
{
    double r = 0.0;
    for (int tries = 0; tries <= 1000 && !(isfinite(r) && r != 0.0); ++tries) {
        r = 0.0;
        for (int counter = 0; counter <= 1000; ++counter) {      // r_mag
            const double rr = rng.uniform() * comp.bound;
            const double u = rng.uniform();
            if (rr * rr * m.den(dark, rr) / comp.rhoMax > u) { r = rr; break; }
        }
    }
    double v = 0.0;
    if (isfinite(r) && r != 0.0) {
        const double vesc = 0.99 * sqrt(fabs(2.0 * m.psi(r)));
        const double dfMax = ic_df_max(w, m, r, dark, 0.0, 0.5 * vesc, vesc, 10, 1.0e-2);
        for (int tries = 0; tries <= 1000 && !(isfinite(v) && v != 0.0); ++tries) {
            v = 0.0;
            for (int counter = 0; counter <= 1000; ++counter) {  // vel_mag
                const double vv = rng.uniform() * vesc;
                const double u = rng.uniform();
                if (fabs(ic_df(w, m, vv, r, dark) / dfMax) > u) { v = vv; break; }
            }
        }
    }
    rOut = r;
    vOut = v;
}

// One body per warp: radius and speed by rejection, isotropic directions.  ALL_PLUMMER: every
// dwarf of the table has two Plummer components (their model in registers).
constexpr int kIcWarps = 4;
template <bool ALL_PLUMMER>
__global__ void __launch_bounds__(32 * kIcWarps, 5)
k_ic_sample(const NbIcDwarf* __restrict__ dwarfs, int nD, int n,
                            double* __restrict__ px, double* __restrict__ py,
                            double* __restrict__ pz, double* __restrict__ vx,
                            double* __restrict__ vy, double* __restrict__ vz,
                            double* __restrict__ mass, int* __restrict__ types,
                            NbScalars* __restrict__ sc)
{
    __shared__ double terms[kIcWarps][32];
    const NbIcWarp w{(int) (threadIdx.x & 31), terms[threadIdx.x >> 5]};
    for (int i = blockIdx.x * kIcWarps + (threadIdx.x >> 5); i < n; i += gridDim.x * kIcWarps) {
        const NbIcDwarf& d = dwarfs[ic_dwarf_of(dwarfs, nD, i)];
        const int k = i - d.first;
        const bool dark = k >= d.nBaryon;
        NbRng rng{ic_mix(d.seed ^ ic_mix((unsigned long long) k + 0x51ED27ull))};
        const NbIcComp& comp = dark ? d.D : d.L;
        double r, v;
        if (ALL_PLUMMER) {
            const NbIcPlummerModel m(d.L.M, d.L.a, d.D.M, d.D.a, dark);
            ic_sample_rv(w, m, comp, dark, rng, r, v);
        } else {
            const NbIcModel m{&d.L, &d.D};
            ic_sample_rv(w, m, comp, dark, rng, r, v);
        }
        if (!(isfinite(r) && r != 0.0 && isfinite(v) && v != 0.0)) {
            nb_raise(sc, NBODY_ERROR);                // the reference exits here
            r = v = 0.0;
        }
        double dv[3], dr[3];
        ic_direction(rng, v, dv);
        ic_direction(rng, r, dr);
        if (w.lane != 0) continue;
        px[i] = dr[0]; py[i] = dr[1]; pz[i] = dr[2];
        vx[i] = dv[0]; vy[i] = dv[1]; vz[i] = dv[2];
        const int nDark = d.count - d.nBaryon;
        mass[i] = dark ? (nDark ? d.D.M / (double) nDark : 0.0)
                       : (d.nBaryon ? d.L.M / (double) d.nBaryon : 0.0);
        types[i] = dark ? -1 : 1;
    }
}

// Per (dwarf, component): sums of m x and m v, one block per component.  Each thread adds its
// strided share of the component's bodies in index order and the block combines the threads'
// sums by a fixed tree, so the sums -- and the recentred bodies -- are the same on every run
// (floating-point atomics would add in arrival order).
constexpr int kIcMomentThreads = 512;

__global__ void __launch_bounds__(kIcMomentThreads)
k_ic_moments(const NbIcDwarf* __restrict__ dwarfs, int nD,
             const double* __restrict__ px, const double* __restrict__ py,
             const double* __restrict__ pz, const double* __restrict__ vx,
             const double* __restrict__ vy, const double* __restrict__ vz,
             const double* __restrict__ mass, double* __restrict__ sums)
{
    __shared__ double part[6][kIcMomentThreads];
    const int seg = blockIdx.x;                       // 2 * dwarf + (dark component)
    const NbIcDwarf& d = dwarfs[seg >> 1];
    const bool dark = seg & 1;
    const int lo = d.first + (dark ? d.nBaryon : 0);
    const int hi = dark ? d.first + d.count : d.first + d.nBaryon;
    double s[6] = {0, 0, 0, 0, 0, 0};
    for (int i = lo + (int) threadIdx.x; i < hi; i += kIcMomentThreads) {
        const double mi = mass[i];
        s[0] += mi * px[i]; s[1] += mi * py[i]; s[2] += mi * pz[i];
        s[3] += mi * vx[i]; s[4] += mi * vy[i]; s[5] += mi * vz[i];
    }
    for (int c = 0; c < 6; ++c) part[c][threadIdx.x] = s[c];
    __syncthreads();
    for (int w = kIcMomentThreads / 2; w > 0; w >>= 1) {
        if ((int) threadIdx.x < w)
            for (int c = 0; c < 6; ++c) part[c][threadIdx.x] += part[c][threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x < 6) sums[6 * (size_t) seg + threadIdx.x] = part[threadIdx.x][0];
}

// x - cm + shift, v - cv + shift per component (cm = sum m x / component mass)
__global__ void k_ic_shift(const NbIcDwarf* __restrict__ dwarfs, int nD, int n,
                           double* __restrict__ px, double* __restrict__ py,
                           double* __restrict__ pz, double* __restrict__ vx,
                           double* __restrict__ vy, double* __restrict__ vz,
                           const double* __restrict__ sums)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int dwi = ic_dwarf_of(dwarfs, nD, i);
        const NbIcDwarf& d = dwarfs[dwi];
        const bool dark = i - d.first >= d.nBaryon;
        const double cm = dark ? d.D.M : d.L.M;
        const double* s = sums + 6 * (size_t) (2 * dwi + dark);
        px[i] = px[i] - s[0] / cm + d.pos[0];
        py[i] = py[i] - s[1] / cm + d.pos[1];
        pz[i] = pz[i] - s[2] / cm + d.pos[2];
        vx[i] = vx[i] - s[3] / cm + d.vel[0];
        vy[i] = vy[i] - s[4] / cm + d.vel[1];
        vz[i] = vz[i] - s[5] / cm + d.vel[2];
    }
}

}  // namespace

namespace {

// The component's constants as nbGenerateMixedDwarfCore sets them up: set_vars
// (nbody_mixeddwarf.c:696-726), the sampling bound with get_extra_nfw_mass for NFW and cored
// components (:728-762, :797-831), the cored potential's constants (cored_pot,
// nbody_dwarf_potential.c:139-175) and the maximum of r^2 rho at its analytic radius (:873-903).
// rscaleL and rscaleD: both components' scale lengths (the Plummer/Hernquist bound).
NbIcComp nb_ic_setup(const NBodyCudaDwarfComponent& in, double rscaleL, double rscaleD)
{
    NbIcComp c{};
    c.type = in.type;
    c.M = in.mass;
    c.a = in.scaleLength;
    c.r1 = in.r1;
    c.rc = in.rc;
    const double rs = c.a, r1 = c.r1, rc = c.rc;
    const bool cored = c.type == NBCUDA_DWARF_CORED;
    const double r200 = cbrt(c.M / kVolPcrit);
    if (cored) {
        const double D1 = r1 * ((1.0 + r1 / rs) * (1.0 + r1 / rs)) / (rs + rs * ((r1 / rc) * (r1 / rc)));
        const double D2 = (rs * rs * rs) * (nb_log_rn(1.0 + r200 / rs) - nb_log_rn(1.0 + r1 / rs) -
                                            r200 / (rs + r200) + r1 / (rs + r1));
        const double D3 = (rc * rc) * (r1 - rc * nb_atan_rn(r1 / rc));
        c.p0 = c.M / (4.0 * M_PI * (D1 * D2 + D3));
        c.ps = c.p0 * D1;
    } else {
        const double conc = r200 / rs;
        const double term = nb_log_rn(1.0 + conc) - conc / (1.0 + conc);
        c.p0 = 200.0 * (conc * conc * conc) * kPcrit / (3.0 * term);
    }
    if (c.type == NBCUDA_DWARF_NFW || cored) {
        c.bound = 5.0 * r200;
        const double r = c.bound;                    // the mass inside the bound
        if (cored) {
            const double C1 = 0;
            const double C3 = C1 + 4 * M_PI * (c.ps * (rs * rs * rs) * (nb_log_rn((1 + r1 / rs)) - r1 / (rs + r1)) -
                                               c.p0 * (rc * rc) * (r1 - rc * nb_atan_rn(r1 / rc)));
            if (r <= r1)
                c.M = 4.0 * M_PI * c.p0 * (rc * rc) * (r - rc * nb_atan_rn(r / rc)) - C1;
            else
                c.M = 4.0 * M_PI * c.ps * (rs * rs * rs) * (nb_log_rn((rs + r) / rs) - r / (rs + r)) - C3;
        } else {
            c.M = 4.0 * M_PI * c.p0 * (rs * rs * rs) * (nb_log_rn((rs + r) / rs) - r / (rs + r));
        }
    } else {
        c.bound = 50.0 * (rscaleL + rscaleD);
    }
    if (cored) {
        c.C3 = 4.0 * M_PI * (c.ps * (rs * rs * rs) * (nb_log_rn((1.0 + r1 / rs)) - r1 / (rs + r1)) -
                             c.p0 * (rc * rc) * (r1 - rc * nb_atan_rn(r1 / rc)));
        c.C2 = c.C3 / r1 - (4.0 * M_PI) / r1 *
                               (c.ps * (rs * rs * rs) * nb_log_rn(1 + r1 / rs) +
                                c.p0 * (((rc * rc) * r1) / 2.0 * nb_log_rn((r1 * r1) + (rc * rc)) +
                                        (rc * rc * rc) * nb_atan_rn(r1 / rc)));
    }
    double rmax;
    switch (c.type) {
    case NBCUDA_DWARF_NFW: rmax = rs; break;
    case NBCUDA_DWARF_GEN_HERNQUIST: rmax = rs / 2.0; break;
    case NBCUDA_DWARF_CORED: rmax = rs > r1 ? rs : r1; break;
    default: rmax = sqrt(2.0 / 3.0) * rs; break;
    }
    c.rhoMax = (rmax * rmax) * c.den(rmax);
    return c;
}

}  // namespace

// The two components' particle masses as the sampler assigns them (after the NFW/cored reset).
void nb_ic_particle_masses(const NBodyCudaMixedDwarf& h, double out[2])
{
    const NbIcComp L = nb_ic_setup(h.light, h.light.scaleLength, h.dark.scaleLength);
    const NbIcComp D = nb_ic_setup(h.dark, h.light.scaleLength, h.dark.scaleLength);
    const int nDark = h.nbody - h.nbodyBaryon;
    out[0] = h.nbodyBaryon ? L.M / (double) h.nbodyBaryon : 0.0;
    out[1] = nDark ? D.M / (double) nDark : 0.0;
}

// Samples every dwarf of the table into the SoA body arrays (bodies [first, first + count) of
// each dwarf) and their types; scratch needs 12 doubles per dwarf.  One launch per phase for all
// dwarfs.  Returns the number of launches.
int nb_launch_ic(const NBodyCudaMixedDwarf* host, int nD, const int* firsts, void* dTable,
                 double* scratch, NbTreeBuffers& b, int* types, int n, int numSMs, NbScalars* sc,
                 cudaStream_t s)
{
    std::vector<NbIcDwarf> t(nD);
    for (int k = 0; k < nD; ++k) {
        const NBodyCudaMixedDwarf& h = host[k];
        NbIcDwarf& d = t[k];
        d.first = firsts[k];
        d.count = h.nbody;
        d.nBaryon = h.nbodyBaryon;
        d.L = nb_ic_setup(h.light, h.light.scaleLength, h.dark.scaleLength);
        d.D = nb_ic_setup(h.dark, h.light.scaleLength, h.dark.scaleLength);
        for (int c = 0; c < 3; ++c) { d.pos[c] = h.position[c]; d.vel[c] = h.velocity[c]; }
        d.seed = h.seed;
    }
    cudaMemcpyAsync(dTable, t.data(), sizeof(NbIcDwarf) * nD, cudaMemcpyHostToDevice, s);
    cudaMemsetAsync(scratch, 0, sizeof(double) * 12 * (size_t) nD, s);
    const NbIcDwarf* dt = (const NbIcDwarf*) dTable;
    // few bodies per warp, many warps: the per-body work is long and uneven
    const int g = min((n + kIcWarps - 1) / kIcWarps, numSMs * 64);
    bool allPlummer = true;
    for (const NbIcDwarf& d : t)
        allPlummer = allPlummer && d.L.type == NBCUDA_DWARF_PLUMMER && d.D.type == NBCUDA_DWARF_PLUMMER;
    if (allPlummer)
        k_ic_sample<true><<<g, 32 * kIcWarps, 0, s>>>(dt, nD, n, b.px, b.py, b.pz, b.vx, b.vy, b.vz, b.mass, types, sc);
    else
        k_ic_sample<false><<<g, 32 * kIcWarps, 0, s>>>(dt, nD, n, b.px, b.py, b.pz, b.vx, b.vy, b.vz, b.mass, types, sc);
    const int g2 = min((n + 255) / 256, numSMs * 8);
    k_ic_moments<<<2 * nD, kIcMomentThreads, 0, s>>>(dt, nD, b.px, b.py, b.pz, b.vx, b.vy, b.vz,
                                                     b.mass, scratch);
    k_ic_shift<<<g2, 256, 0, s>>>(dt, nD, n, b.px, b.py, b.pz, b.vx, b.vy, b.vz, scratch);
    nb_count_launch(3);
    return 3;
}

size_t nb_ic_table_bytes(int nD) { return sizeof(NbIcDwarf) * (size_t) nD; }
