// One RK stage of the plain FP64 form over the digit-product transforms (tcdft.cu).
//
// With the transforms off the FP64 pipe, the stage is a sequence of passes over the fields: the
// nonlinear term, one update kernel for all components, the wall round trips of vx, vy and theta as one
// batch, one Poisson kernel that also takes the wall sums of vz, the pressure's and theta's inverse
// transforms as one batch, one correction kernel with the precomputed profile spectra, and theta's
// forward transform.  Mathematics and order are the reference's (hd_rkstep2.f90, bouss_rkstep2.f90,
// rotbouss_rkstep2.f90, vboundary.f90:67-151, boundary_mod.fpp:197-402).  The elementwise kernels are
// bound by the FP64 pipe (about 25 operations a point each), so factors that the components share are
// formed once a point.
#include "chain.h"
#include "fast.h"
#include "kernels_elem.cuh"
#include "smem.h"
#include "stage_f64.h"
#include "tcdft.h"

namespace sg {

namespace {

#define SG_TRY(x)                  \
    do {                           \
        int _st = (x);             \
        if (_st != OK) return _st; \
    } while (0)

__device__ __forceinline__ double2 axpy(double2 y, double s, double2 x) {
    y.x = fma(s, x.x, y.x);
    y.y = fma(s, x.y, y.y);
    return y;
}

// v = C + dt/o * (nu * (-k^2 v) - filter * N), N with the Coriolis, buoyancy and heat-current terms
struct UpdateArgs {
    const double2 *n[4], *v[4], *c[4];
    double2 *out[4];
    double anu, akappa, adt;  // dt/o * nu, dt/o * kappa, dt/o
    double xmom, xtemp, om[3];
    int nc, rot;
};
__global__ void __launch_bounds__(256) k_stage_update(Geo g, UpdateArgs a) {
    chain_wait();
    SG_ELEMS_BEGIN(g, 0, g.nz)
        const double kxv = g.kx[kx], kyv = g.ky[ky], kzv = g.kz[z];
        const double k2 = kxv * kxv + kyv * kyv + kzv * kzv;
        const double f = -a.adt * (g.fx[kx] * g.fy[ky] * g.fz[z]), anu = -a.anu * k2;
        double2 v[4], n[4];
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (i < a.nc) {
                v[i] = a.v[i][q];
                n[i] = a.n[i][q];
            }
        if (a.rot) {
            n[0] = axpy(axpy(n[0], 2 * a.om[1], v[2]), -2 * a.om[2], v[1]);
            n[1] = axpy(axpy(n[1], 2 * a.om[2], v[0]), -2 * a.om[0], v[2]);
            n[2] = axpy(axpy(n[2], 2 * a.om[0], v[1]), -2 * a.om[1], v[0]);
        }
        if (a.nc == 4) {
            n[2] = axpy(n[2], -a.xmom, v[3]);
            n[3] = axpy(n[3], -a.xtemp, v[2]);
        }
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (i < a.nc) a.out[i][q] = axpy(axpy(a.c[i][q], i == 3 ? -a.akappa * k2 : anu, v[i]), f, n[i]);
    SG_ELEMS_END
}

// no-slip walls of vx, vy from the previous pressure (k_noslip) and theta = 0 at the walls
__global__ void __launch_bounds__(64) k_stage_walls(Geo g, double2 *vx, double2 *vy, double2 *th, const double2 *pr, double tmp,
                                                    WallVel vb) {
    chain_wait();
    const int kx = blockIdx.x * blockDim.x + threadIdx.x, ky = blockIdx.y;
    if (kx >= g.nxh) return;
    for (int w = 0; w < 2; w++) {
        const size_t q = fidx<double>(g, w == 0 ? 0 : g.nzp - 1, ky, kx);
        const double2 p = pr[q];
        vx[q] = cscale(cimk(g.kx[kx], p), tmp);
        vy[q] = cscale(cimk(g.ky[ky], p), tmp);
        if (kx == 0 && ky == 0) {
            const double nn = (double)g.nx * g.ny;
            vx[q] = make_double2(nn * (w == 0 ? vb.x : vb.z), 0.0);
            vy[q] = make_double2(nn * (w == 0 ? vb.y : vb.w), 0.0);
        }
        if (th) th[q] = make_double2(0.0, 0.0);
    }
}

// Poisson solve and correction of the velocity (boundary_mod.fpp:405-448, :245-281), the wall values of
// vz by direct sums over kz, and from them the Neumann laplace_z coefficients (:521-549); theta's filter
// beside it.  A block holds 32 kx of one ky, eight slices of kz.
constexpr int kSlices = 8;
__global__ void __launch_bounds__(32 * kSlices) k_stage_poisson(Geo g, double2 *vx, double2 *vy, double2 *vz, double2 *d,
                                                                double2 *th, double2 *coef) {
    __shared__ double4 red[kSlices][32];
    const int kx = blockIdx.x * 32 + threadIdx.x, ky = blockIdx.y;
    const bool on = kx < g.nxh;
    chain_wait();
    double4 w = make_double4(0, 0, 0, 0);
    if (on) {
        const double kxv = g.kx[kx], kyv = g.ky[ky], kh2 = kxv * kxv + kyv * kyv, fxy = th ? g.fx[kx] * g.fy[ky] : 0.0;
        const double2 *wt = (const double2 *)g.wtw;
#pragma unroll 2
        for (int z = threadIdx.y; z < g.nz; z += kSlices) {
            const size_t q = fidx<double>(g, z, ky, kx);
            const double kzv = g.kz[z];
            double2 A = vx[q], B = vy[q], C = vz[q];
            const double k2 = fma(kzv, kzv, kh2);
            const double r = q == 0 ? 0.0 : 1.0 / k2;
            const double sx = kxv * A.x + kyv * B.x + kzv * C.x, sy = kxv * A.y + kyv * B.y + kzv * C.y;
            const double2 D = make_double2(sy * r, -sx * r);  // -i s / k^2
            A = csub(A, cimk(kxv, D));
            B = csub(B, cimk(kyv, D));
            C = csub(C, cimk(kzv, D));
            vx[q] = A;
            vy[q] = B;
            vz[q] = C;
            d[q] = D;
            const double2 t = __ldg(wt + z);
            w.x += C.x;
            w.y += C.y;
            w.z += C.x * t.x - C.y * t.y;
            w.w += C.x * t.y + C.y * t.x;
            if (th) th[q] = cscale(th[q], fxy * g.fz[z]);
        }
    }
    red[threadIdx.y][threadIdx.x] = w;
    __syncthreads();
    if (threadIdx.y || !on) return;
    for (int i = 1; i < kSlices; i++) {
        const double4 o = red[i][threadIdx.x];
        w.x += o.x; w.y += o.y; w.z += o.z; w.w += o.w;
    }
    const double inv = 1.0 / (double)g.nz;
    const double2 b1 = make_double2(w.x * inv, w.y * inv), b2 = make_double2(w.z * inv, w.w * inv);
    const size_t col = (size_t)ky * g.nxh + kx;
    double2 c1 = b1, c2 = make_double2(0.0, 0.0);
    if (kx || ky) {
        const double *lc = g.lapc + col * 3;  // kh, exp(-kh Lz), 1 / (kh (1 - exp(-2 kh Lz)))
        const double e = lc[1], t = lc[2];
        c1 = make_double2((b2.x - b1.x * e) * t, (b2.y - b1.y * e) * t);
        c2 = make_double2((-b1.x + b2.x * e) * t, (-b1.y + b2.y * e) * t);
    }
    coef[2 * col] = c1;
    coef[2 * col + 1] = c2;
}

// pr = the harmonic profile c1 exp(kh (z - Lz)) + c2 exp(-kh z) on the physical rows (the potential's
// inverse transform is added to it).  Two exponentials a row would bind it to the FP64 pipe (6.4 ms at
// 512^2 x 513); with z = (32 i + j) dz, exp(-kh z) is the product of two table entries, and
// exp(kh (z - Lz)) is the same read from the other wall.  A block holds 32 columns.
constexpr int kProfJ = 32;
// With `deriv` also the profile's z derivative, and then all nz rows (those above nzp one by one).
__global__ void __launch_bounds__(256) k_stage_profile(Geo g, const double2 *coef, double2 *prof, double2 *deriv, double dz) {
    extern __shared__ double tab[];  // [32 + ni][32 columns]: exp(-kh j dz), then exp(-kh 32 i dz)
    const int c = threadIdx.x, kx = blockIdx.x * 32 + c, ky = blockIdx.y;
    const bool on = kx < g.nxh;
    const size_t col = (size_t)ky * g.nxh + (on ? kx : 0);
    const double kh = g.lapc[col * 3];
    const int ni = (g.nzp + kProfJ - 1) / kProfJ;
    for (int t = threadIdx.y; t < kProfJ + ni; t += blockDim.y) {
        const double z = t < kProfJ ? t * dz : (t - kProfJ) * (kProfJ * dz);
        tab[t * 32 + c] = exp(-(kh * z));
    }
    __syncthreads();
    chain_wait();
    if (!on) return;
    const double2 c1 = coef[2 * col], c2 = coef[2 * col + 1];
    auto ex = [&](int z) { return tab[(z % kProfJ) * 32 + c] * tab[(kProfJ + z / kProfJ) * 32 + c]; };
    const int rows = deriv ? g.nz : g.nzp;
    for (int z = threadIdx.y; z < rows; z += blockDim.y) {
        const size_t q = fidx<double>(g, z, ky, kx);
        if (kx == 0 && ky == 0) {
            prof[q] = make_double2(c1.x * g.z[z] + c2.x, 0.0);
            if (deriv) deriv[q] = make_double2(c1.x, 0.0);
            continue;
        }
        double e1, e2;
        if (z < g.nzp) {
            e1 = ex(g.nzp - 1 - z);
            e2 = ex(z);
        } else {
            e1 = exp(kh * (g.z[z] - g.Lz));
            e2 = exp(-(kh * g.z[z]));
        }
        prof[q] = make_double2(c1.x * e1 + c2.x * e2, c1.y * e1 + c2.y * e2);
        if (deriv) deriv[q] = make_double2(kh * (c1.x * e1 - c2.x * e2), kh * (c1.y * e1 - c2.y * e2));
    }
}

// harmonic correction with the spectra E1, E2 of the unit profiles: with p = c1 E1 + c2 E2 and
// b = kh (c1 E1 - c2 E2), vx -= i kx p, vy -= i ky p, vz -= b (boundary_mod.fpp:385-399, :635-675)
__global__ void __launch_bounds__(256) k_stage_correct(Geo g, double2 *vx, double2 *vy, double2 *vz, const double2 *E1,
                                                       const double2 *E2, const double2 *coef) {
    chain_wait();
    SG_ELEMS_BEGIN(g, 0, g.nz)
        const size_t col = (size_t)ky * g.nxh + kx;
        const double2 c1 = coef[2 * col], c2 = coef[2 * col + 1];
        double2 p, b;
        if (kx == 0 && ky == 0) {  // profile c1.x z, its derivative c1.x (E2 is the spectrum of 1)
            const double2 e1 = E1[q], e2 = E2[q];
            p = cscale(e1, c1.x);
            b = cscale(e2, c1.x);
        } else {
            const double2 t1 = cmul(c1, E1[q]), t2 = cmul(c2, E2[q]);
            p = cadd(t1, t2);
            b = cscale(csub(t1, t2), __ldg(g.lapc + col * 3));
        }
        vx[q] = csub(vx[q], cimk(g.kx[kx], p));
        vy[q] = csub(vy[q], cimk(g.ky[ky], p));
        vz[q] = csub(vz[q], b);
    SG_ELEMS_END
}

// theta's c2r / r2c round trip leaves the kx = 0 and kx = nx/2 columns Hermitian over (ky, -ky)
__global__ void __launch_bounds__(128) k_stage_herm(Geo g, double2 *th) {
    chain_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x, sel = blockIdx.y;
    const int h = g.ny / 2 + 1;
    if (i >= h * g.nzp) return;
    const int ky = i % h, z = i / h, km = (g.ny - ky) % g.ny, kx = sel ? g.nxh - 1 : 0;
    const size_t q = fidx<double>(g, z, ky, kx), qm = fidx<double>(g, z, km, kx);
    const double2 p = th[q], m = th[qm];
    const double2 r = make_double2(0.5 * (p.x + m.x), 0.5 * (p.y - m.y));
    th[q] = r;
    if (km != ky) th[qm] = make_double2(r.x, -r.y);
}

int elem_blocks(const Plan &P) {
    const long long n = (long long)P.nz * P.ny * P.nxh, b = (n + 255) / 256;
    return (int)(b > kSMs * 16 ? kSMs * 16 : b);
}

}  // namespace

bool f64_stage_ok(const Plan &P) { return tc_length_ok(P.nz); }

int f64_poisson(Plan &P, void *vx, void *vy, void *vz, void *d, void *th, double2 *coef) {
    const double field = (double)P.nz * P.ny * P.nxh * 16.0;
    Launch L(P, "stage_poisson", (7.0 + (th ? 2.0 : 0.0)) * field);
    chain(k_stage_poisson, dim3(cdiv(P.nxh, 32), P.ny), dim3(32, kSlices), 0, P.stream, 
        P.geo, (double2 *)vx, (double2 *)vy, (double2 *)vz, (double2 *)d, (double2 *)th, coef);
    return check_launch("poisson");
}

int f64_profile(Plan &P, const double2 *coef, void *prof, void *deriv) {
    Launch L(P, "stage_profile", (deriv ? 2.0 * P.nz : (double)P.nzp) * P.ny * P.nxh * 16.0);
    const size_t sm = (size_t)(kProfJ + cdiv(P.nzp, kProfJ)) * 32 * sizeof(double);
    allow_smem(k_stage_profile, sm);
    chain(k_stage_profile, dim3(cdiv(P.nxh, 32), P.ny), dim3(32, 8), sm, P.stream, P.geo, coef, (double2 *)prof, (double2 *)deriv, P.dz);
    return check_launch("profile");
}

int f64_stage(Plan &P, const StageParams &sp, int o, const void *const vin[4], const void *const cold[4],
              void *const vout[4], void *pr, void *const E[2]) {
    const bool bouss = sp.solver >= 1, rot = sp.solver == 2;
    const int nc = bouss ? 4 : 3;
    const double field = (double)P.nz * P.ny * P.nxh * 16.0, mixed = (double)P.nzp * P.ny * P.nxh * 16.0;
    void *N[4] = {nullptr, nullptr, nullptr, nullptr}, *d = P.scratch_field(0);
    for (int i = 0; i < nc; i++) N[i] = P.scratch_field(18 + i);
    double2 *coef = (double2 *)P.scratch_field(16);
    if (!d || !coef || !N[0] || !N[1] || !N[2] || (bouss && !N[3])) {
        set_error("out of device memory (FP64 stage)");
        return ERR_OOM;
    }
    const void *v3[3] = {vin[0], vin[1], vin[2]};
    SG_TRY(Ops<double>::nonlinear(P, v3, bouss ? vin[3] : nullptr, N, 0, nc));
    const double rmp = 1 / (double)o;
    {
        UpdateArgs a{};
        for (int i = 0; i < nc; i++) {
            a.n[i] = (const double2 *)N[i];
            a.v[i] = (const double2 *)vin[i];
            a.c[i] = (const double2 *)cold[i];
            a.out[i] = (double2 *)vout[i];
        }
        a.adt = sp.dt * rmp;
        a.anu = a.adt * sp.nu;
        a.akappa = a.adt * sp.kappa;
        a.xmom = sp.xmom;
        a.xtemp = sp.xtemp;
        for (int i = 0; i < 3; i++) a.om[i] = sp.omega[i];
        a.nc = nc;
        a.rot = rot;
        Launch L(P, "stage_update", 4.0 * nc * field);
        chain(k_stage_update, elem_blocks(P), 256, 0, P.stream, P.geo, a);
    }
    // wall round trips of vx, vy (no slip) and theta (zero walls): rows above nzp are rebuilt by the
    // continuation
    double2 *x = (double2 *)vout[0], *y = (double2 *)vout[1], *w = (double2 *)vout[2], *th = (double2 *)vout[3];
    void *trip[3] = {x, y, th};
    const int nt = bouss ? 3 : 2;
    auto done = [](int st) {
        if (st != kNoFast) return st;
        set_error("no memory for the digit tables (FP64 stage)");
        return (int)ERR_OOM;
    };
    auto inverse = [&](void *const in[], void *const out[], const void *const add[], int n) {
        ZInvArgs z{};
        for (int i = 0; i < n; i++) {
            z.in[i] = in[i];
            z.out0[i] = out[i];
            z.add[i] = add ? add[i] : nullptr;
        }
        z.nrows = z.scale_rows = P.nzp;
        z.scale = 1.0 / (double)P.nz;
        return done(tc_z_inverse(P, z, n, n * (field + mixed)));
    };
    auto forward = [&](void *const f[], int n) {
        ZFwdArgs z{};
        for (int i = 0; i < n; i++) {
            z.in[i] = f[i];
            z.out[i] = f[i];
        }
        z.in_scale = 1.0;
        return done(tc_z_forward(P, z, n, n * (field + mixed)));
    };
    SG_TRY(inverse(trip, trip, nullptr, nt));
    double tmp = rmp;
    if (o != sp.ord) tmp = (double)(o + 1) * tmp;
    {
        const WallVel vb{sp.vzsta[0], sp.vzsta[1], sp.vzend[0], sp.vzend[1]};
        Launch L(P, "walls", 8.0 * P.ny * P.nxh * 16.0);
        chain(k_stage_walls, dim3(cdiv(P.nxh, 64), P.ny), 64, 0, P.stream, P.geo, x, y, bouss ? th : nullptr, (const double2 *)pr, tmp, vb);
    }
    SG_TRY(forward(trip, nt));
    const bool trip2 = bouss && !rot;
    SG_TRY(f64_poisson(P, x, y, w, d, trip2 ? th : nullptr, coef));
    SG_TRY(f64_profile(P, coef, pr, nullptr));
    {
        void *in[2] = {d, th}, *out[2] = {pr, th};
        const void *add[2] = {pr, nullptr};
        SG_TRY(inverse(in, out, add, trip2 ? 2 : 1));
    }
    {
        Launch L(P, "stage_correct", 8.0 * field);
        chain(k_stage_correct, elem_blocks(P), 256, 0, P.stream, P.geo, x, y, w, (const double2 *)E[0], (const double2 *)E[1], coef);
    }
    if (trip2) {
        {
            Launch L(P, "theta_herm", 4.0 * P.ny * P.nzp * 16.0);
            chain(k_stage_herm, dim3(cdiv((P.ny / 2 + 1) * P.nzp, 128), 2), 128, 0, P.stream, P.geo, th);
        }
        void *f[1] = {th};
        SG_TRY(forward(f, 1));
    }
    return check_launch("FP64 stage");
}

}  // namespace sg
