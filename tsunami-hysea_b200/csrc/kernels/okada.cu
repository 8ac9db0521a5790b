// Okada seafloor deformation on the GPU, in FP64 (the dislocation formulas
// cancel strongly near the fault; FP32 would lose centimetres of uplift).
//
// Per cell (src/GPU/Deformacion.cu:55-116): station coordinates on the
// lon/lat lattice lon0 + i*dlon, lat0 + j*dlat; Gauss-Krueger projection
// about the fault centre (src/GPU/prtoxy.cu:33-54); rotation by the strike;
// vertical surface displacement of a rectangular dislocation (Okada 1985,
// BSSA 75(4), closed-form surface solution, which the reference's DC3D of
// Okada 1992 equals at z = 0) divided by the depth scale.  Then optional
// relative / absolute cropping and the update bathymetry -= U_Z,
// eta_initial += U_Z (src/GPU/Deformacion.cu:13-53,118-143); the water depth
// h is unchanged, so the surface rises by U_Z.
//
// What bounds it: FP64 instructions.  A cell takes 4 corners of the dislocation
// with 2 logarithms and 2 arc tangents each in the closed form.  For the
// reference's double state (thy_apply_okada) the corners' sum is evaluated as
// one logarithm of each kind (of the ratio of the corners' arguments), one atan2
// (of the product of the corners' complex numbers, with its turns counted) and
// one division for all the fractions; the sines of the fault's angles come from
// the host and those of a row are shared by a thread's cells.  2048^2 cells on a
// B200: 3041 -> 1134 instructions a cell (1227 -> 549 of them FP64), 550 -> 192 us;
// the FP64 pipe is busy 65 % of that.  The kernel that computes the deformation
// applies it; relative cropping, which needs the largest one first, computes it
// twice where the caller brings no scratch, which is less than an allocation costs
// (0.4 to 1.3 ms).  Calls of thy_apply_okada, 2048^2: 1.9 -> 0.24 ms, with
// relative cropping 0.42 ms; 256^2 0.67 -> 0.06 ms.  R + E, R + X and R + dt, which
// cancel beside a fault's lines, are formed as quotients (22 instructions a corner,
// 0.03 ms a pass): the error against extended precision over 4 million points of
// random faults is 1e-16 to 1e-15 of the slip (rms), 5e-14 to 3e-13 corner by
// corner.
// Scenarios keep the corners' own closed form: their fields are single precision,
// and the arrival time is a threshold on them, so that last bits of the double
// which round the other way move it in a few cells.
#include <algorithm>
#include <cmath>

#include "device.cuh"
#include "kernels.h"

namespace thy {

__device__ void gauss_krueger(double lat, double lon, double lat0, double lon0, double &x, double &y)
{
    // reference constants: Bessel-type ellipsoid a = 6378.16 km, e^2 = 0.0066946053,
    // e'^2 = 0.0067397251, a(1-e^2) = 6335.4607362597517 km, 57.29578 deg/rad,
    // 6 * 57.29578^2 and pi/180 rounded to single precision
    const double deg = 0.017453292371619689;
    const double rlat = lat * deg, slat = sin(rlat), clat = cos(rlat);
    const double v2 = clat * 0.0067397251 * clat + 1.0;
    const double dl = lon - lon0;
    const double ph1 = lat + v2 * 0.5 * dl * dl * slat * clat * deg;
    const double s1 = sin(ph1 * deg), s2 = sin((ph1 + lat0) * 0.5 * deg);
    const double d = sqrt(1.0 - s2 * 0.0066946053 * s2);
    const double rm = 6335.4607362597517 / (d * (d * d));
    const double rn = 6378.16 / sqrt(1.0 - s1 * 0.0066946053 * s1);
    y = (ph1 - lat0) / (57.29578 / rm);
    x = dl * clat / (57.29578 / rn) * (dl * dl * cos(rlat * 2.0) / 19696.838434850401 + 1.0);
}

// u_z at the surface; x along strike, y across (km), d centroid depth (km),
// fault length L and width W (km) centred on the reference point, U1
// strike-slip and U2 dip-slip (m).  mu/(lambda+mu) = 1/2 (alpha = 2/3).
__device__ double okada_closed(double x, double y, double d, double dip_deg, double L, double W, double U1, double U2)
{
    const double two_pi = 6.283185307179586, eps = 1e-6, k = 0.5;
    double sd = sin(dip_deg * (two_pi / 360.0)), cd = cos(dip_deg * (two_pi / 360.0));
    if (fabs(cd) < eps) { cd = 0.0; sd = (sd > 0.0) ? 1.0 : -1.0; }
    double xi[2] = {x + 0.5 * L, x - 0.5 * L};
    if (fabs(xi[0]) < eps) xi[0] = 0.0;
    if (fabs(xi[1]) < eps) xi[1] = 0.0;
    const double p = y * cd + d * sd;
    double q = y * sd - d * cd;
    double et[2] = {p + 0.5 * W, p - 0.5 * W};
    if (fabs(q) < eps) q = 0.0;
    if (fabs(et[0]) < eps) et[0] = 0.0;
    if (fabs(et[1]) < eps) et[1] = 0.0;
    if ((q == 0.0) && ((xi[0] * xi[1] <= 0.0 && et[0] * et[1] == 0.0) || (et[0] * et[1] <= 0.0 && xi[0] * xi[1] == 0.0)))
        return 0.0;
    int kxi[2] = {0, 0}, ket[2] = {0, 0};
    {
        const double r12 = sqrt(xi[0] * xi[0] + et[1] * et[1] + q * q);
        const double r21 = sqrt(xi[1] * xi[1] + et[0] * et[0] + q * q);
        const double r22 = sqrt(xi[1] * xi[1] + et[1] * et[1] + q * q);
        if (xi[0] < 0.0 && r21 + xi[1] < eps) kxi[0] = 1;
        if (xi[0] < 0.0 && r22 + xi[1] < eps) kxi[1] = 1;
        if (et[0] < 0.0 && r12 + et[1] < eps) ket[0] = 1;
        if (et[0] < 0.0 && r22 + et[1] < eps) ket[1] = 1;
    }
    double uz = 0.0;
#pragma unroll
    for (int kk = 0; kk < 2; kk++) {
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const double sgn = (j + kk == 1) ? -1.0 : 1.0;
            const double X = xi[j], E = et[kk];
            const double R = sqrt(X * X + E * E + q * q);
            if (R == 0.0) continue;
            const double dt = E * sd - q * cd;
            const double theta = (q == 0.0) ? 0.0 : atan(X * E / (q * R));
            const double inv_rx = kxi[kk] ? 0.0 : 1.0 / (R + X);
            double inv_re, ln_re;
            if (ket[j]) { inv_re = 0.0; ln_re = -log(R - E); }
            else { inv_re = 1.0 / (R + E); ln_re = log(R + E); }
            double I4, I5;
            if (cd != 0.0) {
                const double Xs = sqrt(X * X + q * q);
                I4 = k / cd * (log(R + dt) - sd * ln_re);
                I5 = (X == 0.0) ? 0.0 : k * 2.0 / cd * atan((E * (Xs + q * cd) + Xs * (R + Xs) * sd) / (X * (R + Xs) * cd));
            } else {
                I4 = -k * q / (R + dt);
                I5 = -k * X * sd / (R + dt);
            }
            const double fss = dt * q / R * inv_re + q * sd * inv_re + I4 * sd;
            const double fds = dt * q / R * inv_rx + sd * theta - I5 * sd * cd;
            uz += sgn * (-U1 / two_pi * fss - U2 / two_pi * fds);
        }
    }
    return uz;
}

__global__ void okada_kernel(int nx, int ny, double *__restrict__ def, double lon0, double dlon, double lat0, double dlat,
                             OkadaFault f, double Hs)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= nx || y >= ny) return;
    const double rad = M_PI / 180.0;
    const double lon = lon0 + x * dlon, lat = lat0 + y * dlat;
    const double ss = sin(rad * f.strike), cs = cos(rad * f.strike);
    double xp, yp;
    gauss_krueger(lat, lon, f.lat_c, f.lon_c, xp, yp);
    const double uz = okada_closed(xp * ss + yp * cs, -xp * cs + yp * ss, f.depth_c, f.dip, f.length, f.width,
                               f.slip * cos(rad * f.rake), f.slip * sin(rad * f.rake));
    def[(size_t)y * nx + x] = uz / Hs;
}

void launch_okada(const ScenarioDev *s_host, double *def, double lon0, double dlon, double lat0, double dlat,
                  const OkadaFault &f, double Hs, cudaStream_t st)
{
    dim3 block(32, 4);
    dim3 grid((s_host->nx + 31) / 32, (s_host->ny + 3) / 4);
    okada_kernel<<<grid, block, 0, st>>>(s_host->nx, s_host->ny, def, lon0, dlon, lat0, dlat, f, Hs);
}

// max over cells of (float)|U_Z| as float bits (non-negative floats order as unsigned)
__global__ void absmax_kernel(const double *__restrict__ def, long long n, unsigned int *max_bits)
{
    float m = 0.f;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        m = fmaxf(m, (float)fabs(def[i]));
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    __shared__ float red[8];
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < (int)(blockDim.x >> 5); k++) m = fmaxf(m, red[k]);
        atomicMax(max_bits, __float_as_uint(m));
    }
}

void launch_absmax(const double *def, long long n, unsigned int *max_bits, cudaStream_t st)
{
    cudaMemsetAsync(max_bits, 0, sizeof(unsigned int), st);
    absmax_kernel<<<296, 256, 0, st>>>(def, n, max_bits);
}

__global__ void apply_deformation_kernel(ScenarioDev s, const double *__restrict__ def, int crop_flag, double crop_value,
                                         const unsigned int *__restrict__ max_bits)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x >= s.nx || y >= s.ny) return;
    double U = def[(size_t)y * s.nx + x];
    if (crop_flag == 1) {
        const double thr = crop_value * (double)__uint_as_float(*max_bits);
        if (fabs(U) < thr) U = 0.0;
    } else if (crop_flag == 2) {
        if (fabs(U) < crop_value) U = 0.0;
    }
    const int p = s.ctl->parity;
    const size_t idx = (size_t)y * s.pitch + x;
    const float eta = s.eta[p][idx], dep = s.dep[idx];
    const double h = (double)eta + (double)dep;   // exact in double
    const float dep_n = (float)((double)dep - U);
    // eta and the depth are rounded independently: deriving eta from the
    // rounded depth would quantise the surface to an ulp of the depth
    // (0.24 mm at 4 km); h absorbs that rounding instead (6e-8 relative)
    float eta_n = (float)((double)eta + U);
    if (h == 0.0 || !((double)eta_n + (double)dep_n > 0.0)) eta_n = -dep_n;   // dry stays dry, exactly
    s.dep[idx] = dep_n;
    s.eta[p][idx] = eta_n;
    s.eta_ini[idx] = (float)((double)s.eta_ini[idx] + U);
}

void launch_apply_deformation(const ScenarioDev *s_host, const double *def, int crop_flag, double crop_value,
                              const unsigned int *max_bits, cudaStream_t st)
{
    dim3 grid((s_host->nx + 255) / 256, s_host->ny);
    apply_deformation_kernel<<<grid, 256, 0, st>>>(*s_host, def, crop_flag, crop_value, max_bits);
}

// ---- the reference's double state ----
namespace {

// what the cells of a fault share
struct OkadaConst {
    double lon0, dlon, lat0, dlat;     // the lattice
    double lon_c, lat_c, d;            // reference point, its depth (km)
    double ss, cs, sd, cd, kcd;        // sine and cosine of strike and dip, k / cd
    double hl, hw, u1, u2;             // half length and width (km), slips over -2 pi (m)
    double inv_scale;                  // 1 / depth scale
    OkadaFault f;                      // for the points left to okada_closed
};

// The projection with a row's shares of it taken once.
struct OkadaRow {
    double lat, a, b, e;
};

constexpr double kDeg = 0.017453292371619689;

__device__ inline OkadaRow okada_row(const OkadaConst &c, int y)
{
    OkadaRow r;
    r.lat = c.lat0 + y * c.dlat;
    double s, co;
    sincos(r.lat * kDeg, &s, &co);
    const double v2 = co * 0.0067397251 * co + 1.0;
    r.a = v2 * 0.5 * s * co * kDeg;
    r.b = co * (6378.16 / 57.29578);
    r.e = cos(r.lat * kDeg * 2.0) / 19696.838434850401;
    return r;
}

__device__ inline void gauss_krueger(const OkadaConst &c, const OkadaRow &r, int x, double &px, double &py)
{
    const double dl = c.lon0 + x * c.dlon - c.lon_c, dl2 = dl * dl;
    const double ph1 = r.lat + r.a * dl2;
    const double s1 = sin(ph1 * kDeg), s2 = sin((ph1 + c.lat_c) * 0.5 * kDeg);
    const double im = rsqrt(1.0 - s2 * 0.0066946053 * s2), in = rsqrt(1.0 - s1 * 0.0066946053 * s1);
    py = (ph1 - c.lat_c) * (6335.4607362597517 / 57.29578) * (im * (im * im));
    px = dl * r.b * in * (dl2 * r.e + 1.0);
}

// (re, im) *= (w, s), w > 0: the argument grows by less than a quarter turn
// either way; turns counts its passes of the negative real axis
__device__ inline void turn(double &re, double &im, int &turns, double w, double s)
{
    const double r = re * w - im * s, i = re * s + im * w;
    turns += (im >= 0.0 && s > 0.0 && i < 0.0) ? 1 : 0;
    turns -= (im < 0.0 && s < 0.0 && i >= 0.0) ? 1 : 0;
    re = r;
    im = i;
}

// The same for the other points: no corner coordinate, q or cd vanishes.  The
// corners' sum with its logarithms, arc tangents and divisions taken together.
__device__ inline double okada_uz(const OkadaConst &c, double x, double y)
{
    const double eps = 1e-6;
    const double xi[2] = {x + c.hl, x - c.hl};
    const double p = y * c.cd + c.d * c.sd, q = y * c.sd - c.d * c.cd;
    const double et[2] = {p + c.hw, p - c.hw};
    const double qq = q * q, aq = fabs(q), qc = q * c.cd;
    bool regular = aq >= eps && c.cd != 0.0;
    double n4[4], n5[4], D[4], S[4], A[4], Ss[4], As[4];   // by corner: kk * 2 + j
    double re = 1.0, im = 0.0;
    int turns = 0;
#pragma unroll
    for (int j = 0; j < 2; j++) {
        const double X = xi[j], X2q = X * X + qq, Xs = sqrt(X2q), aX = fabs(X) * fabs(c.cd);
        const bool neg = (X < 0.0) != (c.cd < 0.0);
        regular = regular && fabs(X) >= eps;
#pragma unroll
        for (int kk = 0; kk < 2; kk++) {
            const int k = 2 * kk + j;
            const double E = et[kk], R = sqrt(X2q + E * E);
            const double dt = E * c.sd - qc, o = E * c.cd + q * c.sd;
            // R + E, R + X and R + dt as quotients p / s without cancellation
            const double ap = E < 0.0 ? X2q : R + E, as = E < 0.0 ? R - E : 1.0;
            const double bp = X < 0.0 ? E * E + qq : R + X, bs = X < 0.0 ? R - X : 1.0;
            const double tp = dt < 0.0 ? X * X + o * o : R + dt, ts = dt < 0.0 ? R - dt : 1.0;
            // (a corner that the general formula takes apart)
            regular = regular && ap >= eps * as && bp >= eps * bs && tp > 0.0 && fabs(E) >= eps;
            A[k] = ap;
            As[k] = as;
            S[k] = tp;
            Ss[k] = ts;
            D[k] = R * ap * bp;
            n4[k] = bp * (c.sd * ap - qc * as);
            n5[k] = ap * bs * dt;
            // theta = atan(X E / (q R)) and the arc tangent of I5, each as the
            // argument of a number with a positive real part; the corner's sign
            // and the minus of I5 are conjugations
            const double g = R + Xs;
            const double w1 = aq * R, v1 = X * E, w2 = aX * g, v2 = E * (Xs + qc) + Xs * g * c.sd;
            const bool minus = j + kk == 1;
            const double s1 = ((q < 0.0) != minus) ? -v1 : v1, s2 = (neg != minus) ? v2 : -v2;
            turn(re, im, turns, w1, s1);
            turn(re, im, turns, w2, s2);
        }
    }
    // one division for the corners' fractions and the two ratios
    const double D01 = D[0] * D[1], D23 = D[2] * D[3], da = A[1] * A[2] * (As[0] * As[3]),
                 ds = S[1] * S[2] * (Ss[0] * Ss[3]);
    const double dd = D01 * D23, dr = da * ds;
    const double inv = 1.0 / (dd * dr), id = inv * dr, ir = inv * dd;
    const double i01 = id * D23, i23 = id * D01;
    const double w0 = i01 * D[1], w1 = i01 * D[0], w2 = i23 * D[3], w3 = i23 * D[2];
    const double f4 = n4[0] * w0 - n4[1] * w1 - n4[2] * w2 + n4[3] * w3;
    const double f5 = n5[0] * w0 - n5[1] * w1 - n5[2] * w2 + n5[3] * w3;
    const double ls = log(S[0] * S[3] * (Ss[1] * Ss[2]) * (ir * da)), la = log(A[0] * A[3] * (As[1] * As[2]) * (ir * ds));
    const double angle = atan2(im, re) + 6.283185307179586 * turns;
    const double uz = c.u1 * (q * f4 + c.sd * c.kcd * (ls - c.sd * la)) + c.u2 * (q * f5 + c.sd * angle);
    if (regular && fabs(uz) <= 1e300) return uz;
    const double two_pi = 6.283185307179586;
    return okada_closed(x, y, c.d, c.f.dip, c.f.length, c.f.width, -c.u1 * two_pi, -c.u2 * two_pi);
}

OkadaConst okada_const(double lon0, double dlon, double lat0, double dlat, const OkadaFault &f, double Hs)
{
    const double rad = M_PI / 180.0, two_pi = 6.283185307179586, k = 0.5;   // k = mu / (lambda + mu)
    OkadaConst c;
    c.lon0 = lon0;
    c.dlon = dlon;
    c.lat0 = lat0;
    c.dlat = dlat;
    c.lon_c = f.lon_c;
    c.lat_c = f.lat_c;
    c.d = f.depth_c;
    c.ss = std::sin(rad * f.strike);
    c.cs = std::cos(rad * f.strike);
    c.sd = std::sin(f.dip * (two_pi / 360.0));
    c.cd = std::cos(f.dip * (two_pi / 360.0));
    if (std::fabs(c.cd) < 1e-6) c.cd = 0.0;   // (vertical: the general formula)
    c.kcd = k / c.cd;
    c.hl = 0.5 * f.length;
    c.hw = 0.5 * f.width;
    c.u1 = f.slip * std::cos(rad * f.rake) / -two_pi;
    c.u2 = f.slip * std::sin(rad * f.rake) / -two_pi;
    c.inv_scale = 1.0 / Hs;
    c.f = f;
    return c;
}

// the reference's device state, double2 (h, H) per cell
struct ReferenceState {
    double *state, *eta_initial;
    __device__ __forceinline__ void operator()(size_t i, double U) const
    {
        state[2 * i + 1] -= U;
        if (eta_initial) eta_initial[i] += U;
    }
};

// the cropping of U_Z (src/GPU/Deformacion.cu:13-36)
struct OkadaCrop {
    int flag;
    double value;
    const unsigned int *max_bits;   // flag 1: the largest (float)|U_Z|, as float bits
    __device__ __forceinline__ double limit() const
    {
        return flag == 1 ? value * (double)__uint_as_float(*max_bits) : flag == 2 ? value : 0.0;
    }
    static __device__ __forceinline__ double apply(double U, double limit) { return fabs(U) < limit ? 0.0 : U; }
};

// A block takes `per` x kOkadaThreads cells of a row (OkadaSplit).  max_bits given: only the
// largest (float)|U_Z| (non-negative floats order as unsigned) and, with def
// given, U_Z itself; else U_Z is applied.  One kernel for all of them: a cell's
// U_Z is the same bits in each.
__global__ void __launch_bounds__(kOkadaThreads, 5) okada_reference_kernel(unsigned nx, OkadaSplit split, OkadaConst c, ReferenceState out,
                                                                           OkadaCrop crop, unsigned int *max_bits,
                                                                           double *__restrict__ def)
{
    const unsigned y = blockIdx.x / split.segs, x0 = okada_first_cell(split, blockIdx.x - y * split.segs) + threadIdx.x;
    const OkadaRow row = okada_row(c, (int)y);
    const double limit = max_bits ? 0.0 : crop.limit();
    float m = 0.f;
#pragma unroll 1
    for (unsigned k = 0, x = x0; k < split.per && x < nx; k++, x += kOkadaThreads) {
        double px, py;
        gauss_krueger(c, row, (int)x, px, py);
        const double U = okada_uz(c, px * c.ss + py * c.cs, -px * c.cs + py * c.ss) * c.inv_scale;
        const size_t i = (size_t)y * nx + x;
        if (max_bits) {
            m = fmaxf(m, (float)fabs(U));
            if (def) def[i] = U;
        } else {
            out(i, OkadaCrop::apply(U, limit));
        }
    }
    if (max_bits) {
        const unsigned int v = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
        if ((threadIdx.x & 31) == 0 && v > *(volatile unsigned int *)max_bits) atomicMax(max_bits, v);
    }
}

// applies the U_Z of a scratch field
__global__ void apply_reference_kernel(size_t n, const double *__restrict__ def, ReferenceState out, OkadaCrop crop)
{
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i < n) out(i, OkadaCrop::apply(def[i], crop.limit()));
}

}  // namespace

void launch_okada_reference(int nx, int ny, int sms, double lon0, double dlon, double lat0, double dlat, const OkadaFault &f,
                            double Hs, int crop_flag, double crop_value, double *state, double *eta_initial,
                            unsigned int *max_bits, double *def, cudaStream_t st)
{
    const OkadaConst c = okada_const(lon0, dlon, lat0, dlat, f, Hs);
    const ReferenceState out{state, eta_initial};
    const OkadaCrop crop{crop_flag, crop_value, max_bits};
    const long long n = (long long)nx * ny;
    const OkadaSplit split = okada_split(nx, ny, sms);
    const unsigned blocks = split.segs * (unsigned)ny;
    if (crop_flag == 1) {
        cudaMemsetAsync(max_bits, 0, sizeof(unsigned int), st);
        okada_reference_kernel<<<blocks, kOkadaThreads, 0, st>>>(nx, split, c, out, crop, max_bits, def);
        if (def) {
            apply_reference_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>((size_t)n, def, out, crop);
            return;
        }
    }
    okada_reference_kernel<<<blocks, kOkadaThreads, 0, st>>>(nx, split, c, out, crop, nullptr, nullptr);
}

cudaError_t preload_okada_kernels()
{
    cudaFuncAttributes a;
    cudaError_t e;
    if ((e = cudaFuncGetAttributes(&a, okada_kernel)) || (e = cudaFuncGetAttributes(&a, absmax_kernel)) ||
        (e = cudaFuncGetAttributes(&a, apply_deformation_kernel)))
        return e;
    return cudaSuccess;
}

}  // namespace thy
