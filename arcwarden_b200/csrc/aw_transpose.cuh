// aw_transpose.cuh — the adjoints' transposed solves, one k-space mode at a time
// (included inside an anonymous namespace by the sources that apply them).
#ifndef AW_KSPACE_MODES
#define AW_KSPACE_MODES
// wavenumbers of R2C mode (i, j) and the Nyquist test, as the forward solves take them
__device__ __forceinline__ double kx_of(int i, double dkx) { return i * dkx; }
__device__ __forceinline__ double ky_of(int j, int ny, double dky) { return ((j <= ny / 2) ? j : j - ny) * dky; }
__device__ __forceinline__ bool nyquist(int i, int j, int nx, int ny) {
    return ((nx % 2 == 0) && i == nx / 2) || ((ny % 2 == 0) && j == ny / 2);
}
#endif
// k-space transposes: the conjugates of the forward multipliers, with the 1/N scale.
// lE (3) -> ldcu (3), lamu (4): E_T = -gT P (dcu - i S(amu)).
__device__ __forceinline__ void et_T_k(int i, int j, const SpecGeo& g, double eps0, double c, double n0,
                                       const cufftComplex (&L)[3], cufftComplex (&out)[7]) {
    const double kx = kx_of(i, g.dkx), ky = ky_of(j, g.ny, g.dky);
    const double k2 = kx * kx + ky * ky;
    cufftComplex z; z.x = z.y = 0.0f;
    if (nyquist(i, j, g.nx, g.ny) || k2 == 0.0) {
        for (int f = 0; f < 7; ++f) out[f] = z;
        return;
    }
    const double G = -1.0 / (eps0 * c * c * k2 + n0) * (g.ff ? g.ff[j * g.nkx + i] : 1.0);
    double pr[3], pi[3];
    for (int d = 0; d < 3; ++d) { pr[d] = G * L[d].x; pi[d] = G * L[d].y; }
    const double kdr = (kx * pr[0] + ky * pr[1]) / k2, kdi = (kx * pi[0] + ky * pi[1]) / k2;
    pr[0] -= kx * kdr; pi[0] -= kx * kdi;
    pr[1] -= ky * kdr; pi[1] -= ky * kdi;
    for (int d = 0; d < 3; ++d) {
        cufftComplex o; o.x = static_cast<float>(pr[d]) * g.invN; o.y = static_cast<float>(pi[d]) * g.invN;
        out[d] = o;
    }
    // lamu = conj(-i) S^T PL = i S^T PL: i (re + i im) = -im + i re
    const double w0r = -pi[0], w0i = pr[0], w1r = -pi[1], w1i = pr[1], w2r = -pi[2], w2i = pr[2];
    const double ar[4] = {kx * w0r - ky * w1r, ky * w0r + kx * w1r, kx * w2r, ky * w2r};
    const double ai[4] = {kx * w0i - ky * w1i, ky * w0i + kx * w1i, kx * w2i, ky * w2i};
    for (int m = 0; m < 4; ++m) {
        cufftComplex o; o.x = static_cast<float>(ar[m]) * g.invN; o.y = static_cast<float>(ai[m]) * g.invN;
        out[3 + m] = o;
    }
}
// (lE_L x y, lB x y z) -> (lrho, lJx, lJy, lJz): the transpose of k_kspace_elb.
__device__ __forceinline__ void elb_T_k(int i, int j, const SpecGeo& g, double eps0, double c, const cufftComplex (&L)[5],
                                        cufftComplex (&out)[4]) {
    const double kx = kx_of(i, g.dkx), ky = ky_of(j, g.ny, g.dky);
    const double k2 = kx * kx + ky * ky;
    cufftComplex z; z.x = z.y = 0.0f;
    if (nyquist(i, j, g.nx, g.ny) || k2 == 0.0) {
        for (int f = 0; f < 4; ++f) out[f] = z;
        return;
    }
    const double ff = g.ff ? g.ff[j * g.nkx + i] : 1.0;
    const double gE = ff / (eps0 * k2), gB = ff / (eps0 * c * c * k2);
    const cufftComplex lx = L[0], ly = L[1], bx = L[2], by = L[3], bz = L[4];
    // forward: ELx = -i kx gE rho, ELy = -i ky gE rho; Bx = i gB ky Jz, By = -i gB kx Jz,
    // Bz = i gB (kx Jy - ky Jx). transpose: conj of each factor, i.e. i <-> -i.
    // (re + i im) * i f = -f im + i f re; (re + i im) * (-i f) = f im - i f re
    // lrho <- conj(-i kx gE) lEx + conj(-i ky gE) lEy = gE (i kx lEx + i ky lEy)
    const double rr = -gE * (kx * lx.y + ky * ly.y), ri = gE * (kx * lx.x + ky * ly.x);
    double Jxr, Jxi, Jyr, Jyi, Jzr, Jzi;
    // Jx <- conj(-i gB ky) bz = (i gB ky) bz = gB ky (-bz.y + i bz.x)
    Jxr = -gB * ky * bz.y; Jxi = gB * ky * bz.x;
    // Jy <- conj(i gB kx) bz = (-i gB kx) bz = gB kx (bz.y - i bz.x)
    Jyr = gB * kx * bz.y; Jyi = -gB * kx * bz.x;
    // Jz <- conj(i gB ky) bx + conj(-i gB kx) by = gB ky (bx.y - i bx.x) + gB kx (-by.y + i by.x)
    Jzr = gB * ky * bx.y - gB * kx * by.y; Jzi = -gB * ky * bx.x + gB * kx * by.x;
    cufftComplex o;
    o.x = static_cast<float>(rr) * g.invN; o.y = static_cast<float>(ri) * g.invN; out[0] = o;
    o.x = static_cast<float>(Jxr) * g.invN; o.y = static_cast<float>(Jxi) * g.invN; out[1] = o;
    o.x = static_cast<float>(Jyr) * g.invN; o.y = static_cast<float>(Jyi) * g.invN; out[2] = o;
    o.x = static_cast<float>(Jzr) * g.invN; o.y = static_cast<float>(Jzi) * g.invN; out[3] = o;
}
// (lEx, lEy) -> lrho: lrho_k = sum_d conj(K_d) lE_d,k with K_d = -i k_d / (eps0 k^2)
// (times 1/N for the unnormalised inverse), zero at k = 0 and on the Nyquist lines
// like the forward solve.
__device__ __forceinline__ void es_T_k(int i, int j, const SpecGeo& g, double eps0, const cufftComplex (&L)[2],
                                       cufftComplex& r) {
    const double kx = kx_of(i, g.dkx), ky = ky_of(j, g.ny, g.dky);
    const double k2 = kx * kx + ky * ky;
    r.x = r.y = 0.0f;
    if (k2 > 0.0 && !nyquist(i, j, g.nx, g.ny)) {
        const double gr = 1.0 / (eps0 * k2) * static_cast<double>(g.invN) * (g.ff ? g.ff[j * g.nkx + i] : 1.0);
        const double zx = kx * L[0].x + ky * L[1].x, zy = kx * L[0].y + ky * L[1].y;   // k . lE
        r.x = static_cast<float>(-zy * gr);                                            // i z
        r.y = static_cast<float>(zx * gr);
    }
}
