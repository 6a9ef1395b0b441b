// CPU check of the filtered pixel rule (xpulse_recon_b200/csrc/xpr_pixel.cuh): for voxels of
// random bricks of given projections, the kernel's window coordinates (their single-precision
// operations restated, the reciprocal off by up to its documented error either way) must give
// the contract's pixel wherever their fraction does not call for the contract itself.
// usage: check W H P ex ey ez row_off rows voxel ox oy oz strict bricks < P records of 20 floats
// prints: bricks, pairs, pairs decided by the filter, wrong ones, chunks of 8 x 32 voxels
// (lanes across x) with at least one close voxel, largest E
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "xpr_pixel.cuh"

using namespace xpr;

struct Rec { float m[20]; };

static float pos(int i, float vx, float o, bool strict)
{
    if (strict) { const volatile float t = (float)i * vx; return t + o; }
    return fmaf((float)i, vx, o);
}
static float num(const float *c, float x, float y, float z)
{
    volatile float a = c[0] * x, b = c[1] * y, s = a + b, t = c[2] * z;
    s = s + t;
    return s + c[3];
}
static float colf(const float *c, float x, float z)
{
    volatile float t = c[2] * z;
    return fmaf(c[0], x, c[3]) + t;
}
// floor(y) by the kernel's two steps
static long fl(float y) { return (long)std::floor((double)y); }

static void contract(const Rec &q, float x, float y, float z, float off, bool strict, double &iu, double &iv)
{
    const float *cu = q.m, *cv = q.m + 4, *cw = q.m + 12;
    if (strict) {
        const volatile float u = num(cu, x, y, z) / num(cw, x, y, z), v = num(cv, x, y, z) / num(cw, x, y, z);
        const volatile float t = v - off;
        iu = roundf(u);
        iv = roundf(t);
    } else {
        const volatile float rw = 1.0f / fmaf(cw[1], y, colf(cw, x, z));
        const volatile float a = cu[1] * rw, b = cv[1] * rw;
        iu = std::floor((double)fmaf(y, a, fmaf(colf(cu, x, z), rw, 0.5f)));
        iv = std::floor((double)fmaf(y, b, fmaf(colf(cv, x, z), rw, 0.5f - off)));
    }
}

int main(int argc, char **argv)
{
    if (argc < 15) return 2;
    const int W = atoi(argv[1]), H = atoi(argv[2]), P = atoi(argv[3]), ex = atoi(argv[4]), ey = atoi(argv[5]),
              ez = atoi(argv[6]), off = atoi(argv[7]), rows = atoi(argv[8]);
    const float vx = (float)atof(argv[9]), o[3] = {(float)atof(argv[10]), (float)atof(argv[11]), (float)atof(argv[12])};
    const bool strict = atoi(argv[13]) != 0;
    const int bricks = atoi(argv[14]);
    std::vector<Rec> rec(P);
    for (auto &r : rec)
        for (float &x : r.m)
            if (scanf("%f", &x) != 1) return 2;
    srand(12345);
    long used = 0, pairs = 0, decided = 0, wrong = 0, chunks = 0, close_chunks = 0, maxE = 0;
    for (int n = 0; n < bricks; ++n) {
        const Rec &q = rec[rand() % P];
        const float *cu = q.m, *cv = q.m + 4, *cw = q.m + 12;
        PixBrick k;
        const int nx = (W + ex - 1) / ex, ny = (H + ey - 1) / ey, nz = (W + ez - 1) / ez;
        const int at[3] = {rand() % nx * ex, rand() % ny * ey, rand() % nz * ez}, ext[3] = {ex, ey, ez};
        for (int i = 0; i < 3; ++i) {
            k.vox[i] = vx;
            k.org[i] = o[i];
            k.idx0[i] = at[i];
            k.ext[i] = ext[i];
        }
        k.row_off = (float)off;
        double um = 1e30, uM = -1e30, vm = 1e30, vM = -1e30, wm = 1e30, wM = -1e30, n0[3] = {0, 0, 0};
        for (int c = 0; c < 8; ++c) {
            const double X = (double)(at[0] + ((c & 1) ? ex - 1 : 0)) * vx + o[0],
                         Y = (double)(at[1] + ((c & 2) ? ey - 1 : 0)) * vx + o[1],
                         Z = (double)(at[2] + ((c & 4) ? ez - 1 : 0)) * vx + o[2];
            const double a = cu[0] * X + cu[1] * Y + cu[2] * Z + cu[3], b = cv[0] * X + cv[1] * Y + cv[2] * Z + cv[3],
                         w = cw[0] * X + cw[1] * Y + cw[2] * Z + cw[3];
            if (c == 0) { n0[0] = a; n0[1] = b; n0[2] = w; }
            um = fmin(um, a / w); uM = fmax(uM, a / w);
            vm = fmin(vm, b / w - off); vM = fmax(vM, b / w - off);
            wm = fmin(wm, w); wM = fmax(wM, w);
        }
        if (wm <= 0) continue;
        k.wmin = (float)wm * 0.99999f;
        k.wmax = (float)wM * 1.00001f;
        const float *vp = q.m + 16;
        k.l = std::max((int)ceilf(vp[0]), std::max(0, (int)floor(um) - 2));
        k.r = std::min((int)ceilf(vp[1]), std::min(W, (int)ceil(uM) + 3));
        k.b = std::max((int)ceilf(vp[2]), std::max(0, (int)floor(vm) - 2));
        k.t = std::min((int)ceilf(vp[3]), std::min(rows, (int)ceil(vM) + 3));
        if (k.r <= k.l || k.t <= k.b) continue;
        const PixRow ru = pix_row(cu, cw, n0[0], n0[2], k.l, k.vox), rv = pix_row(cv, cw, n0[1], n0[2], k.b + off, k.vox),
                     rw = pix_row(cw, cw, n0[2], n0[2], 0.0, k.vox);
        const int E = pix_bound(cu, cv, cw, ru, rv, rw, k, strict);
        if (!E) continue;
        ++used;
        maxE = std::max<long>(maxE, E);
        const bool tilt = !(cu[1] == 0.0f && cw[1] == 0.0f);
        const float C = kPixBias + 0.5f + (float)E / 65536.0f;
        for (int z = 0; z < ez; ++z) {
            std::vector<char> close_chunk(ey / 8 + 1, 0);
            for (int x = 0; x < ex; ++x) {
                const float fx = (float)x, fz = (float)z;
                const float nw = fmaf(rw.cx, fx, fmaf(rw.cz, fz, rw.c0)), nv = fmaf(rv.cx, fx, fmaf(rv.cz, fz, rv.c0)),
                            nu = fmaf(ru.cx, fx, fmaf(ru.cz, fz, ru.c0));
                // the reciprocal: anything within 2^-22 of the exact one, and a Newton step
                const double wob = (rand() % 2001 - 1000) * (1e-3 / 4194304.0);
                const float ya = (float)(1.0 / (double)nw * (1.0 + wob));
                const float y = fmaf(fmaf(-nw, ya, 1.0f), ya, ya);
                const float V0 = fmaf(nv, y, C), U0 = fmaf(nu, y, C);
                volatile float V1 = rv.cy * y, V2 = 0, U1 = 0, U2 = 0;
                if (tilt) {
                    const volatile float e = rw.cy * y, nvy = nv * y, nuy = nu * y, ucy = ru.cy * y;
                    V1 = fmaf(-nvy, e, V1);
                    V2 = -(V1 * e);
                    U1 = fmaf(-nuy, e, ucy);
                    U2 = -(U1 * e);
                }
                const float px = pos(at[0] + x, vx, o[0], strict), pz = pos(at[2] + z, vx, o[2], strict);
                for (int c0 = 0; c0 < ey; c0 += 8) {
                    const float k0 = (float)c0;
                    const float v0 = tilt ? fmaf(k0, fmaf(k0, V2, V1), V0) : fmaf(k0, V1, V0),
                                u0 = tilt ? fmaf(k0, fmaf(k0, U2, U1), U0) : U0,
                                v1 = tilt ? fmaf(2 * k0, V2, V1) : V1, u1 = tilt ? fmaf(2 * k0, U2, U1) : 0.0f;
                    for (int j = 0; j < 8; ++j) {
                        const float kk = (float)j;
                        const float v = tilt ? fmaf(kk, fmaf(kk, V2, v1), v0) : fmaf(kk, v1, v0),
                                    u = tilt ? fmaf(kk, fmaf(kk, U2, u1), u0) : U0;
                        const long dv = fl(v) - 128, du = fl(u) - 128;
                        ++pairs;
                        const bool cv_ = (pix_bits_of(v) & 0xffffu) < 2u * E, cu_ = (pix_bits_of(u) & 0xffffu) < 2u * E;
                        if (cv_ || (tilt && cu_)) close_chunk[c0 / 8] = 1;
                        double iu, iv;
                        contract(q, px, pos(at[1] + c0 + j, vx, o[1], strict), pz, (float)off, strict, iu, iv);
                        const bool in = iu >= k.l && iu < k.r && iv >= k.b && iv < k.t;
                        const bool got = du >= 0 && du < k.r - k.l && dv >= 0 && dv < k.t - k.b;
                        if (cv_ || cu_) continue;
                        ++decided;
                        if (in != got || (in && (iu - k.l != du || iv - k.b != dv))) ++wrong;
                    }
                }
            }
            for (int c = 0; c < ey / 8; ++c) {
                ++chunks;
                close_chunks += close_chunk[c];
            }
        }
    }
    printf("%ld %ld %ld %ld %ld %ld %ld\n", used, pairs, decided, wrong, close_chunks, chunks, maxE);
    return wrong ? 1 : 0;
}
