// The published pair evaluation (angular dislocations, image and free-surface
// correction: pair_tractions, pair_tractions_hs) in long double, for the CPU tests: a
// yardstick where its FP64 evaluation loses digits (far receivers of thin triangles).
// Test infrastructure only.  stdin and stdout as in seg_host_check.cpp.
#include <cmath>
#include <cstdio>

typedef long double Wide;
#define PQ3D_OPCOUNT
#define double Wide
#include "../pyquake3d_gb300/csrc/hs_device.cuh"
#undef double

using namespace pq3d::gf;

struct Arr {
    const Wide *f;
    Wide operator()(int i) const { return f[i]; }
};

int main()
{
    int n;
    double ratio;
    if (scanf("%d %lf", &n, &ratio) != 2) return 1;
    const Wide mu = 32038120320.0L, lam = ratio * mu, pi = 3.14159265358979323846264338327950288L;
    const Wide nu = 1.0L / (1.0L + lam / mu) / 2.0L, k = 1.0L / (8.0L * pi * (1.0L - nu));
    for (int c = 0; c < n; ++c) {
        Wide v[21];
        unsigned bits;
        for (int i = 0; i < 21; ++i) {
            double d;
            if (scanf("%lf", &d) != 1) return 1;
            v[i] = d;
        }
        if (scanf("%u", &bits) != 1) return 1;
        const Wide *P1 = v, *P2 = v + 3, *P3 = v + 6, *R = v + 9;
        const Wide Q1[3] = {v[0], v[1], -v[2]}, Q2[3] = {v[3], v[4], -v[5]}, Q3[3] = {v[6], v[7], -v[8]};
        Wide src[kSrcStride], img[kSrcStride], g[kFscStride], t[4][3];
        setup_source(P1, P2, P3, src, 1);
        setup_source(Q1, Q2, Q3, img, 1);
        setup_fsc(P1, P2, P3, g, 1);
        pair_tractions(Arr{src}, R, nu, k, 2 * mu, lam, t[0], t[1]);
        pair_tractions_hs(Arr{src}, Arr{img}, Arr{g}, R, nu, k, 2 * mu, lam, t[2], t[3]);
        for (int q = 0; q < 4; ++q)
            for (int i = 0; i < 3; ++i) printf("%.20Lg ", t[q][i]);
        printf("\n");
    }
    return 0;
}
