/* Red-black SOR in long double (64 bits of fraction or more), the reference's
 * scheme (src/solver-rb.c:50-151): p [nz + 2][ny + 2][nx + 2], rhs alike,
 * `iterations` of them; p is rounded to double at the end. */
#include <stdlib.h>

int rb_exact(int nx, int ny, int nz, double dx, double dy, double dz, double omega, int iterations,
    double *p, const double *rhs)
{
  const size_t sj = nx + 2, sk = sj * (ny + 2), n = sk * (nz + 2);
  const long double x2 = (long double)dx * dx, y2 = (long double)dy * dy, z2 = (long double)dz * dz;
  const long double factor = omega * 0.5L * (x2 * y2 * z2) / (y2 * z2 + x2 * z2 + x2 * y2);
  long double *q = malloc(n * sizeof *q);
  if (!q) return 1;
  for (size_t c = 0; c < n; c++) q[c] = p[c];
  for (int it = 0; it < iterations; it++) {
    for (int colour = 1; colour >= 0; colour--) {
#pragma omp parallel for
      for (int k = 1; k <= nz; k++)
        for (int j = 1; j <= ny; j++)
          for (int i = 1; i <= nx; i++) {
            const size_t c = k * sk + j * sj + i;
            if (((i + j + k) & 1) != colour) continue;
            const long double lap = (q[c - 1] - 2 * q[c] + q[c + 1]) / x2 +
                                    (q[c - sj] - 2 * q[c] + q[c + sj]) / y2 +
                                    (q[c - sk] - 2 * q[c] + q[c + sk]) / z2;
            q[c] -= factor * (rhs[c] - lap);
          }
    }
    for (int k = 1; k <= nz; k++)
      for (int j = 1; j <= ny; j++)
        for (int i = 1; i <= nx; i++) {
          const size_t c = k * sk + j * sj + i;
          if (i == 1) q[c - 1] = q[c];
          if (i == nx) q[c + 1] = q[c];
          if (j == 1) q[c - sj] = q[c];
          if (j == ny) q[c + sj] = q[c];
          if (k == 1) q[c - sk] = q[c];
          if (k == nz) q[c + sk] = q[c];
        }
  }
  for (size_t c = 0; c < n; c++) p[c] = (double)q[c];
  free(q);
  return 0;
}
