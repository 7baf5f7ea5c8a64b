// Test harness (built by tests/test_gpu_fp64_forms.py): the FP64 forms of pip_fp64_forms.cuh
// on the device.  Solvers against the literal forms of pip_physics.cuh evaluated on the host
// (no contraction, as the CPU restatement) over seeded faces of six kinds (unrelated states, some supersonic; nearby states; mirror pairs with vn and Bn
// negated, and with the tangential fields negated; a near-zero Bn; states at the floors), the
// difference relative to p + rho vn^2 + |B|^2 of the larger side; the limited face states
// against minmod<double> bit for bit; the roots against IEEE ones in ulps.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include "../pip_b200/csrc/pip_fp64_forms.cuh"

using namespace pip;

__global__ void run(int n, const double *vl, const double *vr, double gm, double *fd, double *fc) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double igm1 = 1.0 / (gm - 1.0);
  double a[9], b[9], o[9], ha[5], hb[5], ho[5];
  for (int k = 0; k < 9; ++k) {
    a[k] = vl[9ll * i + k];
    b[k] = vr[9ll * i + k];
  }
  for (int k = 0; k < 5; ++k) {
    ha[k] = a[k];
    hb[k] = b[k];
  }
  hlld_flux_fast<9>(a, b, o, gm, igm1, 1.5);
  for (int k = 0; k < 9; ++k) fd[9ll * i + k] = o[k];
  hllc_flux_fast(ha, hb, ho, gm, igm1);
  for (int k = 0; k < 5; ++k) fc[5ll * i + k] = ho[k];
}

__global__ void scalars(int n, const double *x, double *out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double v = fabs(x[4ll * i]);
  out[6ll * i] = sqrt_nr(v);
  out[6ll * i + 1] = rsqrt_nr(v);
  face_pair(x[4ll * i], x[4ll * i + 1], x[4ll * i + 2], x[4ll * i + 3], out[6ll * i + 2], out[6ll * i + 3]);
  out[6ll * i + 4] = x[4ll * i + 1] + 0.5 * minmod<double>(x[4ll * i], x[4ll * i + 1], x[4ll * i + 2]);
  out[6ll * i + 5] = x[4ll * i + 2] - 0.5 * minmod<double>(x[4ll * i + 1], x[4ll * i + 2], x[4ll * i + 3]);
}

static int64_t ordered(double v) {
  int64_t b;
  std::memcpy(&b, &v, sizeof b);
  return b < 0 ? INT64_MIN - b : b;
}

template <typename T>
static T *dev(const std::vector<T> &h) {
  T *d;
  if (cudaMalloc(&d, sizeof(T) * h.size()) != cudaSuccess) exit(2);
  cudaMemcpy(d, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice);
  return d;
}

int main(int argc, char **argv) {
  const int n = argc > 1 ? atoi(argv[1]) : 3 << 18;
  std::mt19937_64 g(977);
  std::uniform_real_distribution<double> U(-1.0, 1.0);
  std::vector<double> vl(9ull * n), vr(9ull * n), fd(9ull * n), fc(5ull * n);
  for (int i = 0; i < n; ++i) {
    const int kind = i % 6;
    double *l = &vl[9ull * i], *r = &vr[9ull * i];
    l[0] = 1.0 + 0.9 * U(g);
    l[4] = 0.5 + 0.45 * U(g);
    for (int k : {1, 2, 3}) l[k] = (kind == 0 ? 2.0 : 0.5) * U(g);
    for (int k : {5, 6, 7, 8}) l[k] = U(g);
    if (kind == 0 && i % 12 == 0) l[1] += 6.0 * U(g);
    for (int k = 0; k < 9; ++k) r[k] = l[k];
    if (kind == 0) {
      r[0] = 1.0 + 0.9 * U(g);
      r[4] = 0.5 + 0.45 * U(g);
      for (int k : {1, 2, 3, 5, 6, 7}) r[k] = l[k] + U(g);
    } else if (kind == 1) {
      for (int k = 0; k < 9; ++k) r[k] = l[k] * (1.0 + 0.05 * U(g));
    } else if (kind == 2) {
      r[1] = -l[1];
      r[5] = -l[5];
    } else if (kind == 3) {
      r[1] = -l[1];
      r[6] = -l[6];
      r[7] = -l[7];
    } else if (kind == 4) {
      l[5] = r[5] = 1e-4 * U(g);
      for (int k : {0, 1, 2, 3, 4, 6, 7}) r[k] = l[k] * (1.0 + 0.3 * U(g));
    } else {
      l[0] = 1e-8;
      l[4] = 1e-8;
      if (i % 12 == 5)
        for (int k : {5, 6, 7}) l[k] = 0.0;
      for (int k = 0; k < 9; ++k) r[k] = l[k] * (1.0 + 0.05 * U(g));
    }
  }
  double *dl = dev(vl), *dr = dev(vr), *a = dev(fd), *b = dev(fc);
  run<<<(n + 127) / 128, 128>>>(n, dl, dr, 5.0 / 3.0, a, b);
  if (cudaDeviceSynchronize() != cudaSuccess) return 1;
  cudaMemcpy(fd.data(), a, sizeof(double) * fd.size(), cudaMemcpyDeviceToHost);
  cudaMemcpy(fc.data(), b, sizeof(double) * fc.size(), cudaMemcpyDeviceToHost);
  double wd[6] = {0}, wc[6] = {0};
  long nonfinite = 0, wall = 0;
  for (int i = 0; i < n; ++i) {
    const double *l = &vl[9ull * i], *r = &vr[9ull * i];
    auto scale = [](const double *v, bool mag) {
      double s = v[4] + v[0] * v[1] * v[1];
      if (mag) s += v[5] * v[5] + v[6] * v[6] + v[7] * v[7] + std::fabs(v[8]);
      return s;
    };
    const double sd = std::fmax(scale(l, true), scale(r, true));
    const double sh = std::fmax(scale(l, false), scale(r, false));
    double a9[9], b9[9], rd[9], a5[5], b5[5], rc[5];
    for (int k = 0; k < 9; ++k) {
      a9[k] = l[k];
      b9[k] = r[k];
      if (k < 5) a5[k] = l[k], b5[k] = r[k];
    }
    hlld_flux<double, 9>(a9, b9, rd, 5.0 / 3.0, 1.5);
    hllc_flux<double>(a5, b5, rc, 5.0 / 3.0);
    for (int k = 0; k < 9; ++k) {
      if (!std::isfinite(fd[9ull * i + k])) ++nonfinite;
      wd[i % 6] = std::fmax(wd[i % 6], std::fabs(fd[9ull * i + k] - rd[k]) / sd);
    }
    for (int k = 0; k < 5; ++k) {
      if (!std::isfinite(fc[5ull * i + k])) ++nonfinite;
      wc[i % 6] = std::fmax(wc[i % 6], std::fabs(fc[5ull * i + k] - rc[k]) / sh);
    }
    // a wall passes no mass
    if (i % 6 == 2 && (fd[9ull * i] != 0.0 || fc[5ull * i] != 0.0)) ++wall;
  }
  // roots over every exponent, slopes over small integers (ties, zeros) and random values
  const int m = 1 << 20;
  std::vector<double> x(4ull * m), out(6ull * m);
  std::uniform_int_distribution<int> E(-900, 900), I(-2, 2);
  for (int i = 0; i < m; ++i)
    for (int k = 0; k < 4; ++k) x[4ull * i + k] = i & 1 ? (double)I(g) : std::ldexp(U(g), k ? 0 : E(g));
  double *dx = dev(x), *dout = dev(out);
  scalars<<<(m + 127) / 128, 128>>>(m, dx, dout);
  if (cudaDeviceSynchronize() != cudaSuccess) return 1;
  cudaMemcpy(out.data(), dout, sizeof(double) * out.size(), cudaMemcpyDeviceToHost);
  int64_t us = 0, ur = 0;
  long slopes = 0;
  for (int i = 0; i < m; ++i) {
    const double v = std::fabs(x[4ull * i]), *o = &out[6ull * i];
    if (v > 1e-270) {
      us = std::max<int64_t>(us, std::llabs(ordered(o[0]) - ordered(std::sqrt(v))));
      const double y = (double)(1.0L / std::sqrt((long double)v));
      ur = std::max<int64_t>(ur, std::llabs(ordered(o[1]) - ordered(y)));
    } else if (o[0] < 0.0 || o[0] > 1e-134 || !std::isfinite(o[1])) {
      ++nonfinite;
    }
    if (o[2] != o[4] || o[3] != o[5]) ++slopes;
  }
  printf("faces %d nonfinite %ld wall_mass %ld slopes %ld sqrt_ulp %lld rsqrt_ulp %lld\n", n, nonfinite, wall,
         slopes, (long long)us, (long long)ur);
  for (int k = 0; k < 6; ++k) printf("kind %d hlld %.3e hllc %.3e\n", k, wd[k], wc[k]);
  return 0;
}
