// Rounding errors of FP64 kernels against 80-bit sums, beside those of a plain
// FP64 evaluation of the same sums on the host.  Built and run by
// tests/test_gpu_errors.py; one line per check: name, error, bound.
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "rtfmm_kernels.cuh"
#include "rtfmm_rsqrt.cuh"

using namespace rtfmm_b200;
using LD = long double;

#define CK(x)                                                          \
  do {                                                                 \
    cudaError_t e_ = (x);                                              \
    if (e_ != cudaSuccess) {                                           \
      std::printf("%s: %s\n", #x, cudaGetErrorString(e_));             \
      std::exit(2);                                                    \
    }                                                                  \
  } while (0)

template <typename T>
T* up(const std::vector<T>& h) {
  T* d = nullptr;
  CK(cudaMalloc(&d, sizeof(T) * h.size()));
  CK(cudaMemcpy(d, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice));
  return d;
}
template <typename T>
void down(std::vector<T>& h, const T* d) {
  CK(cudaDeviceSynchronize());
  CK(cudaMemcpy(h.data(), d, sizeof(T) * h.size(), cudaMemcpyDeviceToHost));
}

template <typename T>
struct C {
  T r, i;
};
template <typename T>
void cmad(C<T>& o, C<T> a, C<T> b) {
  o.r = std::fma(a.r, b.r, o.r);
  o.r = std::fma(-a.i, b.i, o.r);
  o.i = std::fma(a.r, b.i, o.i);
  o.i = std::fma(a.i, b.r, o.i);
}
double sq(LD x) { return (double)(x * x); }

// -- reciprocal square roots ------------------------------------------------
__global__ void k_rsqrt(const double* x, int n, double* full, double* twice) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  full[i] = rsqrt_or_zero(x[i]);
  twice[i] = rsqrt_twice(x[i]);
}
void check_rsqrt() {
  std::mt19937_64 g(1);
  std::uniform_real_distribution<double> e(-100, 100), m(1, 4);
  std::vector<double> x(1 << 20);
  for (size_t i = 0; i < x.size(); ++i) x[i] = i % 4 ? m(g) * std::exp2(2 * std::floor(e(g))) : std::pow(10.0, e(g));
  x[0] = 0.0;
  std::vector<double> f(x.size()), t(x.size());
  double *dx = up(x), *df = up(f), *dt = up(t);
  k_rsqrt<<<(int)((x.size() + 255) / 256), 256>>>(dx, (int)x.size(), df, dt);
  CK(cudaGetLastError());
  down(f, df);
  down(t, dt);
  double ef = 0, et = 0;
  for (size_t i = 1; i < x.size(); ++i) {
    const LD r = 1 / sqrtl((LD)x[i]);
    ef = std::max(ef, (double)fabsl(f[i] / r - 1));
    et = std::max(et, (double)fabsl(t[i] / (2 * r) - 1));
  }
  // the last rounding (2^-53) and that of x y in the residual, halved (2^-54);
  // the other roundings are of terms a millionth of the result
  std::printf("rsqrt %.3e 1.67e-16\n", ef);
  // one Newton step from a seed good to 9.1e-7: 3/2 of its square
  std::printf("rsqrt_twice %.3e 1.3e-12\n", et);
  std::printf("rsqrt_zero %.3e 0\n", std::abs(f[0]) + std::abs(t[0]));
}

// -- the 8x8 Hadamard ----------------------------------------------------------
// Coefficients that depend on the offset of a child pair; `heavy`: most of the
// sums comes from the first direction and from the children at x = 1, as for a
// cluster.
void check_hadamard(bool heavy) {
  const int Nf = 4, nsrc = 60, ntar = 130;
  std::mt19937_64 g(2);
  std::normal_distribution<double> n;
  std::vector<double> cc((size_t)26 * 64 * Nf * 2), Q((size_t)Nf * nsrc * 16), Pk((size_t)Nf * ntar * 16);
  std::vector<int> src((size_t)26 * ntar);
  for (int d = 0; d < 26; ++d)
    for (int f = 0; f < Nf; ++f) {
      C<double> v[3][3][3];
      for (auto& a : v)
        for (auto& b : a)
          for (auto& c : b) c = {n(g), n(g)};
      for (int s = 0; s < 8; ++s)
        for (int t = 0; t < 8; ++t) {
          const int dx = (s >> 2) - (t >> 2), dy = (s >> 1 & 1) - (t >> 1 & 1), dz = (s & 1) - (t & 1);
          const double k = heavy ? (d ? 0.01 : 1.0) * (dx ? 0.1 : 1.0) : 1.0;
          double* o = &cc[(((size_t)d * 64 + s * 8 + t) * Nf + f) * 2];
          o[0] = k * v[dx + 1][dy + 1][dz + 1].r;
          o[1] = k * v[dx + 1][dy + 1][dz + 1].i;
        }
    }
  // source spectra in chunks of two slots
  auto q = [&](int f, int s, int slot) { return &Q[(((size_t)f * 4 + slot / 2) * nsrc + s) * 4 + slot % 2 * 2]; };
  for (int f = 0; f < Nf; ++f)
    for (int s = 0; s < nsrc; ++s)
      for (int j = 0; j < 8; ++j)
        for (int c = 0; c < 2; ++c) q(f, s, j)[c] = n(g) * (heavy && j < 4 ? 0.05 : 1.0);
  std::uniform_int_distribution<int> any(-nsrc / 2, nsrc - 1), some(0, nsrc - 1);
  for (int d = 0; d < 26; ++d)
    for (int t = 0; t < ntar; ++t) src[(size_t)d * ntar + t] = d ? std::max(-1, any(g)) : some(g);
  double *dcc = up(cc), *dQ = up(Q), *dPk = up(Pk), *dG = nullptr;
  int* dsrc = up(src);
  CK(cudaMalloc(&dG, sizeof(double) * g8_layout_size(Nf, false)));
  CK(launch_g8_layout(dcc, Nf, dG, nullptr));
  CK(launch_m2l_hadamard8(dQ, dG, dsrc, ntar, nsrc, Nf, dPk, nullptr));
  down(Pk, dPk);
  double ek = 0, eh = 0;
  for (int f = 0; f < Nf; ++f)
    for (int t = 0; t < ntar; ++t)
      for (int j = 0; j < 8; ++j) {
        C<LD> ref{};
        C<double> sum{};
        for (int d = 0; d < 26; ++d) {
          const int s = src[(size_t)d * ntar + t];
          if (s < 0) continue;
          C<double> part{};  // of one direction
          for (int k = 0; k < 8; ++k) {
            const double *o = &cc[(((size_t)d * 64 + k * 8 + j) * Nf + f) * 2], *x = q(f, s, k);
            cmad(ref, C<LD>{o[0], o[1]}, C<LD>{x[0], x[1]});
            cmad(part, C<double>{o[0], o[1]}, C<double>{x[0], x[1]});
          }
          sum.r += part.r;
          sum.i += part.i;
        }
        const double* p = &Pk[(((size_t)f * ntar + t) * 8 + j) * 2];
        ek += sq(p[0] - ref.r) + sq(p[1] - ref.i);
        eh += sq(sum.r - ref.r) + sq(sum.i - ref.i);
      }
  std::printf("hadamard%s %.3f 1.1\n", heavy ? "_heavy" : "", std::sqrt(ek / eh));
}

// -- the transforms ---------------------------------------------------------------
template <typename T>
struct Grid {  // one child's transform, separable, each sum in order
  int P, N;
  std::vector<T> c, s;
  Grid(int P_) : P(P_), N(2 * P_ - 1) {
    for (int m = 0; m < N; ++m) {
      c.push_back(sizeof(T) == 8 ? (T)std::cos(2.0 * M_PI * m / N) : (T)cosl(2.0L * acosl(-1.0L) * m / N));
      s.push_back(sizeof(T) == 8 ? (T)std::sin(2.0 * M_PI * m / N) : (T)sinl(2.0L * acosl(-1.0L) * m / N));
    }
  }
  // corner [z][y][x] -> spectrum [kz][ky][kx]
  std::vector<C<T>> forward(const std::vector<T>& v) const {
    std::vector<C<T>> a(P * P * P), b(P * N * P), o(N * N * P);
    for (int l = 0; l < P * P; ++l)
      for (int k = 0; k < P; ++k)
        for (int x = 0; x < P; ++x) {
          a[l * P + k].r = std::fma(v[l * P + x], c[k * x % N], a[l * P + k].r);
          a[l * P + k].i = std::fma(v[l * P + x], -s[k * x % N], a[l * P + k].i);
        }
    for (int z = 0; z < P; ++z)
      for (int k = 0; k < N; ++k)
        for (int x = 0; x < P; ++x)
          for (int y = 0; y < P; ++y)
            cmad(b[(z * N + k) * P + x], a[(z * P + y) * P + x], C<T>{c[k * y % N], -s[k * y % N]});
    for (int k = 0; k < N; ++k)
      for (int l = 0; l < N * P; ++l)
        for (int z = 0; z < P; ++z) cmad(o[k * N * P + l], b[z * N * P + l], C<T>{c[k * z % N], -s[k * z % N]});
    return o;
  }
  // spectrum -> the corner [P-1, 2P-2]^3
  std::vector<T> inverse(const std::vector<C<T>>& f) const {
    std::vector<C<T>> a(P * N * P), b(P * P * P);
    std::vector<T> o(P * P * P);
    auto w = [&](int k, int x) { return C<T>{c[k * (P - 1 + x) % N], s[k * (P - 1 + x) % N]}; };
    for (int z = 0; z < P; ++z)
      for (int l = 0; l < N * P; ++l)
        for (int k = 0; k < N; ++k) cmad(a[z * N * P + l], f[k * N * P + l], w(k, z));
    for (int z = 0; z < P; ++z)
      for (int y = 0; y < P; ++y)
        for (int x = 0; x < P; ++x)
          for (int k = 0; k < N; ++k) cmad(b[(z * P + y) * P + x], a[(z * N + k) * P + x], w(k, y));
    for (int l = 0; l < P * P; ++l)
      for (int x = 0; x < P; ++x) {
        T acc = 0;
        for (int k = 1; k < P; ++k) {
          acc = std::fma(b[l * P + k].r, w(k, x).r, acc);
          acc = std::fma(-b[l * P + k].i, w(k, x).i, acc);
        }
        o[l * P + x] = b[l * P].r + 2 * acc;
      }
    return o;
  }
};

void check_transforms(int P, bool smooth) {
  const int N = 2 * P - 1, Nf = N * N * P, np = 3;
  std::mt19937_64 g(3);
  std::normal_distribution<double> n;
  auto value = [&]() { return smooth ? 1 + 0.01 * n(g) : n(g); };
  std::vector<int> ijk;
  for (int i = 0; i < P; ++i)
    for (int j = 0; j < P; ++j)
      for (int k = 0; k < P; ++k)
        if (i == 0 || i == P - 1 || j == 0 || j == P - 1 || k == 0 || k == P - 1)
          for (int c : {i, j, k}) ijk.push_back(c);
  const int ns = (int)ijk.size() / 3, spu = m2l_up_slots<double>(P), spd = m2l_down_slots<double>(P);
  auto items = [&](int sp) {
    std::vector<int> v;
    for (int p = 0; p < np; ++p)
      for (int s = 0; s < 8; s += sp) {
        std::vector<int> it(10, -1);
        it[0] = p;
        it[1] = s;
        for (int j = 0; j < sp; ++j) it[2 + j] = 8 * p + s + j;
        v.insert(v.end(), it.begin(), it.end());
      }
    return v;
  };
  const Grid<double> G(P);
  const Grid<LD> L(P);
  std::vector<double> tw(2 * N), scale(np, 1.0), qe((size_t)8 * np * ns), Q((size_t)Nf * np * 16), Pk(Q.size()),
      chk(qe.size(), 0.0);
  for (int m = 0; m < N; ++m) {
    tw[2 * m] = G.c[m];
    tw[2 * m + 1] = -G.s[m];
  }
  for (double& v : qe) v = value();
  for (double& v : Pk) v = value();
  const std::vector<int> iu = items(spu), id = items(spd);
  double *dq = up(qe), *dQ = up(Q), *dP = up(Pk), *dc = up(chk), *dt = up(tw), *ds = up(scale);
  int *du = up(iu), *dd = up(id), *dj = up(ijk);
  CK(launch_m2l_up<double>(dq, du, (int)iu.size() / 10, dj, dt, P, ns, np, spu, dQ, nullptr));
  CK(launch_m2l_down<double>(dP, dd, ds, (int)id.size() / 10, dj, dt, P, ns, np, spd, dc, nullptr));
  down(Q, dQ);
  down(chk, dc);
  double uk = 0, uh = 0, dk = 0, dh = 0;
  for (int p = 0; p < np; ++p)
    for (int j = 0; j < 8; ++j) {
      std::vector<double> v(P * P * P, 0.0);
      std::vector<C<double>> f(Nf);
      for (int i = 0; i < ns; ++i)
        v[(ijk[3 * i + 2] * P + ijk[3 * i + 1]) * P + ijk[3 * i]] = qe[(size_t)(8 * p + j) * ns + i];
      for (int k = 0; k < Nf; ++k) {
        const double* x = &Pk[(((size_t)k * np + p) * 8 + j) * 2];
        f[k] = {x[0], x[1]};
      }
      const auto F = G.forward(v);
      const auto FL = L.forward(std::vector<LD>(v.begin(), v.end()));
      std::vector<C<LD>> fl(Nf);
      for (int k = 0; k < Nf; ++k) fl[k] = {f[k].r, f[k].i};
      const auto I = G.inverse(f);
      const auto IL = L.inverse(fl);
      for (int k = 0; k < Nf; ++k) {
        const double* x = &Q[(((size_t)k * 4 + j / 2) * np + p) * 4 + j % 2 * 2];
        uk += sq(x[0] - FL[k].r) + sq(x[1] - FL[k].i);
        uh += sq(F[k].r - FL[k].r) + sq(F[k].i - FL[k].i);
      }
      for (int i = 0; i < ns; ++i) {
        const int o = (ijk[3 * i + 2] * P + ijk[3 * i + 1]) * P + ijk[3 * i];
        dk += sq(chk[(size_t)(8 * p + j) * ns + i] - IL[o]);
        dh += sq(I[o] - IL[o]);
      }
    }
  std::printf("up_%d%s %.3f 1.1\n", P, smooth ? "_smooth" : "", std::sqrt(uk / uh));
  std::printf("down_%d%s %.3f 1.1\n", P, smooth ? "_smooth" : "", std::sqrt(dk / dh));
}

int main() {
  check_rsqrt();
  check_hadamard(false);
  check_hadamard(true);
  for (int P = 4; P <= 10; ++P)
    for (bool smooth : {false, true}) check_transforms(P, smooth);
}
