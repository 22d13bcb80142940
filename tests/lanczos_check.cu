// Checks the precision of a Lanczos step's kernels (kernels.cuh, nbspmv.cuh) on
// the device, each against the value that its FP64 arithmetic must give:
//   alpha of a diagonal operator whose products are whole multiples of 2^-24
//     below 1: the sum is exact in FP64 in any order, and must be it;
//   the start vector over its norm, and the next one over beta: one rounding
//     (FP32: of a quotient rounded to FP64 before, or of 1 / beta before).
// Prints one line a check; exits 0 when all hold.
#include <cmath>
#include <cstdio>
#include <vector>

#include "kernels.cuh"
#include "nbspmv.cuh"

using namespace simp;

template <class T>
T* device(const std::vector<T>& h) {
  T* d = nullptr;
  if (cudaMalloc(&d, h.size() * sizeof(T)) != cudaSuccess) exit(2);
  if (cudaMemcpy(d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice) != cudaSuccess) exit(2);
  return d;
}

template <class T>
std::vector<T> host(const T* d, size_t n) {
  std::vector<T> h(n);
  if (cudaMemcpy(h.data(), d, n * sizeof(T), cudaMemcpyDeviceToHost) != cudaSuccess) exit(2);
  return h;
}

unsigned long long state = 0x9E3779B97F4A7C15ull;
unsigned random24() {
  state ^= state << 13;
  state ^= state >> 7;
  state ^= state << 17;
  return static_cast<unsigned>(state >> 40);
}

// One step of nodes * B unknowns, a row's values all in its node's own block,
// those off the diagonal zero.
template <int VS, int B, class T>
int check(const char* name, int nodes) {
  const int n = nodes * B;
  std::vector<int> node_of(n), first(nodes + 1), self(nodes), nbr(nodes), off(nodes, 0), ptr(nodes + 1), rowptr(n + 1),
      col(n * B);
  std::vector<T> val(static_cast<size_t>(n) * B, T(0));
  std::vector<double> start(n);
  for (int I = 0; I <= nodes; ++I) first[I] = B * I, ptr[I] = I;
  for (int I = 0; I < nodes; ++I) nbr[I] = self[I] = I;
  for (int i = 0; i <= n; ++i) rowptr[i] = i * B;
  double norm = 0.0;
  for (int i = 0; i < n; ++i) {
    node_of[i] = i / B;
    for (int k = 0; k < B; ++k) col[i * B + k] = i / B * B + k;
    start[i] = 1.0 + 0.5 * std::sin(1.7 * i + 0.3);
    norm += start[i] * start[i];
    val[static_cast<size_t>(i) * B + i % B] = static_cast<T>((random24() | 1) * 0x1p-24);
  }
  norm = std::sqrt(norm);
  for (double& x : start) x /= norm;
  const NodeView pat{device(ptr), device(nbr), device(off)};
  int *dnode = device(node_of), *dfirst = device(first), *dself = device(self), *drow = device(rowptr), *dcol = device(col);
  T* dval = device(val);
  double* dstart = device(start);
  const std::vector<T> zero(n, T(0)), one(n, T(1));
  T *s = device(zero), *w = device(zero), *t = device(zero), *v = device(zero);
  double* dinv = device(std::vector<double>(n, 0.0));
  const unsigned grid = VS == kNodeWarp ? (nodes * 32 + 255) / 256 : (static_cast<unsigned>(n) * VS + 255) / 256;
  double *ab = device(std::vector<double>(4, 0.0)), *part = device(std::vector<double>(grid + 1024, 0.0));
  LzScalars* sc = device(std::vector<LzScalars>(1));
  int bad = 0;
  auto report = [&](const char* what, double worst, double limit) {
    printf("%s %s: %g (limit %g)\n", name, what, worst, limit);
    if (!(worst <= limit)) bad = 1;
  };

  // the start vector
  k_lz_reset<<<1, 1>>>(sc);
  k_level_start<T><<<(n + 255) / 256, 256>>>(n, dnode, dfirst, dself, pat, drow, dval, dstart, dinv, nullptr, s, w,
                                             t, v, 0, sc);
  const auto w0 = host(w, n);
  double worst = 0.0;
  for (int i = 0; i < n; ++i) worst = std::fmax(worst, std::fabs(static_cast<double>(w0[i]) - static_cast<T>(start[i])));
  report("start", worst, 0.0);

  // alpha with s = w = t = 1: the row products are the diagonal
  for (T* x : {s, w, t}) cudaMemcpy(x, one.data(), n * sizeof(T), cudaMemcpyHostToDevice);
  cudaMemcpy(v, zero.data(), n * sizeof(T), cudaMemcpyHostToDevice);
  k_lz_rows<VS, B, T><<<grid, 256>>>(n, dnode, pat, drow, dcol, dval, t, s, w, v, ab, part, sc);
  double exact = 0.0;
  for (int i = 0; i < n; ++i) exact += static_cast<double>(val[static_cast<size_t>(i) * B + i % B]);
  const double alpha = host(ab, 1)[0];
  report("alpha", std::fabs(alpha - exact), 0.0);

  // beta, and the next vector over it
  k_lz_norm<T><<<8, 256>>>(s, w, v, t, n, ab, part, sc);
  const auto u = host(w, n);
  const double beta = host(ab, 2)[1];
  k_lz_rows<VS, B, T><<<grid, 256>>>(n, dnode, pat, drow, dcol, dval, t, s, w, v, ab + 2, part, sc);
  const auto v1 = host(v, n);
  worst = 0.0;
  for (int i = 0; i < n; ++i) {
    if (sizeof(T) == 4) {
      const float f = static_cast<float>(u[i]) * static_cast<float>(1.0 / beta);
      worst = std::fmax(worst, std::fabs(static_cast<double>(v1[i]) - f));
    } else {  // units in the last place of the quotient
      const long double q = static_cast<long double>(u[i]) / beta;
      const double rounded = static_cast<double>(q), ulp = std::fabs(std::nextafter(rounded, INFINITY) - rounded);
      if (rounded != 0.0) worst = std::fmax(worst, static_cast<double>(std::fabs((static_cast<long double>(v1[i]) - q) / ulp)));
    }
  }
  report("next", worst, sizeof(T) == 4 ? 0.0 : 0.501);
  if (cudaDeviceSynchronize() != cudaSuccess) return 1;
  return bad;
}

int main() {
  int bad = 0;
  bad |= check<4, 3, float>("float, 4 lanes a row", 999);
  bad |= check<8, 3, float>("float, 8 lanes a row", 999);
  bad |= check<32, 2, float>("float, 32 lanes a row", 101);
  bad |= check<kNodeWarp, 6, float>("float, a warp a node", 333);
  bad |= check<4, 3, double>("double, 4 lanes a row", 999);
  bad |= check<8, 6, double>("double, 8 lanes a row", 57);
  return bad;
}
