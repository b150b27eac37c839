// The fixed-point transforms' arithmetic (fx64.cuh) on the host: pencils of a
// length go through its steps as the kernels take them, in the scale that
// pencil_scale gives them.
//   fx64_check list                 lines "L kind radices...": every transform that can run
//   fx64_check run L kind radices   pencils on stdin, results on stdout (doubles)
// kinds: s strided (complex in, complex out, forward), c two spectra of kz <= L/2
// (complex) to two real rows, r two real rows to two spectra.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "fx64_len.cuh"

using namespace fx;

namespace {
int word(double v) {  // high word
  long long b;
  std::memcpy(&b, &v, 8);
  return int(b >> 32);
}
long long bits(double v) {
  long long b;
  std::memcpy(&b, &v, 8);
  return b;
}

template <int R> void dft(I2 *v) { Dft<R>::run(v); }
void butterfly(int R, I2 *v) {
  switch (R) {
    case 2: return dft<2>(v);
    case 3: return dft<3>(v);
    case 4: return dft<4>(v);
    case 5: return dft<5>(v);
    case 6: return dft<6>(v);
    case 7: return dft<7>(v);
    case 8: return dft<8>(v);
    case 9: return dft<9>(v);
    case 10: return dft<10>(v);
    case 12: return dft<12>(v);
    case 14: return dft<14>(v);
    case 15: return dft<15>(v);
    case 16: return dft<16>(v);
    case 18: return dft<18>(v);
    case 20: return dft<20>(v);
    case 21: return dft<21>(v);
    case 24: return dft<24>(v);
    default: std::abort();
  }
}

void transform(std::vector<I2> &a, const std::vector<int> &R) {
  const int L = int(a.size());
  std::vector<I2> b(L);
  int NS = 1;
  for (size_t q = 0; q < R.size(); ++q) {
    const int r = R[q], nb = L / r;
    for (int j = 0; j < nb; ++j) {
      I2 v[24];
      const int lo = j % NS, hi = j / NS, inc = lo * (nb / NS);
      for (int e = 0; e < r; ++e) {
        v[e] = a[j + e * nb];
        if (q == 0) continue;
        int4 cp;
        int2 m;
        twiddle_constants(e * inc, L, &cp, &m);
        if (doubled(int(q), int(R.size()))) v[e] = v[e] + v[e];
        v[e] = e == 0 ? quarter(v[0]) : twiddle4(v[e], cp, m);
      }
      butterfly(r, v);
      for (int e = 0; e < r; ++e) b[hi * NS * r + lo + e * NS] = v[e];
    }
    a.swap(b);
    NS *= r;
  }
}

int scale(double top, int sum, const std::vector<int> &R, FxKind kind) {
  return pencil_scale(word(top), sum, int(R.size()), [&](int q) {
    int ns = 1;
    for (int p = 0; p <= q; ++p) ns *= R[p];
    return growth(ns, kind);
  });
}
int exponent(double top) { return word(top) >> 20; }

void list() {
  auto line = [](int L, char kind, const int *R, int n, bool rev) {
    std::printf("%d %c", L, kind);
    for (int q = 0; q < n; ++q) std::printf(" %d", R[rev ? n - 1 - q : q]);
    std::printf("\n");
  };
#define ENTRY(L_, PADDED, GRID)                                          \
  {                                                                      \
    const int R[3] = {Len<L_>::R(0), Len<L_>::R(1), Len<L_>::R(2)};      \
    line(L_, 's', R, Len<L_>::steps, true);                              \
    line(L_, 'c', R, Len<L_>::steps, true);                              \
    if (PADDED) line(L_, 's', R, Len<L_>::steps, false);                 \
    if (PADDED) line(L_, 'r', R, Len<L_>::steps, false);                 \
  }
  FX_LENGTHS(ENTRY)
  for (int L = 8; L <= 1152; L += 2) {
    FxPlan p;
    if (!fx_plan(L, FX_STRIDED, &p)) continue;
    for (char kind : {'s', 'c', 'r'}) line(L, kind, p.R, p.steps, false);
  }
}

void run(int L, char kind, const std::vector<int> &R) {
  const int h = L / 2, words = kind == 's' ? 2 * L : (kind == 'c' ? 4 * (h + 1) : 2 * L);
  std::vector<double> in(words), out;
  const int steps = int(R.size()), losses = bits_lost(steps - 1, steps);
  while (std::fread(in.data(), 8, words, stdin) == size_t(words)) {
    double top = 0.0;
    if (kind == 'c')  // only the real parts of the modes 0 and L / 2 count
      for (int row = 0; row < 2; ++row) in[2 * row * (h + 1) + 1] = in[2 * (row * (h + 1) + h) + 1] = 0.0;
    for (double v : in) top = std::max(top, std::fabs(v));
    float sum = 0.f;  // of the larger components; of all values of real rows
    for (int e = 0; e < words; e += kind == 'r' ? 1 : 2)
      sum += sum_term(word(kind == 'r' ? std::fabs(in[e]) : std::max(std::fabs(in[e]), std::fabs(in[e + 1]))), sum_base(word(top)));
    const int sw = sum_word(sum, word(top)) + (kind == 'r' ? 0 : kSqrt2) + (kind == 'c' ? kTwice : 0);
    const int k = scale(top, sw, R, kind == 'c' ? FX_C2R : FX_STRIDED), sh = shift_of(exponent(top), k);
    const bool round = kind == 'c' && steps > 2;
    auto fix = [&](double v) { return round ? to_fixed_r(bits(v), sh) : to_fixed_p(bits(v), sh); };
    auto back = [&](long long v, int half) { return std::ldexp(double(v), losses - k - half); };
    std::vector<I2> a(L, I2{0, 0});
    out.clear();
    if (kind == 's') {
      for (int e = 0; e < L; ++e) a[e] = {fix(in[2 * e]), fix(in[2 * e + 1])};
      transform(a, R);
      for (const I2 &v : a) {
        out.push_back(back(v.x, 0));
        out.push_back(back(v.y, 0));
      }
    } else if (kind == 'c') {
      const double *A = in.data(), *B = A + 2 * (h + 1);
      for (int e = 0; e <= h; ++e) {
        const long long ax = fix(A[2 * e]), ay = fix(A[2 * e + 1]), bx = fix(B[2 * e]), by = fix(B[2 * e + 1]);
        if (e == 0 || e == h) {
          a[e] = {bx, ax};
        } else {
          a[e] = {ay + bx, ax - by};
          a[L - e] = {bx - ay, ax + by};
        }
      }
      transform(a, R);
      for (const I2 &v : a) out.push_back(back(v.y, 0));
      for (const I2 &v : a) out.push_back(back(v.x, 0));
    } else {
      for (int e = 0; e < L; ++e) a[e] = {fix(in[e]), fix(in[L + e])};
      transform(a, R);
      for (int second = 0; second < 2; ++second)
        for (int e = 0; e <= h; ++e) {
          const I2 u = a[e], w = a[e ? L - e : 0];
          out.push_back(back(second ? u.y + w.y : u.x + w.x, 1));
          out.push_back(back(second ? w.x - u.x : u.y - w.y, 1));
        }
    }
    std::fwrite(out.data(), 8, out.size(), stdout);
  }
}
}  // namespace

int main(int argc, char **argv) {
  if (argc > 1 && std::string(argv[1]) == "list") {
    list();
  } else if (argc > 4) {
    std::vector<int> R;
    for (int q = 4; q < argc; ++q) R.push_back(std::atoi(argv[q]));
    run(std::atoi(argv[2]), argv[3][0], R);
  } else {
    return 2;
  }
  return 0;
}
