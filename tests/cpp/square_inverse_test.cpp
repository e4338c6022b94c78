// hg::SquareInverse (heu_gb300/csrc/host_bn.hpp) against the general inverse,
// and its time.  Prints one line per case: bits, n, x, result (hex).
#include <chrono>
#include <cstdio>
#include <string>

#include "../../heu_gb300/csrc/host_bn.hpp"

using hg::BN;

static std::string hex(const BN& v) {
  if (v.is_zero()) return "0";
  std::string s;
  static const char* dig = "0123456789abcdef";
  for (size_t i = v.d.size(); i-- > 0;)
    for (int b = 28; b >= 0; b -= 4) s.push_back(dig[(v.d[i] >> b) & 0xf]);
  return s.substr(s.find_first_not_of('0'));
}

int main() {
  hg::Xoshiro prg(7);
  for (size_t bits : {512, 1024, 1000, 2048, 3072}) {
    const size_t H = (bits + 31) / 32, S = 2 * H;
    BN n = prg.randbits(bits);
    n.d.resize(H, 0);
    n.d[0] |= 1u;
    n.d[(bits - 1) / 32] |= 1u << ((bits - 1) % 32);
    n.trim();
    const BN N = n * n, R = BN(1).shl(32 * S);
    hg::SquareInverse sq;
    sq.n = n;
    sq.N = N;
    sq.R2 = ((R % N) * (R % N)) % N;
    sq.rh2 = R % n;
    const BN ri = BN::invmod(R % n, n);
    sq.rm2 = (ri * ri) % n;
    sq.S = S;
    std::vector<uint32_t> xr(S), out(S);
    const BN cases[] = {BN(1), BN(2), N - BN(1), R % N, n + BN(1), prg.randbits(2 * bits - 1) % N,
                        prg.randbits(2 * bits - 1) % N, BN(0), n, (n * BN(5)) % N};
    for (const BN& x : cases) {
      x.to_limbs(xr.data(), S);
      const bool ok = sq.root_inverse(xr.data(), out.data());
      std::printf("case %zu %s %s %s\n", S, hex(n).c_str(), hex(x).c_str(),
                  ok ? hex(BN::from_limbs(out.data(), S)).c_str() : "none");
    }
    cases[5].to_limbs(xr.data(), S);
    auto us = [&](auto&& f) {
      const auto t0 = std::chrono::steady_clock::now();
      for (int i = 0; i < 5; ++i) f();
      return std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count() * 2e5;
    };
    const double a = us([&] { hg::mont_root_inverse(xr.data(), N, S, out.data()); });
    const double b = us([&] { sq.root_inverse(xr.data(), out.data()); });
    std::printf("time %zu %.1f %.1f\n", bits, a, b);
  }
  return 0;
}
