// The host calls on a device with little free memory, simulated: the linker
// routes the library's cudaMalloc, cudaFree and cudaMemGetInfo through the
// functions below, which keep to a budget.  An optional workspace (the exact
// contractions') must never make a call fail that its mandatory memory allows,
// and every way of doing without it must give the same results: the same bits
// where an operand outside the contraction's range sends the call to the FP64
// kernels anyway, others (the contraction's) where none does.
#include <cmath>
#include <cstdio>
#include <functional>
#include <map>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "sigma_ff.h"
#include "sigma_gpp.h"

extern "C" {
cudaError_t __real_cudaMalloc(void** p, size_t n);
cudaError_t __real_cudaFree(void* p);
}
static size_t g_budget = ~size_t(0) / 4, g_used = 0, g_peak = 0;
static int g_large = 0;         // allocations above 8 MB
static bool g_kept = false;     // the calls' workspaces are small enough to be kept between calls
static std::map<void*, size_t> g_size;
extern "C" cudaError_t __wrap_cudaMalloc(void** p, size_t n) {
  if (g_used + n > g_budget) return cudaErrorMemoryAllocation;
  const cudaError_t e = __real_cudaMalloc(p, n);
  if (e != cudaSuccess) return e;
  g_size[*p] = n;
  g_large += n > 8u << 20;
  g_used += n;
  g_peak = g_used > g_peak ? g_used : g_peak;
  return e;
}
extern "C" cudaError_t __wrap_cudaFree(void* p) {
  const auto it = g_size.find(p);
  if (it != g_size.end()) {
    g_used -= it->second;
    g_size.erase(it);
  }
  return __real_cudaFree(p);
}
extern "C" cudaError_t __wrap_cudaMemGetInfo(size_t* f, size_t* t) {
  *f = g_used > g_budget ? 0 : g_budget - g_used;
  *t = g_budget;
  return cudaSuccess;
}

using cd = sigma_complex128;
static unsigned long long g_rng = 1;
static double uni(double lo, double hi) {
  g_rng = g_rng * 6364136223846793005ull + 1442695040888963407ull;
  return lo + (hi - lo) * (double)(g_rng >> 11) * 0x1p-53;
}
static std::vector<cd> cplx(size_t n, double lo = -1, double hi = 1, double ilo = -1, double ihi = 1) {
  std::vector<cd> v(n);
  for (auto& x : v) x = cd{uni(lo, hi), uni(ilo, ihi)};
  return v;
}
static std::vector<double> real(size_t n, double lo, double hi) {
  std::vector<double> v(n);
  for (auto& x : v) x = uni(lo, hi);
  return v;
}

using Call = std::function<int(std::vector<double>&)>;
static int g_bad = 0;

// The call without limits, with the least memory it takes (found by
// bisection: no optional one), and over budgets from that on.
enum Range { kInside, kOutside, kPartly };  // the operands, of every contraction or of some
static void check(const std::string& name, const Call& call, Range range = kInside) {
  std::vector<double> want, got;
  auto run = [&](size_t budget, std::vector<double>& out) {
    sigma_shutdown();
    g_budget = budget;
    g_peak = g_used;
    return call(out);
  };
  auto same = [&]() {
    double worst = 0, top = 0;
    for (double x : want) top = std::max(top, std::fabs(x));
    for (size_t i = 0; i < want.size(); ++i) worst = std::max(worst, std::fabs(want[i] - got[i]));
    return want.size() == got.size() && worst <= 1e-12 * top;  // NaN fails
  };
  const size_t all = ~size_t(0) / 4;
  int st = run(all, want);
  const size_t full = g_peak;
  if (st != 0) g_bad++, printf("%s: status %d\n", name.c_str(), st);
  size_t low = 0, least = full;
  while (least - low > 1 << 20) {
    const size_t mid = (low + least) / 2;
    st = run(mid, got);
    if (st != 0 && st != SIGMA_ERR_ALLOC) g_bad++, printf("%s with %zu MB: status %d\n", name.c_str(), mid >> 20, st);
    (st == 0 ? least : low) = mid;
  }
  st = run(least, got);
  if (st != 0 || !same()) g_bad++, printf("%s without optional memory: status %d, results %d\n", name.c_str(), st, (int)same());
  if (range != kPartly && (want == got) != (range == kOutside))
    g_bad++, printf("%s: the contraction's range check\n", name.c_str());
  if (range != kInside) return;
  printf("%s: %zu MB with the contraction, %zu MB without\n", name.c_str(), full >> 20, least >> 20);
  if (full < least + (8 << 20)) g_bad++, printf("%s: no contraction ran\n", name.c_str());
  size_t last = 0;
  for (int k = 0; k <= 16; ++k) {
    const size_t budget = least + (2 * full - least) / 16 * k;
    st = run(budget, got);
    if (st != 0 || !same() || g_peak > budget)
      g_bad++, printf("%s with %zu MB: status %d, results %d\n", name.c_str(), budget >> 20, st, (int)same());
    if (k == 16) last = g_peak;
    // the same call again, from its caches
    g_large = 0;
    st = call(got);
    // (the half sum's plan holds its transposed inputs)
    if (k == 16 && g_kept && g_large > (name == "half sum")) g_bad++, printf("%s again: %d large allocations\n", name.c_str(), g_large);
    if (st != 0 || !same()) g_bad++, printf("%s again with %zu MB: status %d, results %d\n", name.c_str(), budget >> 20, st, (int)same());
  }
  if (last != full) g_bad++, printf("%s: %zu MB of %zu at the largest budget\n", name.c_str(), last >> 20, full >> 20);
}

static void all_calls(int nb, int nvb, int nc, int ng, int nf, int ngf) {
  std::vector<int> inv(ng), ind(nc), iota(nc);
  for (int g = 0; g < ng; ++g) inv[g] = (g + 1) * (nc - 1) / ng;
  for (int k = 0; k < nc; ++k) ind[k] = iota[k] = k;
  const std::vector<double> wx = {3.0, 4.0, 5.0}, v = real(nc, 0.1, 10);
  auto am = cplx((size_t)nb * nc), an = cplx((size_t)nb * nc), ie = cplx((size_t)ng * nc),
             wt = cplx((size_t)ng * nc, 0.5, 5, -0.1, 0.1);
  auto rm = real((size_t)nb * nc, -1, 1), rn = real((size_t)nb * nc, -1, 1), re = real((size_t)ng * nc, -1, 1),
             rw = real((size_t)ng * nc, 0.5, 5);
  auto put = [](std::vector<double>& out, const std::vector<cd>& z) {
    for (const cd& x : z) out.insert(out.end(), {x.re, x.im});
  };
  const Call gpp_call = [&](std::vector<double>& out) {
    std::vector<cd> ach(3), asx(3), n1(nb);
    const int st = sigma_gpp_fp64(nb, nvb, nc, ng, 0, 3, inv.data(), ind.data(), wx.data(), 1.0, am.data(), an.data(),
                                  ie.data(), wt.data(), v.data(), ach.data(), asx.data(), n1.data(), nullptr);
    out.clear();
    put(out, ach), put(out, asx), put(out, n1);
    return st;
  };
  const Call real_call = [&](std::vector<double>& out) {
    std::vector<double> ach(3), asx(3), n1(nb);
    const int st =
        sigma_gpp_real_fp64(nb, nvb, nc, ng, 0, 3, inv.data(), ind.data(), wx.data(), 1.0, rm.data(), rn.data(),
                            re.data(), rw.data(), v.data(), ach.data(), asx.data(), n1.data(), nullptr);
    out = ach;
    out.insert(out.end(), asx.begin(), asx.end());
    out.insert(out.end(), n1.begin(), n1.end());
    return st;
  };
  const Call half_call = [&](std::vector<double>& out) {
    std::vector<cd> ach(3), asx(3), n1(nb), st1(1);
    const int st = sigma_gpp_halfsum_fp64(nb, nvb, nc, ng, 0, 3, inv.data(), ind.data(), wx.data(), 1.0, am.data(),
                                          an.data(), ie.data(), wt.data(), v.data(), ach.data(), asx.data(), n1.data(),
                                          st1.data(), nullptr);
    out.clear();
    put(out, ach), put(out, asx), put(out, n1), put(out, st1);
    return st;
  };
  const Call static_call = [&](std::vector<double>& out) {
    std::vector<cd> a(1), n1(nb);
    const int st = sigma_gpp_achstemp(nb, nc, ng, inv.data(), ind.data(), am.data(), an.data(), ie.data(), v.data(),
                                      a.data(), n1.data(), SIGMA_FF_FP64, nullptr);
    out.clear();
    put(out, a), put(out, n1);
    return st;
  };
  const int ne = 5;
  auto er = cplx((size_t)nf * ngf * nc), ea = cplx((size_t)nf * ngf * nc), brd = cplx(nf, 0, 0, 0.1, 0.2);
  const Call ff_call = [&](std::vector<double>& out) {
    std::vector<cd> s((size_t)nb * nf);
    const int st = sigma_ff_schdt(nb, nc, ngf, nf, iota.data(), iota.data(), er.data(), an.data(), am.data(), s.data(),
                                  SIGMA_FF_FP64, nullptr);
    out.clear();
    put(out, s);
    return st;
  };
  std::vector<double> ekq(nb), grid = {0, 1, 2.5, 4}, pref(nf, 0.3);  // nf = 4
  for (int n = 0; n < nb; ++n) ekq[n] = -3.0 + 0.1 * n;
  const Call loop_call = [&](std::vector<double>& out) {
    std::vector<cd> a0(1), a1(ne), a2(ne), a3(ne), a4(ne), a5(ne);
    const int st = sigma_ff_sigma(nb, nvb, nc, ngf, nf, ne, iota.data(), iota.data(), am.data(), an.data(), er.data(),
                                  ea.data(), v.data(), ekq.data(), grid.data(), brd.data(), pref.data(), 0.16, 0.0, 0.5,
                                  1.0, nullptr, a0.data(), a1.data(), a2.data(), a3.data(), a4.data(), a5.data(),
                                  SIGMA_FF_FP64, nullptr);
    out.clear();
    put(out, a0), put(out, a1), put(out, a2), put(out, a3), put(out, a4), put(out, a5);
    return st;
  };
  const std::vector<std::pair<std::string, const Call*>> calls = {
      {"GPP", &gpp_call}, {"real GPP", &real_call}, {"half sum", &half_call}, {"static remainder", &static_call},
      {"FF", &ff_call},   {"FF band loop", &loop_call}};
  for (const auto& c : calls) check(c.first, *c.second);
  // one operand element 2^40 above its row
  const double up = 0x1p40;
  auto outlier = [&](cd& x, std::initializer_list<int> which, const char* what, Range range = kOutside) {
    const cd keep = x;
    x = cd{keep.re * up, keep.im * up};
    for (int i : which) check(calls[i].first + ", " + what, *calls[i].second, range);
    x = keep;
  };
  outlier(an[(size_t)17 * nc + 33], {0, 2, 3, 4, 5}, "outlier in aqsn");
  outlier(am[(size_t)1 * nc + 34], {2}, "outlier in an occupied band's aqsm");
  outlier(ie[(size_t)150 * nc + 35], {0, 3}, "outlier in I_eps");
  outlier(ie[(size_t)150 * nc + 35], {2}, "outlier in I_eps", kPartly);  // every band is large beside it
  outlier(er[(size_t)100 * nc + 36], {4, 5}, "outlier in I_epsR");
  outlier(ea[(size_t)100 * nc + 36], {5}, "outlier in I_epsA", kPartly);
  for (double* x : {&rn[(size_t)17 * nc + 33], &rn[(size_t)1 * nc + 33], &re[(size_t)150 * nc + 35]}) {
    const double keep = *x;
    *x *= up;
    check("real GPP, outlier", real_call, kOutside);
    *x = keep;
  }
  // a plan cache left by one call gives way to another call's inputs
  {
    sigma_shutdown();
    g_budget = ~size_t(0) / 4;
    std::vector<cd> ach(3), asx(3), s((size_t)nb * nf);
    auto gpp = [&] {
      return sigma_gpp_fp64(nb, nvb, nc, ng, 0, 3, inv.data(), ind.data(), wx.data(), 1.0, am.data(), an.data(),
                            ie.data(), wt.data(), v.data(), ach.data(), asx.data(), nullptr, nullptr);
    };
    int st = gpp();
    const size_t kept = g_used;
    g_budget = kept + (8u << 20);  // less than the FF call's inputs
    st = st ? st
            : sigma_ff_schdt(nb, nc, ngf, nf, iota.data(), iota.data(), er.data(), an.data(), am.data(), s.data(),
                             SIGMA_FF_FP64, nullptr);
    if (st != 0) g_bad++, printf("FF after GPP: status %d\n", st);
    const cd before = ach[0];
    st = gpp();
    if (st != 0 || std::hypot(ach[0].re - before.re, ach[0].im - before.im) > 1e-12 * std::hypot(before.re, before.im))
      g_bad++, printf("GPP after FF: status %d\n", st);
  }
  sigma_shutdown();
}

int main() {
  // nothing divides; workspaces up to 326 MB, some kept between calls, and from 300 MB on
  g_kept = true;
  all_calls(71, 3, 4099, 203, 4, 57);
  g_kept = false;
  all_calls(71, 3, 8209, 801, 4, 401);
  printf("%d bad\n", g_bad);
  return g_bad != 0;
}
