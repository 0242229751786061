// The team kernels' pivot search and dense elimination (frg_team.cuh) on values that need not
// be finite: prints what went wrong, if anything.
#include <string>

#include "frg_team.cuh"

using namespace frg;
using namespace frg::team;

static uint64_t draws = 0;
static double uniform() { return frg_uniform01(3, 7, draws++); }
static std::map<std::pair<std::string, std::string>, int> failures;
static void check(bool ok, const char* what, const char* type, int k) {
  if (!ok && failures[{type, what}]++ == 0) printf("not so: %s (%s, first in case %d)\n", what, type, k);
}
template <typename T> T special(int kind) {
  const T nan = T(NAN);  // x86 and Arm differ in the sign of a NaN from arithmetic
  return kind == 0 ? std::copysign(nan, T(1)) : kind == 1 ? std::copysign(nan, T(-1)) : T(INFINITY);
}

// The row found is unused, and the first of the largest unless there is a NaN.
template <int RP, typename T>
void search(const char* type) {
  constexpr int CL = 32 / RP;
  for (int k = 0; k < 400; ++k) {
    T v[RP];
    bool used[RP];
    int unused = 0;
    for (int r = 0; r < RP; ++r) {
      used[r] = uniform() < (k % 4) * 0.3;
      v[r] = used[r] ? T(-1) : T(floor(4 * uniform()));
      if (!used[r] && uniform() < (k % 5) * 0.25) v[r] = special<T>((int)(2.999 * uniform()));
      unused += !used[r];
    }
    if (!unused) { used[RP - 1] = false; v[RP - 1] = special<T>(k % 3); }
    const int base = (k % CL) * RP;
    unsigned bit[32];
    emu::launch(1, 32, 0, [&] {
      const int lane = threadIdx.x, r = lane % RP;
      bit[lane] = pivot_lane(lane / RP == base / RP ? v[r] : T(-1));
    });
    int want = -1;
    bool nan = false;
    for (int r = 0; r < RP; ++r) {
      if (used[r]) continue;
      nan = nan || v[r] != v[r];
      if (want < 0 || v[r] > v[want]) want = r;
    }
    for (int l = 0; l < 32; ++l) {
      check(bit[l] == bit[0] && __builtin_popcount(bit[0]) == 1, "one lane", type, k);
      const int row = __builtin_ctz(bit[l]) - base;
      check(row >= 0 && row < RP && !used[row], "an unused row", type, k);
      check(nan || row == want, "the first of the largest", type, k);
    }
  }
}

// The elimination stays inside its matrix, and every row becomes a pivot row once.
template <typename T>
void eliminate(const char* type) {
  constexpr int n = 16 * LDU, extra = 17 * 8 + 64;
  for (int k = 0; k < 60; ++k) {
    std::vector<cx<T>> U(n + extra, cx<T>(T(-77)));
    for (int r = 0; r < 16; ++r)
      for (int c = 0; c < 17; ++c) U[r * LDU + c] = cx<T>(T(uniform() - 0.5), T(uniform() - 0.5));
    for (int r = 0; r < 16; ++r)  // rows, columns or single entries that are not finite
      for (int c = 0; c < 17; ++c)
        if (k >= 3 && (k % 4 == 0 ? r < k / 4 : (k % 4 == 1 ? c == k / 4 : uniform() < 0.004 * k)))
          U[r * LDU + c] = cx<T>(special<T>(k % 3), k % 2 ? special<T>(k % 3) : T(1));
    T pn[16];
    cx<T> pv[16];
    bool finite = true;
    emu::launch(1, 32, 0, [&] {
      T pmax = T(0), pmin = T(3.0e38);
      dense_lu(U.data(), pn, pv, (int)threadIdx.x, pmax, pmin);
    });
    for (int i = n; i < n + extra; ++i)
      check(U[i].re == T(-77) && U[i].im == T(0), "no store past the matrix", type, k);
    for (int i = 0; i < 16; ++i) finite = finite && pn[i] - pn[i] == T(0) && pn[i] > T(0);
    if (k < 3) check(finite, "finite pivots", type, k);
  }
}

int main() {
  search<16, float>("FP32"); search<8, float>("FP32");
  search<16, double>("FP64"); search<8, double>("FP64");
  eliminate<float>("FP32");
  eliminate<double>("FP64");
  return !failures.empty();
}
