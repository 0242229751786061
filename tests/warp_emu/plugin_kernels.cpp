// Runs a plug-in system's two tracking kernels, a path per thread (track_kernel) and a path
// per warp (warp_kernel), on the same paths and compares all they return bit for bit.
// track.inc: frg_track.cu without its kernel launches. Argument: a file with the frg_config.
#include "track.inc"

template <class S> struct Arrays {
  std::vector<cx<double>> starts, finals;
  std::vector<int32_t> codes, work;
  std::vector<frg::Handoff> handoff;
  std::vector<int64_t> list;
  unsigned long long queue = 0, count = 0;
  explicit Arrays(int n)
      : starts(n * (S::NV + S::NP)), finals(n * (S::NV + 2), cx<double>(0.0)), codes(n, -1), work(3 * n, 0), handoff(n),
        list(n, 0) {
    memset((void*)handoff.data(), 0, n * sizeof(frg::Handoff));
  }
};

template <int MODE, typename T, class S>
bool compare(const char* what, int n, const frg_config& cfg) {
  const int np = S::NP;
  std::vector<cx<double>> fpm(np);
  std::vector<cx<float>> fpm_lo(np);
  for (int i = 0; i < np; ++i) {
    fpm[i] = cx<double>(frg_uniform01(5, 1, 2 * i) - 0.5, frg_uniform01(5, 1, 2 * i + 1) - 0.5);
    fpm_lo[i] = cx<float>(fpm[i]);
  }
  const cx<double> gamma(0.6, 0.8);
  const cx<float> gamma_lo(gamma);
  const int64_t task_start[2] = {0, n};
  std::vector<Arrays<S>> got;
  for (int k = 0; k < 2; ++k) {
    got.emplace_back(n);
    Arrays<S>& o = got.back();
    frg::TrackArgs a{};
    a.cfg = cfg;
    a.fpm = fpm.data(); a.gamma = &gamma; a.fpm_lo = fpm_lo.data(); a.gamma_lo = &gamma_lo;
    a.task_start = task_start; a.ntasks = 1; a.npaths = n; a.seed = 9; a.sms = 1;
    a.queue = &o.queue; a.codes = o.codes.data(); a.work = o.work.data(); a.finals = o.finals.data();
    a.handoff = o.handoff.data(); a.handoff_list = o.list.data(); a.handoff_count = &o.count;
    a.starts = o.starts.data();
    emu::launch((n + FRG_TRACK_THREADS - 1) / FRG_TRACK_THREADS, FRG_TRACK_THREADS, 0,
                [&] { frg::plugin_start_kernel<S>(a, o.starts.data()); });
    if (k == 0) emu::launch(1, FRG_TRACK_THREADS, 0, [&] { frg::track_kernel<MODE, T, S>(a); });
    else emu::launch(1, 32 * frg::WARP_PATHS, sizeof(frg::WarpShared<T, S>), [&] { frg::warp_kernel<MODE, T, S>(a); });
  }
  int moved = 0;
  for (int i = 0; i < n; ++i) moved += got[0].work[3 * i + 2] > 0 || got[0].handoff[i].step > 0;
  // -0.0 and 0.0 are the same value; NaN equals NaN
  const auto same = [](const cx<double>& x, const cx<double>& y) {
    return (x.re == y.re || (x.re != x.re && y.re != y.re)) && (x.im == y.im || (x.im != x.im && y.im != y.im));
  };
  bool ok = got[0].codes == got[1].codes && got[0].work == got[1].work && got[0].count == got[1].count;
  for (size_t i = 0; i < got[0].finals.size(); ++i) ok = ok && same(got[0].finals[i], got[1].finals[i]);
  for (int i = 0; i < n; ++i) {
    const frg::Handoff &x = got[0].handoff[i], &y = got[1].handoff[i];
    for (int e = 0; e < S::NV + 2; ++e) ok = ok && same(x.Yc[e], y.Yc[e]) && same(x.Vc[e], y.Vc[e]);
    ok = ok && x.s == y.s && x.step == y.step && x.n_ivp == y.n_ivp && x.n_newton == y.n_newton && x.reason == y.reason;
  }
  printf("%s: %d of %d paths took steps, %s\n", what, moved, n, ok ? "equal" : "different");
  return ok && moved > 0;
}

int main(int argc, char** argv) {
  frg_config cfg;
  FILE* f = argc > 1 ? fopen(argv[1], "rb") : nullptr;
  if (!f || fread(&cfg, sizeof(cfg), 1, f) != 1) return 2;
  typedef frg::EMU_SYSTEM S;  // the generated struct's name
  const bool a = compare<frg::MODE_PLAIN, double, S>("FP64", 5, cfg);
  cfg.cond_switch = 1e30;
  const bool b = compare<frg::MODE_LO, float, S>("FP32 stage", 5, cfg);
  return a && b ? 0 : 1;
}
