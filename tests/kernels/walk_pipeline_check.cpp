// The cooperative walk's pipeline (walk_records_in_order, walk.cuh) on the host, its warps in
// adversarial orders, against the reference's recurrence run serially
// (culbfgsb/lbfgsbcpu.cpp:725-809).  Every result must be equal bit for bit, every block barrier
// reached by all threads alike.
//   walk_pipeline_check {f64|f32} {stop|end|bounded|fixed|limit|nohist|chunks}
#include <type_traits>
#include <vector>

#include "small.cuh"
#include "state.cuh"

namespace lbfgsb_b200 {
struct WalkScratch {
  unsigned int words[64];
};
template <typename R, typename H, typename S>
struct Ctx {
  DevState<S>* st;
  int8_t* code;
  int n;
};
inline uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
template <typename S>
void lds4(uint32_t at, S (&v)[4]) {
  memcpy(v, emu::shared_base + at, sizeof(v));
}
template <typename S>
void sts4(uint32_t at, const S (&v)[4]) {
  memcpy(const_cast<char*>(emu::shared_base) + at, v, sizeof(v));
}
}  // namespace lbfgsb_b200
#include "walk_slice.cuh"

using namespace lbfgsb_b200;

static uint64_t g_rng;
static double uniform() {  // [0, 1), a 64-bit linear congruential generator's upper bits
  g_rng = g_rng * 6364136223846793005ull + 1442695040888963407ull;
  return (double)(g_rng >> 11) * 0x1p-53;
}

struct Setup {
  int cnt, chunks, col, stop;  // keys a chunk; stop: the key that is not passed, -1: none
  bool bounded, fixed, limit;
  int late;
};

template <typename S>
struct Walk {
  std::vector<S> t, dibp, zibp, wmw, e, v;
  S f1, f2, f2org, theta;
};

template <typename S>
static Walk<S> make(const Setup& u, uint64_t seed) {
  g_rng = seed;
  const int n = u.cnt * u.chunks;
  Walk<S> w;
  w.t.resize(n), w.dibp.resize(n), w.zibp.resize(n), w.wmw.resize(n);
  w.e.assign((size_t)n * kRow, S(0)), w.v.assign((size_t)n * kRow, S(0));
  double t = 0;
  w.theta = (S)1.7;
  for (int k = 0; k < n; k++) {
    t += k == u.stop ? 1e6 : 1e-4 * (0.5 + uniform());
    w.t[k] = (S)t;
    w.dibp[k] = (S)((uniform() < 0.5 ? -1 : 1) * (0.01 + 0.05 * uniform()));
    w.zibp[k] = w.dibp[k] * w.t[k];
    w.wmw[k] = (S)(0.2 * uniform());
    for (int j = 0; j < 2 * u.col; j++) {
      const S wbp = (S)(uniform() - 0.5);
      w.e[(size_t)k * kRow + j] = (-w.dibp[k]) * wbp;
      w.v[(size_t)k * kRow + j] = (S)(0.01 * (uniform() - 0.5));
    }
  }
  w.f1 = (S)-5e4;  // the minimum of the piece lies beyond every breakpoint
  w.f2 = (S)9;
  // limit: f'' reaches its lower limit, 8.97, within the first keys and often afterwards
  w.f2org = u.limit ? (S)(8.97 / 5e-16) : (S)9;
  return w;
}

template <typename S>
struct Result {
  S f1, f2, dtm, tsum, tj, p[kRow], c[kRow];
  int nleft, nint, all_fixed, done;
  std::vector<int8_t> code;
};

template <typename S>
static void start_p(S* p, S* c, int col2) {
  for (int j = 0; j < col2; j++) {
    p[j] = (S)(0.3 * (j + 1) * ((j & 1) ? -1 : 1));
    c[j] = (S)(0.01 * j);
  }
}

// lbfgsbcpu.cpp:725-809, one key at a time
template <typename S>
static Result<S> serial(const Setup& u, const Walk<S>& w) {
  Result<S> r{};
  const int n = (int)w.t.size(), col2 = 2 * u.col, nbreak = n;
  const int nvar = u.fixed ? n : n + 3;
  r.code.assign(nvar, 0);
  start_p(r.p, r.c, col2);
  r.f1 = w.f1, r.f2 = w.f2, r.dtm = -w.f1 / w.f2;
  r.nleft = nbreak, r.nint = 1;
  for (int k = 0; k < n; k++) {
    const S tj0 = r.tj;
    r.tj = w.t[k];
    const S dt = r.tj - tj0;
    if (r.dtm < dt) {
      r.done = 1;
      break;
    }
    r.tsum = r.tsum + dt;
    r.nleft--;
    const S dibp = w.dibp[k];
    r.code[k] = dibp > S(0) ? IW_WALK_UPP : IW_WALK_LOW;
    if (r.nleft == 0 && nbreak == nvar) {
      r.dtm = dt;
      for (int j = 0; j < col2; j++) r.c[j] += r.dtm * r.p[j];
      r.all_fixed = 1;
      r.done = 1;
      break;
    }
    r.nint++;
    const S dibp2 = dibp * dibp;
    r.f1 = r.f1 + dt * r.f2 + dibp2 - w.theta * dibp * w.zibp[k];
    r.f2 = r.f2 - w.theta * dibp2;
    if (u.col > 0) {
      const S* v = &w.v[(size_t)k * kRow];
      for (int j = 0; j < col2; j++) r.c[j] += dt * r.p[j];
      const S wmc = sdot(r.c, 1, v, 1, col2), wmp = sdot(r.p, 1, v, 1, col2);
      for (int j = 0; j < col2; j++) r.p[j] += w.e[(size_t)k * kRow + j];
      r.f1 = r.f1 + dibp * wmc;
      r.f2 = r.f2 + (S)2.0 * dibp * wmp - dibp2 * w.wmw[k];
    }
    r.f2 = smax((S)(5e-16 * (double)w.f2org), r.f2);
    if (r.nleft > 0) {
      r.dtm = -r.f1 / r.f2;
      continue;
    }
    if (u.bounded)
      r.f1 = r.f2 = r.dtm = 0;
    else
      r.dtm = -r.f1 / r.f2;
    r.done = 1;
  }
  return r;
}

template <typename S>
static bool pipeline(const Setup& u, const Walk<S>& w, Result<S>& r) {
  const int n = (int)w.t.size(), col2 = 2 * u.col, nvar = u.fixed ? n : n + 3;
  static DevState<S> st;
  static WalkCoop<S> sm;
  memset(&st, 0, sizeof(st));
  memset(&sm, 0xff, sizeof(sm));  // NaN wherever nothing is written
  st.n = nvar, st.col = u.col, st.nbreak = n, st.bnded = u.bounded ? 1 : 0;
  st.theta = w.theta, st.f2org = w.f2org;
  start_p(st.p + 1, st.c + 1, col2);
  sm.f1 = w.f1, sm.f2 = w.f2, sm.dtm = -w.f1 / w.f2, sm.tsum = 0, sm.tj = 0;
  sm.nleft = n, sm.nint = 1, sm.all_fixed = 0, sm.done = 0;
  r.code.assign(nvar, 0);
  Ctx<S, S, S> c{&st, r.code.data(), nvar};
  emu::shared_base = reinterpret_cast<const char*>(&sm);
  emu::late_warp = u.late;
  bool ok = true;
  for (int h = 0; h < u.chunks && !sm.done && ok; h++) {
    const size_t o = (size_t)h * u.cnt;
    std::vector<unsigned long long> hi(u.cnt);
    std::vector<unsigned int> lo(u.cnt);
    for (int k = 0; k < u.cnt; k++) {
      hi[k] = (unsigned long long)__double_as_longlong((double)w.t[o + k]);
      lo[k] = (unsigned int)(o + k);
    }
    WalkRecords<S> rec{};
    rec.hi = hi.data(), rec.lo = lo.data();
    rec.e = const_cast<S*>(&w.e[o * kRow]), rec.v = const_cast<S*>(&w.v[o * kRow]);
    rec.dibp = const_cast<S*>(&w.dibp[o]), rec.zibp = const_cast<S*>(&w.zibp[o]);
    rec.wmw = const_cast<S*>(&w.wmw[o]);
    ok = emu::run_block(kWalkThreads, 0, 1, [&] { walk_records_in_order<S, S, S>(c, rec, u.cnt, sm); });
  }
  r.f1 = sm.f1, r.f2 = sm.f2, r.dtm = sm.dtm, r.tsum = sm.tsum, r.tj = sm.tj;
  r.nleft = sm.nleft, r.nint = sm.nint, r.all_fixed = sm.all_fixed, r.done = sm.done ? 1 : 0;
  memcpy(r.p, st.p + 1, sizeof(r.p));
  memcpy(r.c, st.c + 1, sizeof(r.c));
  return ok;
}

template <typename S>
static int check(Setup u, const char* what) {
  const Walk<S> w = make<S>(u, 12345u + (unsigned)u.cnt);
  const Result<S> a = serial<S>(u, w);
  Result<S> b{};
  const bool ok = pipeline<S>(u, w, b);
  const int col2 = 2 * u.col;
  auto differ = [&](const char* name, double x, double y) {
    if (memcmp(&x, &y, 8) == 0) return 0;
    fprintf(stderr, "%s cnt %d stop %d late %d: %s %.17g, serially %.17g\n", what, u.cnt, u.stop, u.late, name, y, x);
    return 1;
  };
  int bad = ok ? 0 : 1;
  if (!ok) fprintf(stderr, "%s cnt %d stop %d late %d: barriers\n", what, u.cnt, u.stop, u.late);
  bad += differ("f1", a.f1, b.f1) + differ("f2", a.f2, b.f2) + differ("dtm", a.dtm, b.dtm);
  bad += differ("tsum", a.tsum, b.tsum) + differ("tj", a.tj, b.tj);
  bad += differ("nleft", a.nleft, b.nleft) + differ("nint", a.nint, b.nint);
  bad += differ("all_fixed", a.all_fixed, b.all_fixed) + differ("done", a.done, b.done);
  for (int j = 0; j < col2; j++) bad += differ("p", a.p[j], b.p[j]) + differ("c", a.c[j], b.c[j]);
  if (a.code != b.code) bad += differ("code", 0, 1);
  return bad;
}

template <typename S>
static int run(const char* what) {
  int bad = 0, ran = 0;
  auto go = [&](Setup u) {
    bad += check<S>(u, what);
    ran++;
  };
  const auto is = [&](const char* s) { return strcmp(what, s) == 0; };
  for (int late : {-1, 0, 1, 2, 3, 4, 7, 8, 15}) {
    if (is("stop"))  // in the first, a middle and the last sub-batch, at their edges
      for (int stop : {0, 1, 127, 128, 300, 511, 512, 640, 699}) go({700, 1, 4, stop, false, false, false, late});
    if (is("end"))
      for (int cnt : {1, 2, 127, 128, 129, 700}) go({cnt, 1, 8, -1, false, false, false, late});
    if (is("bounded"))
      for (int cnt : {1, 128, 300}) go({cnt, 1, 3, -1, true, false, false, late});
    if (is("fixed"))
      for (int cnt : {1, 2, 128, 129, 300}) go({cnt, 1, 3, -1, true, true, false, late});
    if (is("limit"))
      for (int stop : {-1, 1, 60, 127, 128, 129, 290}) go({300, 1, 2, stop, false, false, true, late});
    if (is("nohist"))
      for (int stop : {-1, 0, 130}) go({260, 1, 0, stop, false, false, stop < 0, late});
    if (is("chunks"))
      for (int stop : {-1, 140, 150, 449}) go({150, 3, 5, stop, false, false, stop == 449, late});
  }
  return bad != 0 || ran == 0;
}

int main(int argc, char** argv) {
  if (argc != 3) return 2;
  return strcmp(argv[1], "f32") == 0 ? run<float>(argv[2]) : run<double>(argv[2]);
}
