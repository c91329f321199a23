// The team routines of scatter_team_math.cuh on an emulated warp: 32 lanes as
// coroutines that meet at every warp-wide operation, shared memory as a plain
// array with a guard after each team's part.  Compared, bit for bit where the
// caller asks for it, with the per-thread functions they stand for.
#include <ucontext.h>

#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <vector>

#define __device__
#define __forceinline__ inline
struct float4 { float x, y, z, w; };
static inline float4 make_float4(float x, float y, float z, float w) { return {x, y, z, w}; }

namespace warp {
constexpr int N = 32;
ucontext_t main_ctx, ctx[N];
std::vector<char> stack[N];
std::function<void(int)> body;
bool done[N];
int cur;
uint64_t slot[N];       // the values of the operation that the lanes are in
long ops[N];            // operations each lane has met
void yield() { swapcontext(&ctx[cur], &main_ctx); }
void entry() {
  body(cur);
  done[cur] = true;
  swapcontext(&ctx[cur], &main_ctx);
}
// Run the lanes; false if they do not meet at the same operations.
bool run(std::function<void(int)> f) {
  body = f;
  for (int i = 0; i < N; i++) {
    stack[i].resize(1 << 18);
    getcontext(&ctx[i]);
    ctx[i].uc_stack.ss_sp = stack[i].data();
    ctx[i].uc_stack.ss_size = stack[i].size();
    ctx[i].uc_link = &main_ctx;
    makecontext(&ctx[i], entry, 0);
    done[i] = false;
    ops[i] = 0;
  }
  for (;;) {
    int left = 0;
    for (int i = 0; i < N; i++)
      if (!done[i]) {
        cur = i;
        swapcontext(&main_ctx, &ctx[i]);
        left += !done[i];
      }
    for (int i = 1; i < N; i++)
      if (ops[i] != ops[0] || done[i] != done[0]) return false;
    if (!left) return true;
  }
}
template <class T>
T exchange(T v, int from) {
  uint64_t b = 0;
  memcpy(&b, &v, sizeof v);
  slot[cur] = b;
  ops[cur]++;
  yield();               // every lane has written
  const uint64_t r = slot[from & 31];
  ops[cur]++;
  yield();               // every lane has read
  T o;
  memcpy(&o, &r, sizeof o);
  return o;
}
unsigned ballot(bool p) {
  slot[cur] = p;
  ops[cur]++;
  yield();
  unsigned m = 0;
  for (int i = 0; i < N; i++) m |= (unsigned)(slot[i] != 0) << i;
  ops[cur]++;
  yield();
  return m;
}
}  // namespace warp
constexpr unsigned FULL = 0xffffffffu;
template <class T> T __shfl_sync(unsigned, T v, int from) { return warp::exchange(v, from); }
template <class T> T __shfl_xor_sync(unsigned, T v, int o) { return warp::exchange(v, warp::cur ^ o); }
static inline unsigned __ballot_sync(unsigned, bool p) { return warp::ballot(p); }
static inline bool __any_sync(unsigned, bool p) { return warp::ballot(p) != 0; }
static inline void __syncwarp() { warp::ops[warp::cur]++; warp::yield(); }

static inline float __fmul_rn(float a, float b) { return a * b; }
static inline double __dmul_rn(double a, double b) { return a * b; }

#include "scatter_physics.cuh"
#include "scatter_team_math.cuh"

using namespace crtm;

namespace {
constexpr float GUARD = 12345.75f;

template <int NZ, int NM, int NV>
struct Shared {
  static constexpr int TF = team_floats<NZ, NM, NV>(), TPW = 32 / team_size<NZ>();
  std::vector<float> raw;
  float* base;
  Shared() : raw((size_t)TPW * (TF + 4) + 8, GUARD) {
    base = raw.data();
    while ((uintptr_t)base % 16) base++;
  }
  float* team(int t) { return base + (size_t)t * (TF + 4); }
  bool intact() {
    for (int t = 0; t < TPW; t++)
      for (int i = 0; i < 4; i++)
        if (team(t)[TF + i] != GUARD) return false;
    return true;
  }
};

template <int NZ>
Team<NZ> team_of(int lane, int n, int nS, bool live) {
  Team<NZ> t;
  t.lane = lane;
  t.r = lane & (team_size<NZ>() - 1);
  t.base = lane - t.r;
  t.n = n;
  t.nS = nS;
  t.live = live;
  return t;
}

// One warp of matrices: per team its size and rows [n][10].  Returns the number
// of values that differ from the per-thread function's, -1 if the lanes parted,
// -2 if a team wrote past its part.
struct Input {
  int n;
  float m[100];
};

template <int NZ>
long inverse(const Input* L, int teams) {
  Shared<NZ, 3, 0> sh;
  std::vector<Mat<NZ, float>> got(sh.TPW);
  std::vector<int> oks(sh.TPW);
  const bool met = warp::run([&](int lane) {
    const int ti = lane / team_size<NZ>();
    const bool live = ti < teams;
    const Input& y = L[live ? ti : 0];
    Team<NZ> t = team_of<NZ>(lane, y.n, y.n - 1, live);
    const int r = t.row() ? t.r : 0;
    float g[NZ];
    for (int j = 0; j < NZ; j++) g[j] = (t.r == j ? 1.0f : 0.0f) - (j < y.n ? y.m[r * 10 + j] : 0.f);
    float* M = sh.team(ti);
    const bool ok = team_invert_adding<NZ>(t, g, M + 2 * team_mat<NZ>(), reinterpret_cast<double*>(M));
    __syncwarp();
    if (t.row())
      for (int j = 0; j < y.n; j++) got[ti].a[r][j] = M[2 * team_mat<NZ>() + r * team_ld<NZ>() + j];
    if (t.r == 0) oks[ti] = ok;
  });
  if (!met) return -1;
  if (!sh.intact()) return -2;
  long bad = 0;
  for (int ti = 0; ti < teams; ti++) {
    const Input& y = L[ti];
    Mat<NZ, float> G;
    for (int i = 0; i < y.n; i++)
      for (int j = 0; j < y.n; j++) G.a[i][j] = (i == j ? 1.0f : 0.0f) - y.m[i * 10 + j];
    const bool ok = invert_fp64<NZ, float>(y.n, G);
    bad += (int)ok != oks[ti];
    for (int i = 0; i < y.n && ok; i++)
      for (int j = 0; j < y.n; j++) {
        bad += memcmp(&got[ti].a[i][j], &G.a[i][j], 4) != 0 && !(got[ti].a[i][j] == 0.f && G.a[i][j] == 0.f);
      }
  }
  return bad;
}
}  // namespace

extern "C" {
int input_bytes() { return (int)sizeof(Input); }
int teams_per_warp(int NZ) { return NZ == 4 ? 8 : (NZ == 10 ? 2 : 4); }
// the adding's inverse, of I - m
long run_inverse(int NZ, const void* inputs, int teams) {
  const Input* L = (const Input*)inputs;
  switch (NZ) {
    case 4: return inverse<4>(L, teams);
    case 5: return inverse<5>(L, teams);
    case 6: return inverse<6>(L, teams);
    case 10: return inverse<10>(L, teams);
  }
  return -3;
}
}
