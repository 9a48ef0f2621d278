// Stands in for the launchers of the cooperative step (sayram_team.h) in a test's process: loaded with
// its symbols global before the library, it is what the library's own calls reach. It refuses launches
// as a device without room for them does, hands them on without any polls for their barriers (the first
// barrier of a team of several blocks gives up), or hands them on as they are.
#include <dlfcn.h>

#include <atomic>
#include <chrono>
#include <thread>

#include "sayram_team.h"

static int g_pass = 0, g_odd = 0, g_give_up = 0, g_calls = 0;
static void* g_lib = nullptr;

// lib: the library's path; the next `pass` launches are handed on, the `odd` after them refused (or, with
// give_up, handed on without polls)
extern "C" int shim_set(const char* lib, int pass, int odd, int give_up) {
  if (!g_lib) g_lib = dlopen(lib, RTLD_LAZY | RTLD_LOCAL);
  g_pass = pass;
  g_odd = odd;
  g_give_up = give_up;
  g_calls = 0;
  return g_lib ? 0 : 1;
}
extern "C" int shim_calls() { return g_calls; }

static std::atomic<int> g_hold{0}, g_held{0}, g_grid{0};
// the next launch waits on the host for ms milliseconds first; shim_held: it is waiting or has waited
extern "C" void shim_hold(int ms) {
  g_held = 0;
  g_hold = ms;
}
extern "C" int shim_held() { return g_held; }
extern "C" int shim_grid() { return g_grid; }  // blocks of the last launch

template <typename F, typename... X>
static cudaError_t on(F* self, sg::TeamArgs ta, const sg::TeamLaunch& l, const X&... x) {
  ++g_calls;
  g_grid = l.grid;
  if (const int ms = g_hold.exchange(0)) {
    g_held = 1;
    std::this_thread::sleep_for(std::chrono::milliseconds(ms));
  }
  if (g_pass > 0) {
    --g_pass;
  } else if (g_odd > 0) {
    --g_odd;
    if (!g_give_up) return cudaErrorCooperativeLaunchTooLarge;
    ta.polls = 0;
  }
  Dl_info info;
  F* f = dladdr(reinterpret_cast<void*>(self), &info) ? reinterpret_cast<F*>(dlsym(g_lib, info.dli_sname)) : nullptr;
  return f && f != self ? f(l, x..., ta) : cudaErrorSymbolNotFound;
}

namespace sg {
#define SHIM(name, T)                                                                                          \
  cudaError_t name(const TeamLaunch& l, const Common& cm, const Geo& geo, const Fields& fl, const Coef<T>& co, \
                   const Kry<T>& kr, const TeamArgs& ta) {                                                     \
    return on(&name, ta, l, cm, geo, fl, co, kr);                                                              \
  }
SHIM(team_launch_f64, double)
SHIM(team_launch_mixed, float)
SHIM(team_launch_dw, float)
}  // namespace sg
