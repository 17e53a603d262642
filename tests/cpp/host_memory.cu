// host_memory.cu -- the library's host side when device memory runs short, on the CPU
// (fake_cudart.cpp in place of the runtime).  Argument: the scenario.  Prints what the
// Python side checks, as key value lines.
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <random>
#include <thread>
#include <vector>

#include "cav_common.cuh"
#include "fake_cudart.h"

namespace {

struct Md {
  cavgpu_ctx *c = nullptr;
  int rc = 0;
  explicit Md(int n, int capacity = 0, double edge = 12.0) {
    cavgpu_params p;
    cavgpu_default_params(&p);
    for (int a = 0; a < 3; ++a) p.hi[a] = edge;
    p.nbr_capacity = capacity;
    std::mt19937 g(1);
    std::uniform_real_distribution<double> u(0.0, edge);
    std::vector<double> x(3 * n);
    for (double &v : x) v = u(g);
    std::vector<uint64_t> t(n, 0);
    rc = cavgpu_create(&p, &c);
    if (!rc) rc = cavgpu_upload(c, n, x.data(), nullptr, t.data(), nullptr);
    if (!rc) rc = cavgpu_setup(c);
  }
  ~Md() { cavgpu_destroy(c); }
};

void say(const char *key, long long v) { std::printf("%s %lld\n", key, v); }

bool is_chunk(const std::string &name) { return name.find("k_chunk") != std::string::npos; }
// first member of the step kernel's argument
cav::Dev &dev_of(void **args) { return *static_cast<cav::Dev *>(args[0]); }

// the list of the first chunk overflows; what happens then is up to the memory limit
int overflow(size_t room) {
  Md m(500, 64);
  say("setup", m.rc);
  int chunks = 0, nulls = 0;
  bool fired = false;
  fake::on_launch = [&](const std::string &name, void **args) {
    if (!is_chunk(name)) return;
    cav::Dev &d = dev_of(args);
    ++chunks;
    if (!d.recv || !d.hw) ++nulls;
    if (!fired) {
      fired = true;
      d.flags[cav::F_HALT] = 1;
      d.flags[cav::F_OVERFLOW] = 200;
      d.flags[cav::F_HALT_STEP] = 3;
      fake::limit = fake::used + room;
    }
  };
  say("run", cavgpu_run(m.c, 400, 0, nullptr));
  int64_t st[8];
  cavgpu_stats(m.c, st);
  say("steps", st[0]);
  say("capacity", st[3]);
  say("chunks", chunks);
  say("nulls", nulls);
  say("graphs", st[6]);
  fake::on_launch = nullptr;
  return 0;
}

int run_all(Md &m, int *nulls) {
  fake::on_launch = [=](const std::string &name, void **args) {
    if (is_chunk(name) && !dev_of(args).recv) ++*nulls;
  };
  const int rc = cavgpu_run(m.c, 200, 0, nullptr);
  fake::on_launch = nullptr;
  return rc;
}

// a context is created where only the exchange arrays of another one leave room for it
int second_context() {
  Md a(500, 64);
  int nulls = 0;
  say("setup", a.rc);
  say("run", run_all(a, &nulls));
  say("exchange_before", cavgpu_pair_exchange(a.c));
  fake::limit = fake::used + (200 << 10);
  {
    Md b(500, 64);
    say("second_setup", b.rc);
    say("second_run", run_all(b, &nulls));
    say("exchange_after", cavgpu_pair_exchange(a.c));
    say("run_again", run_all(a, &nulls));
  }
  fake::limit = (size_t)-1;
  say("run_last", run_all(a, &nulls));
  say("nulls", nulls);
  return 0;
}

// the same while a call on another thread holds the first context: it keeps its arrays
int busy_context() {
  Md a(500, 64);
  say("setup", a.rc);
  fake::limit = fake::used + (200 << 10);
  int second = 1, nulls = 0, chunks = 0;
  fake::on_launch = [&](const std::string &name, void **args) {
    if (!is_chunk(name)) return;
    if (!dev_of(args).recv) ++nulls;
    if (++chunks != 1) return;
    std::thread t([&] { Md b(500, 64); second = b.rc; });
    t.join();
  };
  say("run", cavgpu_run(a.c, 200, 0, nullptr));
  fake::on_launch = nullptr;
  say("second_setup", second);
  say("exchange", cavgpu_pair_exchange(a.c));
  say("nulls", nulls);
  return 0;
}

// the autotuner's snapshot fits once the context's own arrays are given back
int autotune() {
  Md a(4000, 128, 20.0);
  say("setup", a.rc);
  say("exchange_before", cavgpu_pair_exchange(a.c));
  fake::limit = fake::used + (100 << 10);
  say("autotune", cavgpu_autotune(a.c, 4, 0, nullptr));
  int nulls = 0;
  say("run", run_all(a, &nulls));
  say("nulls", nulls);
  return 0;
}

// a barrier of the step kernel gives up
int stall() {
  Md m(500, 64);
  say("setup", m.rc);
  fake::on_launch = [&](const std::string &name, void **args) {
    if (is_chunk(name)) dev_of(args).flags[cav::F_STALL] = 1;
  };
  say("run", cavgpu_run(m.c, 200, 0, nullptr));
  fake::on_launch = nullptr;
  std::vector<double> a(1500);
  int64_t st[8];
  say("run_again", cavgpu_run(m.c, 1, 0, nullptr));
  say("forces", cavgpu_forces(m.c, nullptr, nullptr));
  say("thermo", cavgpu_thermo(m.c, a.data()));
  say("download", cavgpu_download(m.c, a.data(), nullptr, nullptr));
  say("setup_again", cavgpu_setup(m.c));
  say("autotune", cavgpu_autotune(m.c, 0, 0, nullptr));
  say("pairs", cavgpu_export_pairs(m.c, nullptr, 0));
  say("named", std::strstr(cavgpu_last_cuda_error(), "barrier") != nullptr);
  say("stats", cavgpu_stats(m.c, st));
  Md n(500, 64);
  say("other", n.rc ? n.rc : cavgpu_run(n.c, 10, 0, nullptr));
  return 0;
}

// the largest step-kernel grid of a run
unsigned chunk_grid(cavgpu_ctx *c) {
  unsigned g = 0;
  fake::on_launch = [&](const std::string &name, void **) {
    if (is_chunk(name)) g = std::max(g, fake::grid);
  };
  cavgpu_run(c, 100, 0, nullptr);
  fake::on_launch = nullptr;
  return g;
}

// contexts on two devices of different sizes
int devices() {
  fake::sms[1] = 10;
  Md a(4000, 128, 20.0);
  say("first", chunk_grid(a.c));
  fake::device = 1;
  Md b(4000, 128, 20.0);
  say("second", chunk_grid(b.c));
  fake::device = 0;
  say("first_again", chunk_grid(a.c));
  return 0;
}

// what a context that only evaluates forces pins
int pinned() {
  Md m(500, 64);
  say("forces", cavgpu_forces(m.c, nullptr, nullptr));
  say("before", fake::pinned);
  say("run", cavgpu_run(m.c, 10, 0, nullptr));
  say("after", fake::pinned);
  return 0;
}

}  // namespace

int main(int argc, char **argv) {
  const std::string what = argc > 1 ? argv[1] : "";
  // 500 atoms, capacity 64 -> 320: list 0.13 -> 0.64 MB; exchange arrays 1.3 -> 3.2 MB
  if (what == "exchange_lost") return overflow(1 << 20);
  // no room for the new list beside the exchange arrays
  if (what == "list_grows") return overflow(300 << 10);
  if (what == "second_context") return second_context();
  if (what == "busy_context") return busy_context();
  if (what == "autotune") return autotune();
  if (what == "stall") return stall();
  if (what == "devices") return devices();
  if (what == "pinned") return pinned();
  return 1;
}
