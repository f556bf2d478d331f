// Checks of the library's host code on a fake CUDA runtime (fake_cudart.hpp):
// `host_check NAME` runs one, prints what is wrong and exits non-zero then. Built and
// run by tests/test_host_calls.py.
#include <cerrno>
#include <chrono>
#include <cstdio>
#include <cstring>
#include <future>
#include <string>
#include <thread>
#include <vector>

#include <dlfcn.h>
#include <pthread.h>
#include <sys/mman.h>
#include <sys/wait.h>
#include <unistd.h>

#include "../../include/optx.h"
#include "fake_cudart.hpp"

namespace {

bool threads_fail = false;  // pthread_create (below) refuses

int bad = 0;
void expect(bool ok, const std::string& what) {
  if (ok) return;
  std::printf("%s (%s)\n", what.c_str(), optx_last_error());
  ++bad;
}

optx_params cube() {
  optx_params p{};
  p.hx = p.hy = p.hz = 25.0f;
  p.n_scint = 1.63f;
  p.n_det = 1.5f;
  p.n_out = 1.0f;
  p.abs_length = 2000.0f;
  p.scat_length = 500.0f;
  p.tau = 4.0f;
  p.max_steps = 10000;
  p.seed = 12345;
  return p;
}

struct Records {
  std::vector<uint8_t> fate;
  std::vector<uint32_t> nb, ns;
  std::vector<float> t, x, y, z, path;
  explicit Records(uint64_t n) : fate(n), nb(n), ns(n), t(n), x(n), y(n), z(n), path(n) {}
  optx_records c() { return {fate.data(), nb.data(), ns.data(), t.data(), x.data(), y.data(), z.data(), path.data()}; }
  bool right(uint64_t first_id) const {
    for (uint64_t i = 0; i < fate.size(); ++i) {
      const uint64_t id = first_id + i;
      const float f = static_cast<float>(fake::word(id) >> 8);
      if (fate[i] != fake::fate(id) || nb[i] != fake::word(id) || ns[i] != fake::word(id + 1) || t[i] != f ||
          x[i] != static_cast<float>((fake::word(id) >> 8) + 1) || path[i] != static_cast<float>((fake::word(id) >> 8) + 4))
        return false;
    }
    return true;
  }
};

void records_call(const std::string& what, uint64_t n, uint64_t first_id) {
  const optx_params p = cube();
  Records r(n);
  const optx_records c = r.c();
  expect(optx_run_records(&p, nullptr, n, &c, 256, first_id, 0, OPTX_MATH_FAST, nullptr) == OPTX_OK, what + ": records");
  expect(r.right(first_id), what + ": record values");
}
void event_call(const std::string& what, uint64_t n, uint64_t first_id, uint32_t k = 8) {
  const optx_params p = cube();
  Records r(n);
  const optx_records c = r.c();
  expect(optx_run_records_event(&p, nullptr, n, &c, k, 256, first_id, 0, OPTX_MATH_FAST, nullptr, nullptr) == OPTX_OK,
         what + ": event records");
  expect(r.right(first_id), what + ": event record values");
}
void tally_call(const std::string& what, uint32_t xy, int block = 256) {
  const optx_params p = cube();
  const optx_tally_config c{100, 50.0f, xy};
  std::vector<uint64_t> t(5 + 101 + xy * xy + 2);
  expect(optx_run_tally(&p, nullptr, &c, 1000, t.data(), block, 3, OPTX_MATH_FAST, nullptr) == OPTX_OK, what + ": tally");
  expect(t[0] == 1000, what + ": tally values");
}

// Host calls made with another current device than earlier ones use that device's own
// buffers, streams and events.
void devices() {
  for (int d : {0, 1, 0, 1}) {
    fake::current = d;
    const std::string at = "device " + std::to_string(d);
    records_call(at, 5000, 77);
    event_call(at, 5000, 78);
    tally_call(at, 10);
    tally_call(at + ", wide", 230);
  }
  expect(fake::faults == 0, "launches with another device's memory");
  optx_release_cache();
  expect(fake::device_bytes() == 0, "device memory left after optx_release_cache");
  fake::current = 0;
  records_call("after the release", 5000, 79);
}

// A records call and an event-records call on two threads do not wait for each other.
void overlap() {
  std::promise<void> started, event_done;
  bool waited = false;
  std::future<void> done = event_done.get_future();
  fake::on_shares = [&] {  // the records call's kernel, under way until the event call is through
    fake::on_shares = nullptr;
    started.set_value();
    waited = done.wait_for(std::chrono::seconds(5)) == std::future_status::timeout;
  };
  std::thread records([] { records_call("thread", 1200000, 5); });
  started.get_future().wait();
  event_call("main", 1200000, 9);  // large enough for the copy helpers, which both use
  event_done.set_value();
  records.join();
  expect(!waited, "the event-records call waited for the records call");
  std::thread again([] { records_call("thread", 1200000, 6); });
  event_call("main", 1200000, 10);
  again.join();
}

// An engine that runs in several waves makes one graph, whatever its runs cover, and
// each run is launched with its own parameters.
void graphs() {
  const optx_tally_config tc{100, 50.0f, 10};
  optx_wave_config cfg{};
  cfg.cadence = 8;
  optx_engine* e = nullptr;
  expect(optx_engine_create(&tc, 4, 100000, &cfg, &e) == OPTX_OK, "create");
  std::vector<optx_params> ev(4, cube());
  for (uint32_t i = 0; i < 20; ++i) {
    for (uint32_t k = 0; k < 4; ++k) ev[k].seed = 100 * i + k, ev[k].abs_length = 100.0f + static_cast<float>(i + k);
    const std::vector<uint64_t> counts{100 + i, 7, 0, 1000 - i};
    expect(optx_engine_set_events(e, ev.data(), nullptr, counts.data(), 4, 1000 * i, nullptr) == OPTX_OK, "upload");
    expect(optx_engine_run_tally(e, nullptr) == OPTX_OK, "run");
    const optx::WaveArgs& a = fake::runs.back().args;
    expect(fake::runs.size() == 2 * i + 1 && a.first_id == 1000 * i && a.item_lo == 0 && a.total == 1107 && a.keep_tally == 0,
           "a run's arguments");
    expect(optx_engine_run_tally_range(e, 50, 60 + i, 1, nullptr) == OPTX_OK, "range");
    const optx::WaveArgs& r = fake::runs.back().args;
    expect(r.item_lo == 50 && r.total == 60 + i && r.keep_tally == 1, "a range's arguments");
  }
  expect(fake::instantiations == 1, "graphs of the batch: " + std::to_string(fake::instantiations));
  for (uint32_t i = 0; i < 20; ++i) {  // one configuration: the physics is a parameter too
    optx_params p = cube();
    p.seed = i;
    const uint64_t n = 500 + i;
    expect(optx_engine_set_events(e, &p, nullptr, &n, 1, i, nullptr) == OPTX_OK, "upload");
    expect(optx_engine_run_tally(e, nullptr) == OPTX_OK, "run");
    expect(fake::runs.back().p0.key_lo == i && fake::runs.back().args.total == n, "a run's physics");
  }
  expect(fake::instantiations == 2, "graphs: " + std::to_string(fake::instantiations));
  optx_engine_destroy(e);
}

// What event-records calls of several kinds keep on the device stays bounded.
void kept() {
  constexpr uint64_t n = 2000000;
  for (uint32_t k : {2, 4, 8, 16, 32}) {
    event_call("cadence " + std::to_string(k), n, k, k);
    // 256 MB of queues, the call's 29 bytes per photon, and a few MB of tables
    expect(fake::device_bytes() <= (256ull << 20) + 30 * n + (4ull << 20),
           "device memory kept: " + std::to_string(fake::device_bytes() >> 20) + " MB");
  }
  optx_release_cache();
  expect(fake::device_bytes() == 0, "device memory left after optx_release_cache");
}

// Event-records calls of similar sizes use one kept engine.
void sizes() {
  event_call("first", 130000, 1);
  const int before = fake::mallocs;
  for (uint64_t n : {129999, 120001, 100000, 70007}) event_call("size " + std::to_string(n), n, n);
  expect(fake::mallocs == before, "allocations by calls of other sizes: " + std::to_string(fake::mallocs - before));
}

// Records calls into fresh pages where no thread can be started: as with them, slower.
void threads() {
  constexpr uint64_t n = 1000000;
  threads_fail = true;
  for (bool event : {true, false}) {
    std::vector<void*> a;
    for (int k = 0; k < 8; ++k)
      a.push_back(mmap(nullptr, (k ? 4 : 1) * n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
    const auto f = [&](int k) { return static_cast<float*>(a[static_cast<size_t>(k)]); };
    const optx_records c{static_cast<uint8_t*>(a[0]), static_cast<uint32_t*>(a[1]), static_cast<uint32_t*>(a[2]), f(3), f(4),
                         f(5), f(6), f(7)};
    const optx_params p = cube();
    expect((event ? optx_run_records_event(&p, nullptr, n, &c, 8, 256, 3, 0, OPTX_MATH_FAST, nullptr, nullptr)
                  : optx_run_records(&p, nullptr, n, &c, 256, 3, 0, OPTX_MATH_FAST, nullptr)) == OPTX_OK, "records");
    for (uint64_t i = 0; i < n; ++i)
      if (c.fate[i] != fake::fate(3 + i) || c.n_scatter[i] != fake::word(4 + i)) return expect(false, "record values");
  }
  threads_fail = false;
}

// optx_release_cache in a forked child returns, although the copies' helper threads are
// its parent's.
void forked() {
  records_call("parent", 1200000, 5);
  const pid_t child = fork();
  if (child == 0) {
    alarm(10);
    _exit(optx_release_cache());
  }
  int status = 0;
  waitpid(child, &status, 0);
  expect(WIFEXITED(status) && WEXITSTATUS(status) == 0, "the child's release");
  records_call("parent", 1200000, 6);
  optx_release_cache();
}

// A release whose frees fail (after a device reset) leaves no error behind: launches ask
// for the last one and would report it.
void stale() {
  records_call("before", 5000, 1);
  event_call("before", 5000, 2);
  tally_call("before", 10);
  fake::frees_fail = true;
  expect(optx_release_cache() == OPTX_OK, "release");
  fake::frees_fail = false;
  expect(!fake::stale_error(), "the release left an error");
  records_call("after", 5000, 3);
  event_call("after", 5000, 4);
  tally_call("after", 10);
}

// Host tallies with wide histograms fill the SMs whatever block size is asked for.
void wide_blocks() {
  for (int block : {32, 64, 128, 256, 512, 1024}) {
    tally_call("block " + std::to_string(block), 200, block);
    expect(fake::history_block >= 256 && fake::history_block >= block, "threads: " + std::to_string(fake::history_block));
  }
}

// Which tallies run the history kernel: histograms that do not fit beside 28 warps'
// pantries (100 time bins: from 184 x 184 hit-map bins on), and device calls of more
// photons than the wave kernel's cursors count.
void routes() {
  const optx_params p = cube();
  uint64_t* t = nullptr;
  expect(cudaMalloc(reinterpret_cast<void**>(&t), 8 * 60000) == cudaSuccess, "malloc");
  const auto device = [&](uint32_t xy, uint64_t n) {
    const optx_tally_config c{100, 50.0f, xy};
    fake::history_block = 0;
    t[0] = 0;
    expect(optx_tally_device(&p, nullptr, &c, n, 0, t, 64, OPTX_MATH_FAST, nullptr) == OPTX_OK && t[0] == n, "device tally");
    return fake::history_block == 64;
  };
  for (uint32_t xy : {10, 170, 183, 184, 200, 236}) {
    fake::history_block = 0;
    tally_call(std::to_string(xy) + " bins", xy);
    expect((fake::history_block != 0) == (xy >= 184), "route of the host tally, " + std::to_string(xy));
    expect(device(xy, 1000) == (xy >= 184), "route of the device tally, " + std::to_string(xy));
  }
  expect(!device(10, optx::kSharesMaxPhotons), "route of 2^32 - 65536 photons");
  expect(device(10, optx::kSharesMaxPhotons + 1), "route of 2^32 - 65535 photons");
  cudaFree(t);
}

const struct {
  const char* name;
  void (*run)();
} kChecks[] = {{"devices", devices}, {"overlap", overlap}, {"graphs", graphs}, {"kept", kept}, {"sizes", sizes}, {"threads", threads}, {"forked", forked}, {"stale", stale}, {"wide_blocks", wide_blocks}, {"routes", routes}};

}  // namespace

extern "C" int pthread_create(pthread_t* t, const pthread_attr_t* attr, void* (*run)(void*), void* arg) noexcept {
  static const auto real = reinterpret_cast<decltype(&pthread_create)>(dlsym(RTLD_NEXT, "pthread_create"));
  return threads_fail ? EAGAIN : real(t, attr, run, arg);
}

int main(int argc, char** argv) {
  for (const auto& c : kChecks)
    if (argc == 2 && std::strcmp(argv[1], c.name) == 0) {
      c.run();
      return bad != 0;
    }
  std::printf("usage: host_check NAME\n");
  return 2;
}
