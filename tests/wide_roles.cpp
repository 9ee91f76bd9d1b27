// The roles of tilemega_b200/csrc/wide.cuh (persistent products; the loader of portions' keys and values) on host threads, with
// barriers, copies and products that behave as the device's do: copies land in any order, products run one after the other behind
// their issue. A CTA by itself, and a pair whose first CTA issues for both; blocks of keys and values, some halves not full. Every wait
// of every role is made to give up once; a role that never ends, a product or a copy that is still under way where the CTAs go, a
// product on a stage that does not hold its chunk, or a tile written from sums that are not its own ends the program with a message.
#include <unistd.h>

#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <deque>
#include <functional>
#include <mutex>
#include <optional>
#include <random>
#include <thread>
#include <vector>

#include "wide.cuh"

namespace {

constexpr int S = 3, kWarps = 8, kTiles = 7, kStep = 2, kChunks = 4, kBytes = 100;

[[noreturn]] void fail(const char* what, int role, int wait) {
  std::printf("%s (role %d, wait %d)\n", what, role, wait);
  std::fflush(stdout);
  _exit(1);
}

struct Sim {
  std::mutex m;
  std::condition_variable changed;
  std::mt19937 random;
  bool failed = false, stop = false;
  int fail_role, fail_wait, copies = 0, products = 0;
  std::deque<std::function<void()>> queue;                       // products and commits, in order
  std::vector<std::function<void()>> copying;                    // in any order
  std::vector<std::thread> engines;

  struct Bar {
    int count = 1, pending = 1, tx = 0;
    unsigned phase = 0;
    void settle() {
      if (pending == 0 && tx == 0) ++phase, pending = count;
    }
    void arrive(int bytes = 0) { --pending, tx += bytes, settle(); }
    void landed(int bytes) { tx -= bytes, settle(); }
    bool complete(uint32_t parity) const { return (phase & 1u) != parity; }
  };
  struct Stage {
    int tile = -1, chunk = -1;
  };
  struct Sum {
    int tile = -1, chunks = 0;
  };

  Sim(int role, int wait, unsigned seed) : random(seed), fail_role(role), fail_wait(wait) {
    auto engine = [this](bool ordered) {
      std::unique_lock<std::mutex> lock(m);
      for (;;) {
        changed.wait(lock, [&] { return stop || !(ordered ? queue.empty() : copying.empty()); });
        if (ordered ? queue.empty() : copying.empty()) return;
        const unsigned pause = random() % 60;
        lock.unlock();
        std::this_thread::sleep_for(std::chrono::microseconds(pause));
        lock.lock();
        std::function<void()> next;
        if (ordered) {
          next = queue.front();
          queue.pop_front();
        } else {
          const size_t at = random() % copying.size();
          next = copying[at];
          copying.erase(copying.begin() + long(at));
        }
        next();
        changed.notify_all();
      }
    };
    engines.emplace_back(engine, true);
    engines.emplace_back(engine, false);
  }
  ~Sim() {
    {
      std::lock_guard<std::mutex> lock(m);
      stop = true;
    }
    changed.notify_all();
    for (auto& t : engines) t.join();
  }

  // A wait that gives up when it is told to, or, if what it waits for stays away, because another one has.
  bool wait(const Bar& bar, uint32_t parity, int role, int& waits) {
    std::unique_lock<std::mutex> lock(m);
    if (role == fail_role && waits++ == fail_wait) {
      failed = true;
      changed.notify_all();
      return false;
    }
    for (;;) {
      changed.wait(lock, [&] { return bar.complete(parity) || failed; });
      if (bar.complete(parity)) return true;
      if (changed.wait_for(lock, std::chrono::microseconds(random() % 300), [&] { return bar.complete(parity); })) return true;
      return false;
    }
  }
};

// A CTA by itself, or one of a pair (`first` is the one that issues, on whose barriers the copies of both count). Roles: 0 loader,
// 1 issuer, 2 .. writers; of the second CTA of a pair 20 and 22 ...
struct Cta {
  Sim& sim;
  Cta* first;
  Cta* second = nullptr;
  Sim::Bar full[S], empty[S], sum_full[2], sum_empty[2];
  Sim::Stage weights[S], rows[S];
  Sim::Sum sums[2];
  tmb::Filled filled{};
  int met = 0, generation = 0, written[kTiles][kWarps] = {};
  std::condition_variable meeting;

  Cta(Sim& s, Cta* lead) : sim(s), first(lead ? lead : this) {
    if (lead) lead->second = this;
    for (auto* cta : {this, first})
      for (auto& bar : cta->sum_empty) bar.count = bar.pending = lead ? 2 * kWarps : kWarps;
  }
  int role(int of) const { return first == this ? of : 20 + of; }
  int shares() const { return first->second ? 2 : 1; }
  void each(const std::function<void(Cta&)>& f) {
    f(*first);
    if (first->second) f(*first->second);
  }
  void landed(int s, uint32_t parity) {
    std::unique_lock<std::mutex> lock(sim.m);
    if (!sim.changed.wait_for(lock, std::chrono::seconds(2), [&] { return full[s].complete(parity); }))
      fail("copies that never count as landed", sim.fail_role, sim.fail_wait);
  }
  void load() {
    int tile = -1, waits = 0;
    bool there = false;
    auto copy = [&](Sim::Stage* stage, int chunk, int s) {
      const Sim::Stage is{tile, chunk};
      ++sim.copies;
      sim.copying.push_back([=, this] {
        *stage = is;
        first->full[s].landed(kBytes);
        --sim.copies;
      });
      sim.changed.notify_all();
    };
    filled = tmb::fill_stages<S>(
        1, kStep, kTiles, kChunks, [&](int i) { tile = i; },
        [&](int chunk, int s) {
          std::lock_guard<std::mutex> lock(sim.m);
          if (first == this) full[s].arrive(2 * kBytes * shares());
          copy(&weights[s], chunk, s);
        },
        [&] { there = true; },
        [&](int chunk, int s) {
          std::lock_guard<std::mutex> lock(sim.m);
          if (!there) fail("rows before the kernel in front is done", 0, waits);
          copy(&rows[s], chunk, s);
        },
        [&](int s, uint32_t parity) { return sim.wait(empty[s], parity, role(0), waits); });
    if (shares() == 1 && !filled.ok) tmb::drain_stages<S>(filled.chunks, [&](int s, uint32_t parity) { landed(s, parity); });
  }
  // (of a pair's first CTA, behind the end of both)
  void drain() {
    if (filled.ok && second->filled.ok) return;
    auto at = [&](int s, auto what) {
      std::lock_guard<std::mutex> lock(sim.m);
      what(full[s]);
    };
    tmb::drain_pair<S>(
        filled.chunks, second->filled.chunks, [&](int s) { at(s, [](Sim::Bar& bar) { bar.landed(2 * kBytes); }); },
        [&](int s) { at(s, [](Sim::Bar& bar) { bar.arrive(2 * kBytes); }); }, [&](int s, uint32_t parity) { landed(s, parity); });
  }
  void multiply() {
    int waits = 0, tile = -1, sum = 0;
    tmb::multiply_tiles<S>(
        1, kStep, kTiles, kChunks,
        [&](int i, int k) {
          tile = i;
          sum = k & 1;
        },
        [&](int b, uint32_t parity) { return sim.wait(sum_empty[b], parity, 1, waits); },
        [&](int s, uint32_t parity) { return sim.wait(full[s], parity, 1, waits); },
        [&](int chunk, int s) {
          std::lock_guard<std::mutex> lock(sim.m);
          ++sim.products;
          sim.queue.push_back([=, this] {
            each([&](Cta& cta) {
              for (const Sim::Stage* held : {&cta.weights[s], &cta.rows[s]})
                if (held->tile != tile || held->chunk != chunk) fail("a product on another chunk's stage", sim.fail_role, sim.fail_wait);
              if (chunk == 0) cta.sums[sum] = {tile, 0};
              cta.sums[sum].chunks += cta.sums[sum].tile == tile;
              cta.empty[s].arrive();
            });
            --sim.products;
          });
          sim.changed.notify_all();
        },
        [&](int b) {
          std::lock_guard<std::mutex> lock(sim.m);
          sim.queue.push_back([=, this] { each([&](Cta& cta) { cta.sum_full[b].arrive(); }); });
          sim.changed.notify_all();
        },
        [&](int b, uint32_t parity) {
          std::unique_lock<std::mutex> lock(sim.m);
          if (!sim.changed.wait_for(lock, std::chrono::seconds(2), [&] { return sum_full[b].complete(parity); }))
            fail("a wait for products that nobody commits", sim.fail_role, sim.fail_wait);
        });
  }
  void write(int warp) {
    int waits = 0;
    tmb::write_tiles(
        1, kStep, kTiles,
        [&](int, int) {
          std::unique_lock<std::mutex> lock(sim.m);       // a named barrier: it waits for as long as it takes
          const int mine = generation;
          if (++met == kWarps) {
            met = 0;
            ++generation;
            meeting.notify_all();
          } else {
            meeting.wait(lock, [&] { return generation != mine; });
          }
        },
        [&](int b, uint32_t parity) { return sim.wait(sum_full[b], parity, role(2 + warp), waits); },
        [&](int i, int k, bool last) {
          std::lock_guard<std::mutex> lock(sim.m);
          if (!sim.failed && (sums[k & 1].tile != i || sums[k & 1].chunks != kChunks)) fail("a tile from other sums", sim.fail_role, sim.fail_wait);
          if (last != (i + kStep >= kTiles)) fail("not the last tile", sim.fail_role, sim.fail_wait);
          ++written[i][warp];
        },
        [&](int b) {
          std::lock_guard<std::mutex> lock(sim.m);
          first->sum_empty[b].arrive();
          sim.changed.notify_all();
        });
  }
  void start(std::vector<std::thread>& roles) {
    roles.emplace_back([this] { load(); });
    if (first == this) roles.emplace_back([this] { multiply(); });
    for (int w = 0; w < kWarps; ++w) roles.emplace_back([this, w] { write(w); });
  }
};

// Keys and values: role 0 loads, role 1 stands for the products that read them.
struct Blocks {
  static constexpr int KS = 2, VS = 3;
  Sim& sim;
  int count;
  bool ragged;             // the last block is not full
  Sim::Bar k_full[KS], k_empty[KS], v_full[VS], v_empty[VS], v_landed;
  Sim::Stage keys[KS], values[VS];
  int seen = 0;

  Blocks(Sim& s, int n, bool r) : sim(s), count(n), ragged(r) {}
  bool is_part(int b, int half) const { return ragged && (b == count - 1 || (b == 1 && half == 1)); }
  void copy(Sim::Stage* stage, Sim::Stage is, Sim::Bar* bar) {
    bar->arrive(kBytes);
    ++sim.copies;
    sim.copying.push_back([=, this] {
      *stage = is;
      bar->landed(kBytes);
      --sim.copies;
    });
    sim.changed.notify_all();
  }
  void load() {
    int waits = 0, moved = -1;
    auto drained = [&](Sim::Bar& bar, uint32_t parity) {
      std::unique_lock<std::mutex> lock(sim.m);
      if (!sim.changed.wait_for(lock, std::chrono::seconds(2), [&] { return bar.complete(parity); }))
        fail("copies that never count as landed", sim.fail_role, sim.fail_wait);
    };
    tmb::fill_blocks<KS, VS>(
        count,
        [&](int b, int s) {
          std::lock_guard<std::mutex> lock(sim.m);
          copy(&keys[s], {b, 0}, &k_full[s]);
        },
        [&](int b, int half, int s) {
          std::lock_guard<std::mutex> lock(sim.m);
          if (b != moved) fail("values of another block", 0, waits);
          copy(&values[s], {b, half}, is_part(b, half) ? &v_landed : &v_full[s]);
          return is_part(b, half);
        },
        [&](uint32_t parity) { return sim.wait(v_landed, parity, 0, waits); },
        [&](int b, int half, int s) {
          std::lock_guard<std::mutex> lock(sim.m);
          if (values[s].tile != b || values[s].chunk != half) fail("a half that has not landed", sim.fail_role, sim.fail_wait);
          v_full[s].arrive();
          sim.changed.notify_all();
        },
        [&](int b) { moved = b + 1; }, [&](int s, uint32_t parity) { return sim.wait(k_empty[s], parity, 0, waits); },
        [&](int s, uint32_t parity) { return sim.wait(v_empty[s], parity, 0, waits); }, [&](int s, uint32_t parity) { drained(k_full[s], parity); },
        [&](int s, uint32_t parity) { drained(v_full[s], parity); }, [&](uint32_t parity) { drained(v_landed, parity); });
  }
  void read() {
    int waits = 0;
    auto product = [&](Sim::Stage* held, Sim::Stage is, Sim::Bar* empty) {
      std::lock_guard<std::mutex> lock(sim.m);
      sim.queue.push_back([=, this] {
        if (held->tile != is.tile || held->chunk != is.chunk) fail("a product on another block's stage", sim.fail_role, sim.fail_wait);
        empty->arrive();
        ++seen;
      });
      sim.changed.notify_all();
    };
    for (int b = 0; b <= count; ++b) {
      if (b < count) {
        if (!sim.wait(k_full[b % KS], uint32_t(b / KS) & 1u, 1, waits)) return;
        product(&keys[b % KS], {b, 0}, &k_empty[b % KS]);
      }
      for (int v = 2 * b - 2; b > 0 && v < 2 * b; ++v) {
        if (!sim.wait(v_full[v % VS], uint32_t(v / VS) & 1u, 1, waits)) return;
        product(&values[v % VS], {b - 1, v & 1}, &v_empty[v % VS]);
      }
    }
  }
};

// One run; false: its failing wait was never reached.
bool attempt_blocks(int count, int role, int wait, unsigned seed) {
  Sim sim(role, wait, seed);
  Blocks blocks(sim, count, count % 2);
  std::thread load([&] { blocks.load(); }), read([&] { blocks.read(); });
  load.join();
  read.join();
  std::unique_lock<std::mutex> lock(sim.m);
  if (sim.copies) fail("copies under way where the CTA goes", role, wait);
  sim.changed.wait(lock, [&] { return sim.queue.empty(); });
  if (!sim.failed && blocks.seen != 3 * count) fail("a block not read", role, wait);
  return sim.failed;
}

bool attempt(bool pair, int role, int wait, unsigned seed) {
  Sim sim(role, wait, seed);
  Cta one(sim, nullptr);
  std::optional<Cta> other;
  if (pair) other.emplace(sim, &one);
  std::vector<std::thread> roles;
  one.start(roles);
  if (pair) other->start(roles);
  for (auto& thread : roles) thread.join();
  if (pair) one.drain();
  std::lock_guard<std::mutex> lock(sim.m);
  if (sim.products) fail("products under way where tensor memory is freed", role, wait);
  if (sim.copies) fail("copies under way where the CTAs go", role, wait);
  if (sim.failed) return true;
  one.each([&](Cta& cta) {
    for (int i = 1; i < kTiles; i += kStep)
      for (int w = 0; w < kWarps; ++w)
        if (cta.written[i][w] != 1) fail("a tile not written once", role, wait);
  });
  return false;
}

}  // namespace

int main() {
  alarm(110);              // (a role that never ends)
  int runs = 0;
  for (unsigned seed = 0; seed < 3; ++seed) {
    for (int count : {1, 2, 6, 7}) {
      if (attempt_blocks(count, -1, 0, seed)) return 1;
      for (int role : {0, 1})
        for (int wait = 0; attempt_blocks(count, role, wait, seed * 1000 + unsigned(wait)); ++wait) ++runs;
    }
    for (bool pair : {false, true}) {
      if (attempt(pair, -1, 0, seed)) return 1;
      for (int role : {0, 1, 2, 5, 9, 20, 22, 26})
        if (pair || role < 20)
          for (int wait = 0; attempt(pair, role, wait, seed * 1000 + unsigned(wait)); ++wait) ++runs;
    }
  }
  std::printf("%d waits gave up, every role ended\n", runs);
  return 0;
}
