// A persistent pool of host threads for the library's host-side work that
// splits into independent items (the ghost programs' emission after a
// regrid).  Threads are created once, on first use, and wait on a condition
// variable between calls; parallel_for(n, f) runs f(0..n-1) on them and on
// the calling thread and returns when every item is done.  A call made while
// another is running (another host thread, or an item calling parallel_for)
// runs its items on the calling thread alone, so calls never wait for each
// other.
#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <functional>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

#include "hier.h"

namespace bsamg {

namespace {

class Pool {
 public:
  Pool() {
    unsigned n = std::max(1u, std::thread::hardware_concurrency());
    for (unsigned t = 1; t < n; t++) workers_.emplace_back([this] { loop(); });
  }
  ~Pool() {
    {
      std::lock_guard<std::mutex> g(mu_);
      quit_ = true;
    }
    cv_.notify_all();
    for (auto& t : workers_) t.join();
  }
  void run(int n, const std::function<void(int)>& f) {
    std::unique_lock<std::mutex> busy(run_mu_, std::try_to_lock);
    if (!busy.owns_lock() || workers_.empty() || n < 2) {
      for (int x = 0; x < n; x++) f(x);
      return;
    }
    auto b = std::make_shared<Batch>(f, n);
    {
      std::lock_guard<std::mutex> g(mu_);
      batch_ = b;
      gen_++;
    }
    cv_.notify_all();
    work(*b);
    std::unique_lock<std::mutex> g(mu_);
    done_.wait(g, [&] { return b->left.load() == 0; });
    batch_.reset();
  }

 private:
  // One call's items.  Every call has its own counters: a worker that is
  // still leaving an earlier call draws its last number from that call's
  // (with counters shared by all calls it could draw an item of the next one
  // that another thread draws again, and the count of what is left missed
  // zero).  f outlives every item, not the batch.
  struct Batch {
    const std::function<void(int)>& f;
    const int n;
    std::atomic<int> next{0}, left;
    Batch(const std::function<void(int)>& fn, int items) : f(fn), n(items), left(items) {}
  };
  void work(Batch& b) {
    int done = 0;
    for (int x; (x = b.next.fetch_add(1)) < b.n;) {
      b.f(x);
      done++;
    }
    if (done && b.left.fetch_sub(done) == done) {
      std::lock_guard<std::mutex> g(mu_);
      done_.notify_all();
    }
  }
  void loop() {
    unsigned long long seen = 0;
    for (;;) {
      std::shared_ptr<Batch> b;
      {
        std::unique_lock<std::mutex> g(mu_);
        cv_.wait(g, [&] { return quit_ || (gen_ != seen && batch_); });
        if (quit_) return;
        seen = gen_;
        b = batch_;
      }
      work(*b);
    }
  }
  std::vector<std::thread> workers_;
  std::mutex mu_, run_mu_;
  std::condition_variable cv_, done_;
  std::shared_ptr<Batch> batch_;
  unsigned long long gen_ = 0;
  bool quit_ = false;
};

}  // namespace

void parallel_for(int n, const std::function<void(int)>& f) {
  static Pool pool;
  pool.run(n, f);
}

}  // namespace bsamg
