// Workers kept between the phases of a call instead of started for each: a symbolic phase runs about ten
// parallel passes, and starting 16 threads for each of them took 6 of the 8 ms of such a phase at 5,403
// DoFs. A worker that has had nothing to do for kIdle ends, so a program that stops calling the library
// holds no threads of it; at most num_host_threads() - 1 exist at a time.
#include "host_pool.h"

#include <pthread.h>

#include <algorithm>
#include <chrono>
#include <condition_variable>
#include <deque>
#include <exception>
#include <memory>
#include <mutex>
#include <system_error>
#include <thread>

namespace fem2d {

namespace {

constexpr std::chrono::milliseconds kIdle(200);

struct Job {
  const std::function<void(int)>* f;
  int total, next = 0, done = 0;   // guarded by Pool::mu
  std::exception_ptr error;
  std::condition_variable finished;
};

struct Pool {
  std::mutex mu;
  std::condition_variable work;
  std::deque<std::shared_ptr<Job>> jobs;   // with calls not yet taken
  int workers = 0, idle = 0;

  // takes and runs one call of the job; false when none is left. lk is held on entry and return
  bool step(const std::shared_ptr<Job>& j, std::unique_lock<std::mutex>& lk) {
    if (j->next >= j->total) return false;
    const int t = j->next++;
    if (j->next >= j->total) jobs.erase(std::find(jobs.begin(), jobs.end(), j));
    lk.unlock();
    std::exception_ptr err;
    try {
      (*j->f)(t);
    } catch (...) {
      err = std::current_exception();
    }
    lk.lock();
    if (err && !j->error) j->error = err;
    if (++j->done == j->total) j->finished.notify_all();
    return true;
  }

  void worker() {
    std::unique_lock<std::mutex> lk(mu);
    for (;;) {
      while (!jobs.empty()) {
        const std::shared_ptr<Job> j = jobs.front();
        step(j, lk);
      }
      idle++;
      const bool woken = work.wait_for(lk, kIdle, [&] { return !jobs.empty(); });
      idle--;
      if (!woken) break;
    }
    workers--;
  }
};

Pool* g_pool = nullptr;   // never destroyed: a worker may outlive the library's static objects
std::mutex g_pool_mu;

// a forked child has none of the workers, and may have inherited the mutex locked
void after_fork() {
  g_pool = nullptr;
  new (&g_pool_mu) std::mutex;
}

Pool& pool() {
  std::lock_guard<std::mutex> lk(g_pool_mu);
  if (!g_pool) {
    static const int registered = pthread_atfork(nullptr, nullptr, after_fork);
    (void)registered;
    g_pool = new Pool;
  }
  return *g_pool;
}

}  // namespace

int num_host_threads() {
  const unsigned h = std::thread::hardware_concurrency();
  return h == 0 ? 4 : (int)std::min(h, 64u);
}

void run_threads(int nt, const std::function<void(int)>& f) {
  if (nt <= 1) {
    if (nt == 1) f(0);
    return;
  }
  Pool& p = pool();
  auto j = std::make_shared<Job>();
  j->f = &f;
  j->total = nt;
  std::unique_lock<std::mutex> lk(p.mu);
  p.jobs.push_back(j);
  const int limit = num_host_threads() - 1;
  for (int want = nt - 1 - p.idle; want > 0 && p.workers < limit; want--) {
    try {
      std::thread([&p] { p.worker(); }).detach();
    } catch (const std::system_error&) {
      break;   // no more threads to be had: the caller does the work itself
    }
    p.workers++;
  }
  p.work.notify_all();
  while (p.step(j, lk)) {
  }
  j->finished.wait(lk, [&] { return j->done == j->total; });
  if (j->error) std::rethrow_exception(j->error);
}

}  // namespace fem2d
