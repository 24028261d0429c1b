// Shared host-side helpers of the fvmpor_b200 library.
#pragma once

#include "../../include/fvmpor_b200.h"

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstdlib>
#include <exception>
#include <mutex>
#include <stdexcept>
#include <string>
#include <thread>
#include <vector>

namespace fvmb {

struct Error : std::runtime_error {
    int code;
    explicit Error(const std::string& m, int c = -1) : std::runtime_error(m), code(c) {}
};

void set_error(const std::string& msg);

// body(first, last) over runs of [0, n) on the machine's cores (at most 16, none
// for less than `grain` items per thread).  Runs are handed out in order, so of
// several exceptions the one rethrown is the first in item order.
template <class F> void parallel_for(long n, long grain, F&& body) {
    const long want = std::min<long>(16, std::max(1u, std::thread::hardware_concurrency()));
    const long threads = std::max<long>(1, std::min(want, n / std::max<long>(1, grain)));
    if (threads == 1) {
        if (n > 0) body(0l, n);
        return;
    }
    // runs a few times smaller than a thread's share, taken as threads get free
    const long run = std::max<long>(1, n / (4 * threads));
    std::atomic<long> next{0};
    std::exception_ptr error;
    long error_at = n;
    std::mutex guard;
    auto work = [&] {
        long a = 0;
        try {
            while ((a = next.fetch_add(run)) < n) body(a, std::min(n, a + run));
        } catch (...) {
            std::lock_guard<std::mutex> hold(guard);
            if (a < error_at) {
                error_at = a;
                error = std::current_exception();
            }
            next = n;
        }
    };
    std::vector<std::thread> pool;
    pool.reserve(threads - 1);
    try {
        for (long t = 1; t < threads; ++t) pool.emplace_back(work);
    } catch (...) {
        // no thread or no memory for one: those there are do the work (leaving
        // here with threads still running would end the process)
    }
    work();
    for (std::thread& t : pool) t.join();
    if (error) std::rethrow_exception(error);
}

struct Rng {
    uint64_t s;
    bool has_spare = false;
    double spare = 0.0;
    explicit Rng(uint64_t seed);
    uint64_t next();
    double uniform();
    double normal();
};

std::vector<double> gaussian_field(int nx, int ny, int nz, double hx, double hy, double hz,
                                   double var, double Lx, double Ly, double Lz, uint64_t seed);

} // namespace fvmb
