// Host-thread model of the two kernels of the fused layer for ranks that share one GPU (yali_c.h,
// yali_c_simulate_local; kernels/gemm_local.cu).  One host thread plays one pair of CTAs of the GEMM or one CTA of the
// row kernel.  Modelled is what passes between the two and from call to call: the call numbers and who reads and advances
// them when, the release of the dependent kernel, the walk over the items, sums announced by flags or sent as flag-in-data lines,
// rows taken from a counter, the check-in that clears the counter and advances the call number, and the clearing of
// the control words between calls (Communicator::Reset).  The GEMM itself is a formula of (call, row, unit, split).
// Calls follow one another in stream order.  A call's GEMM may start under the rows of the call in front, but all it does before they
// have finished is to set up and to prefetch its weights, which touches none of this: here a call starts when both kernels of
// the one before it have finished.
//
// Parity: the reference has neither the fused layer nor a protocol model.
#include <atomic>
#include <chrono>
#include <cmath>
#include <condition_variable>
#include <cstring>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

#include "../capi/yali_c.h"

namespace {

using Clock = std::chrono::steady_clock;

struct Barrier {
    std::mutex m;
    std::condition_variable cv;
    int count, waiting = 0, gen = 0;
    explicit Barrier(int n) : count(n) {}
    void wait() {
        std::unique_lock<std::mutex> l(m);
        const int g = gen;
        if (++waiting == count) {
            waiting = 0;
            ++gen;
            cv.notify_all();
        } else {
            cv.wait(l, [&] { return g != gen; });
        }
    }
};

struct LocalShared {
    YaliLocalSimConfig cfg;
    uint32_t T, units, ks, tiles;
    std::atomic<uint32_t> gemm_number{0}, gemm_in{0};            // the GEMM's count of calls, its CTAs that have read it
    std::atomic<uint32_t> number{0}, counter{0}, checked_in{0};  // the row kernel's count, unit counter, check-ins
    std::atomic<int> released{0};                                // GEMM CTAs that have released the row kernel
    std::unique_ptr<std::atomic<uint64_t>[]> lines;              // [split][row][unit]: {call number, value}
    std::unique_ptr<std::atomic<uint32_t>[]> flags;              // [tile][split][unit]: call number
    std::unique_ptr<std::atomic<uint32_t>[]> sums;               // [split][row][unit]: value (plain sums)
    std::unique_ptr<std::atomic<uint32_t>[]> out, written;       // [row][unit] value; [row] times written in this call
    std::unique_ptr<Barrier> call_end;
    std::atomic<uint64_t> timeouts{0}, violations{0}, mismatches{0}, writes{0};
    std::atomic<bool> abort{false};
    size_t At(uint32_t split, uint32_t row, uint32_t unit) const { return (static_cast<size_t>(split) * T + row) * units + unit; }
};

float Value(int call, uint32_t row, uint32_t unit, uint32_t split) {
    return static_cast<float>((call * 131 + row * 7 + unit * 3 + split * 29) % 251) * 0.125f - 9.0f;
}
uint32_t Bits(float v) {
    uint32_t b;
    std::memcpy(&b, &v, 4);
    return b;
}
float Unbits(uint32_t b) {
    float v;
    std::memcpy(&v, &b, 4);
    return v;
}

template <typename Ready>
bool WaitFor(LocalShared& s, Ready ready) {
    const auto deadline = Clock::now() + std::chrono::milliseconds(s.cfg.timeout_ms);
    for (uint32_t spins = 1; !ready(); ++spins) {
        if ((spins & 63u) != 0) continue;
        if (s.abort.load() || Clock::now() > deadline) {
            s.timeouts.fetch_add(1);
            s.abort = true;
            return false;
        }
        std::this_thread::yield();
    }
    return true;
}

void GemmCta(LocalShared& s, int c, int call) {
    auto doze = [&] {
        if (c == s.cfg.slow_cta) std::this_thread::sleep_for(std::chrono::milliseconds(3));
    };
    s.released.fetch_add(1, std::memory_order_acq_rel);
    uint32_t number;
    if (s.cfg.shared_number) {
        // As late as it gets: after the row kernel has moved on to the next number, if it does so without this thread.
        const uint32_t before = static_cast<uint32_t>(call) - (s.cfg.reset_at > 0 && call >= s.cfg.reset_at ? s.cfg.reset_at : 0);
        for (int ms = 0; c == s.cfg.slow_cta && ms < 200 && s.number.load() == before; ++ms)
            std::this_thread::sleep_for(std::chrono::milliseconds(1));
        number = s.number.load(std::memory_order_acquire) + 1u;
    } else {
        doze();
        number = s.gemm_number.load(std::memory_order_acquire) + 1u;
        if (s.gemm_in.fetch_add(1) == static_cast<uint32_t>(s.cfg.pairs) - 1) {
            s.gemm_in.store(0);
            s.gemm_number.store(number, std::memory_order_release);
        }
        doze();
    }
    const uint32_t per_tile = s.units * s.ks;
    for (uint32_t i = c; i < s.tiles * per_tile; i += s.cfg.pairs) {
        const uint32_t tile = i / per_tile, split = i % per_tile / s.units, unit = i % s.units;
        if (s.cfg.fault == 1 && call == s.cfg.fault_call && i == static_cast<uint32_t>(c)) continue;  // this item is lost
        const uint32_t hi = std::min(s.T, (tile + 1) * s.cfg.tile_rows);
        for (uint32_t row = tile * s.cfg.tile_rows; row < hi; ++row) {
            const uint32_t bits = Bits(Value(call, row, unit, split));
            if (s.cfg.lines)
                s.lines[s.At(split, row, unit)].store((static_cast<uint64_t>(number) << 32) | bits, std::memory_order_release);
            else
                s.sums[s.At(split, row, unit)].store(bits, std::memory_order_relaxed);
            s.writes.fetch_add(1, std::memory_order_relaxed);
        }
        if (!s.cfg.lines) s.flags[(tile * s.ks + split) * s.units + unit].store(number, std::memory_order_release);
    }
}

void RowCta(LocalShared& s, int c, int call) {
    if (!WaitFor(s, [&] { return s.released.load(std::memory_order_acquire) == s.cfg.pairs * (call + 1); })) return;
    const uint32_t number = s.number.load(std::memory_order_acquire) + 1u, ctas = s.cfg.row_ctas;
    const bool taking = ctas < s.T;
    auto check_in = [&] {
        if (s.checked_in.fetch_add(1) != ctas - 1) return;
        s.checked_in.store(0);
        s.counter.store(0);
        s.number.store(number, std::memory_order_release);
    };
    uint32_t row = taking ? s.counter.fetch_add(1) : static_cast<uint32_t>(c);
    if (row >= s.T) check_in();
    while (row < s.T) {
        const uint32_t mine = row, tile = mine / s.cfg.tile_rows;
        row = taking ? s.counter.fetch_add(1) : s.T;
        if (!s.cfg.lines) {
            for (uint32_t f = tile * s.ks * s.units; f < (tile + 1) * s.ks * s.units; ++f)
                if (!WaitFor(s, [&] { return static_cast<int32_t>(s.flags[f].load(std::memory_order_acquire) - number) >= 0; })) return;
        }
        if (row >= s.T) check_in();  // under the work of the last row
        for (uint32_t unit = 0; unit < s.units; ++unit) {
            float sum = 0.f;
            for (uint32_t split = 0; split < s.ks; ++split) {
                if (s.cfg.lines) {
                    uint64_t w = 0;
                    if (!WaitFor(s, [&] {
                            w = s.lines[s.At(split, mine, unit)].load(std::memory_order_acquire);
                            return static_cast<uint32_t>(w >> 32) == number;
                        }))
                        return;
                    sum += Unbits(static_cast<uint32_t>(w));
                } else {
                    sum += Unbits(s.sums[s.At(split, mine, unit)].load(std::memory_order_relaxed));
                }
            }
            s.out[static_cast<size_t>(mine) * s.units + unit].store(Bits(sum));
        }
        s.written[mine].fetch_add(1);
    }
}

// `c` < pairs: a pair of the GEMM, else a CTA of the row kernel.
void Cta(LocalShared& s, int c) {
    for (int call = 0; call < s.cfg.calls && !s.abort.load(); ++call) {
        if (c < s.cfg.pairs) GemmCta(s, c, call);
        else RowCta(s, c - s.cfg.pairs, call);
        s.call_end->wait();  // stream order
        if (c == 0 && !s.abort.load()) {
            for (uint32_t row = 0; row < s.T; ++row) {
                if (s.written[row].exchange(0) != 1) s.violations.fetch_add(1);
                for (uint32_t unit = 0; unit < s.units; ++unit) {
                    float want = 0.f;
                    for (uint32_t split = 0; split < s.ks; ++split) want += Value(call, row, unit, split);
                    if (std::fabs(Unbits(s.out[static_cast<size_t>(row) * s.units + unit].load()) - want) > 1e-3f) s.mismatches.fetch_add(1);
                }
            }
            if (s.counter.load() != 0 || s.checked_in.load() != 0) s.violations.fetch_add(1);
            if (call + 1 == s.cfg.reset_at) {
                s.number.store(0);
                s.gemm_number.store(0);
                for (uint32_t f = 0; f < s.tiles * s.ks * s.units; ++f) s.flags[f].store(0);
                if (!s.cfg.keep_lines)
                    for (size_t i = 0; i < s.At(s.ks, 0, 0); ++i) s.lines[i].store(0);
            }
        }
        s.call_end->wait();
    }
}

}  // namespace

extern "C" int yali_c_simulate_local(const YaliLocalSimConfig* cfg, YaliSimReport* rep) {
    std::memset(rep, 0, sizeof(*rep));
    rep->timeout_rank = rep->timeout_peer = -1;
    if (!cfg || cfg->pairs < 1 || cfg->pairs > 64 || cfg->row_ctas < 1 || cfg->row_ctas > 64 || cfg->calls < 1 || cfg->rows == 0 ||
        cfg->col_units == 0 || cfg->splits == 0 || cfg->tile_rows == 0 || static_cast<uint32_t>(cfg->row_ctas) > cfg->rows)
        return -1;
    LocalShared s;
    s.cfg = *cfg;
    s.T = cfg->rows;
    s.units = cfg->col_units;
    s.ks = cfg->splits;
    s.tiles = (s.T + cfg->tile_rows - 1) / cfg->tile_rows;
    const size_t n = s.At(s.ks, 0, 0), nflags = static_cast<size_t>(s.tiles) * s.ks * s.units;
    s.lines.reset(new std::atomic<uint64_t>[n]);
    s.sums.reset(new std::atomic<uint32_t>[n]);
    s.flags.reset(new std::atomic<uint32_t>[nflags]);
    s.out.reset(new std::atomic<uint32_t>[static_cast<size_t>(s.T) * s.units]);
    s.written.reset(new std::atomic<uint32_t>[s.T]);
    for (size_t i = 0; i < n; ++i) s.lines[i].store(0), s.sums[i].store(0);
    for (size_t i = 0; i < nflags; ++i) s.flags[i].store(0);
    for (size_t i = 0; i < static_cast<size_t>(s.T) * s.units; ++i) s.out[i].store(0);
    for (uint32_t i = 0; i < s.T; ++i) s.written[i].store(0);
    s.call_end.reset(new Barrier(cfg->pairs + cfg->row_ctas));
    std::vector<std::thread> threads;
    for (int c = 0; c < cfg->pairs + cfg->row_ctas; ++c) threads.emplace_back(Cta, std::ref(s), c);
    for (auto& t : threads) t.join();
    rep->timeouts = s.timeouts.load();
    rep->flag_writes = s.writes.load();
    rep->mismatches = s.violations.load();
    if (rep->mismatches) return rep->status = 3;
    if (rep->timeouts) return rep->status = 2;
    rep->mismatches = s.mismatches.load();
    return rep->status = rep->mismatches ? 1 : 0;
}
