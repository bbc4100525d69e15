// A warp on the host: 32 lanes as coroutines on one thread.  A lane runs until its next
// collective operation, alone and in a chosen order, so code that relies on lanes moving
// in step, which the programming model does not promise, shows here.
#pragma once

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <functional>
#include <ucontext.h>
#include <vector>

namespace emulation {

class Warp {
public:
    enum Collective { NONE, SYNC, BROADCAST };

    // Runs body(warp, lane) for 32 lanes; between two collectives lanes run in ascending
    // (or descending) order.  Returns false, with a line on stderr, if lanes meet at
    // different collectives or some end while others wait.
    bool run(const std::function<void(Warp&, int)>& body, bool ascending)
    {
        body_ = &body;
        lanes_.assign(32, Lane {});
        for (int i = 0; i < 32; ++i) {
            Lane& l = lanes_[i];
            l.stack.resize(128 << 10);
            getcontext(&l.context);
            l.context.uc_stack.ss_sp = l.stack.data();
            l.context.uc_stack.ss_size = l.stack.size();
            l.context.uc_link = &scheduler_;
            const auto self = reinterpret_cast<std::uintptr_t>(this);
            makecontext(&l.context, reinterpret_cast<void (*)()>(&Warp::entry), 2, static_cast<unsigned>(self),
                static_cast<unsigned>(static_cast<std::uint64_t>(self) >> 32));
        }
        while (true) {
            for (int k = 0; k < 32; ++k) {
                current_ = ascending ? k : 31 - k;
                if (!lanes_[current_].ended)
                    swapcontext(&scheduler_, &lanes_[current_].context);
            }
            bool all_ended = true;
            for (const Lane& l : lanes_)
                all_ended = all_ended && l.ended;
            if (all_ended)
                return true;
            for (int i = 0; i < 32; ++i) {
                const Lane& l = lanes_[i];
                if (l.ended || l.at != lanes_[0].at) {
                    std::fprintf(stderr, "lane %d %s while lane 0 %s\n", i, l.ended ? "has ended" : name(l.at),
                        lanes_[0].ended ? "has ended" : name(lanes_[0].at));
                    return false;
                }
            }
        }
    }

    bool leader() const { return current_ == 0; }
    void sync() { meet(SYNC); }
    std::uint64_t broadcast(std::uint64_t v)
    {
        if (current_ == 0)
            value_ = v;
        meet(BROADCAST);
        return value_;
    }
    std::uint64_t fetch_add(unsigned long long* head) { return (*head)++; }
    void stop(unsigned long long* head) { *head |= 1ull << 63; }

private:
    struct Lane {
        ucontext_t context {};
        std::vector<char> stack;
        Collective at = NONE;
        bool ended = false;
    };
    static const char* name(Collective c) { return c == SYNC ? "waits in sync" : (c == BROADCAST ? "waits in broadcast" : "runs"); }
    static void entry(unsigned low, unsigned high)
    {
        auto* w = reinterpret_cast<Warp*>(static_cast<std::uintptr_t>((static_cast<std::uint64_t>(high) << 32) | low));
        const int lane = w->current_;
        (*w->body_)(*w, lane);
        w->lanes_[lane].ended = true;
    }
    void meet(Collective c)
    {
        const int lane = current_;
        lanes_[lane].at = c;
        swapcontext(&lanes_[lane].context, &scheduler_);
        lanes_[lane].at = NONE;
    }

    const std::function<void(Warp&, int)>* body_ = nullptr;
    std::vector<Lane> lanes_;
    ucontext_t scheduler_ {};
    int current_ = 0;
    std::uint64_t value_ = 0;
};

} // namespace emulation
