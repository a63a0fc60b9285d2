/*
 * serve_queue.h -- a server's queued and running queries: host code only, so
 * that what happens to them when a round fails can be tested without a GPU.
 */
#ifndef GLINT_SERVE_QUEUE_H_
#define GLINT_SERVE_QUEUE_H_

#include <stdint.h>

#include <algorithm>
#include <deque>
#include <utility>
#include <vector>

namespace glint {

constexpr uint32_t kMaxHops = 8;

struct PendingQuery {
    uint64_t ticket;
    std::vector<uint32_t> seeds;
    uint32_t hops, t_start, t_end;
};

struct SlotState {
    bool busy = false;
    uint64_t ticket = 0;
    uint32_t hops = 0, hop = 0, frontier = 0;
    const uint32_t *front_ids = nullptr; /* device: the last hop's part of the result list, or the seeds */
    uint64_t reached = 0; /* seeds and every hop's new objects so far */
    std::vector<uint32_t> ids;
    uint64_t hop_end[kMaxHops] = {};
};

struct FinishedQuery {
    std::vector<uint32_t> ids;
    uint64_t hop_end[kMaxHops];
    uint64_t keys_scanned;
};

/* One round's admissions: queued queries into free slots; their seeds, each
 * once, are their first frontier.  The seeds and reached sets of these slots
 * are on the device only when the round's first launches have run, so a round
 * that ends before (its buffers could not be had) gives the queries back to the
 * front of the queue and their slots free: a slot left busy would have a
 * frontier without an address. */
class Admission {
public:
    Admission(std::deque<PendingQuery> &queue, std::vector<SlotState> &state) : queue_(queue), state_(state) {}
    Admission(const Admission &) = delete;
    Admission &operator=(const Admission &) = delete;
    ~Admission() {
        if (kept_) return;
        for (uint32_t k : slots) state_[k] = SlotState();
        for (size_t i = taken_.size(); i-- > 0;) queue_.push_front(std::move(taken_[i]));
    }

    /* seeds from N on are no objects */
    void take(uint32_t N) {
        taken_.reserve(std::min(queue_.size(), state_.size()));
        slots.reserve(taken_.capacity());
        for (uint32_t k = 0; k < state_.size() && !queue_.empty(); ++k) {
            if (state_[k].busy) continue;
            taken_.push_back(std::move(queue_.front()));
            queue_.pop_front();
            PendingQuery &q = taken_.back();
            std::sort(q.seeds.begin(), q.seeds.end());
            q.seeds.erase(std::unique(q.seeds.begin(), q.seeds.end()), q.seeds.end());
            while (!q.seeds.empty() && q.seeds.back() >= N) q.seeds.pop_back();
            SlotState &st = state_[k];
            st = SlotState();
            st.busy = true;
            st.ticket = q.ticket;
            st.hops = q.hops;
            st.frontier = (uint32_t)q.seeds.size();
            st.reached = st.frontier;
            slots.push_back(k);
            seeds.insert(seeds.end(), q.seeds.begin(), q.seeds.end());
            sprefix.push_back((uint32_t)seeds.size());
        }
    }
    /* the query that took slots[i] */
    const PendingQuery &query(size_t i) const { return taken_[i]; }
    /* the round has run */
    void keep() { kept_ = true; }

    std::vector<uint32_t> slots, seeds, sprefix = std::vector<uint32_t>(1, 0);

private:
    std::deque<PendingQuery> &queue_;
    std::vector<SlotState> &state_;
    std::vector<PendingQuery> taken_;
    bool kept_ = false;
};

/* forgets the queries with these tickets (ascending), wherever they are: a
 * caller that gives up a batch leaves nothing of it behind */
template <class Done>
void cancel_queries(const std::vector<uint64_t> &tickets, std::deque<PendingQuery> &queue,
                    std::vector<SlotState> &state, Done &done) {
    auto listed = [&](uint64_t t) { return std::binary_search(tickets.begin(), tickets.end(), t); };
    queue.erase(std::remove_if(queue.begin(), queue.end(), [&](const PendingQuery &q) { return listed(q.ticket); }),
                queue.end());
    for (SlotState &st : state)
        if (st.busy && listed(st.ticket)) st = SlotState();
    for (uint64_t t : tickets) done.erase(t);
}

} // namespace glint

#endif
