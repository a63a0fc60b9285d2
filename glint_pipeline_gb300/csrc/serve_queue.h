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
/* seeds of one round, numbered in 32 bits by grids of up to 2^28 threads */
constexpr uint64_t kMaxRoundSeeds = 0xf0000000ull;

/* a slot's bitmap words: whole scan threads of eight */
inline uint32_t slot_words(uint32_t N) { return (uint32_t)(((uint64_t)N + 255) / 256 * 8); }

/* The slots whose marks one scan counts: each marks up to N objects, and the
 * scan's sums, like its length, have 32 bits.  429 at 10M objects, 64 at 2^26 -
 * 1: a round of the default server is one scan at every size. */
inline uint32_t mark_group(uint32_t N) {
    return (uint32_t)std::min<uint64_t>(0xffffffffull / std::max(N, 1u), 0xf0000000ull / std::max(slot_words(N), 8u));
}

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

    /* seeds from N on are no objects; a query whose seeds would be too many
     * beside the others' waits for the next round */
    void take(uint32_t N, uint64_t max_seeds = kMaxRoundSeeds) {
        taken_.reserve(std::min(queue_.size(), state_.size()));
        slots.reserve(taken_.capacity());
        for (uint32_t k = 0; k < state_.size() && !queue_.empty(); ++k) {
            if (state_[k].busy) continue;
            if (!seeds.empty() && seeds.size() + queue_.front().seeds.size() > max_seeds) break;
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
