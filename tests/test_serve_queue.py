"""A server's queue when a round fails: the queries it had admitted go back to
the front of the queue in their order, their slots are free, and the next round
admits the same ones; a batch that is given up leaves nothing behind.  Host
code, compiled with the host compiler; no GPU needed."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "glint_pipeline_gb300", "csrc")

pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not available")

SOURCE = r"""
#include <cstdio>
#include <unordered_map>
#include "serve_queue.h"
using namespace glint;
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

static void fill(std::deque<PendingQuery> &q) {
    for (uint64_t t = 1; t <= 5; ++t)
        q.push_back(PendingQuery{t, {7, 3, 7, 100, (uint32_t)t}, (uint32_t)t, 10 * (uint32_t)t, 20 * (uint32_t)t});
}

int main() {
    std::deque<PendingQuery> queue;
    std::vector<SlotState> state(4);
    fill(queue);
    state[1].busy = true; /* a query of an earlier round */
    state[1].ticket = 99;
    state[1].frontier = 5;
    const uint32_t ids[1] = {0};
    state[1].front_ids = ids;
    for (int fail = 0; fail < 2; ++fail) {
        Admission a(queue, state);
        a.take(50);
        CHECK(a.slots == std::vector<uint32_t>({0, 2, 3}));
        CHECK(a.seeds == std::vector<uint32_t>({1, 3, 7, 2, 3, 7, 3, 7})); /* each once, none from 50 on */
        CHECK(a.sprefix == std::vector<uint32_t>({0, 3, 6, 8}));
        CHECK(a.query(1).ticket == 2 && a.query(1).t_start == 20 && a.query(1).t_end == 40);
        CHECK(state[2].busy && state[2].ticket == 2 && state[2].hops == 2 && state[2].frontier == 3);
        CHECK(queue.size() == 2);
        /* the round's buffers cannot be had: no keep() */
    }
    CHECK(queue.size() == 5);
    for (uint64_t t = 1; t <= 5; ++t) {
        CHECK(queue[t - 1].ticket == t && queue[t - 1].hops == t);
        CHECK(queue[t - 1].t_start == 10 * t && queue[t - 1].t_end == 20 * t);
    }
    for (int k : {0, 2, 3}) CHECK(!state[k].busy && state[k].frontier == 0 && state[k].front_ids == nullptr);
    CHECK(state[1].busy && state[1].ticket == 99 && state[1].frontier == 5 && state[1].front_ids == ids);
    {
        Admission a(queue, state);
        a.take(50);
        a.keep();
    }
    CHECK(queue.size() == 2 && queue[0].ticket == 4);
    CHECK(state[0].ticket == 1 && state[2].ticket == 2 && state[3].ticket == 3);

    /* a round's seeds and a scan's marks are counted in 32 bits */
    {
        std::deque<PendingQuery> q;
        std::vector<SlotState> st(4);
        fill(q);
        Admission a(q, st);
        a.take(50, 9); /* five seeds a query, three after sorting: 3 + 5, but not 6 + 5 */
        CHECK(a.slots.size() == 2 && q.size() == 3 && q[0].ticket == 3);
    }
    {
        std::deque<PendingQuery> q;
        std::vector<SlotState> st(1);
        fill(q);
        Admission a(q, st);
        a.take(50, 1); /* one query is always taken */
        CHECK(a.slots.size() == 1);
    }
    for (uint32_t N : {1u, 31u, 1000u, 10000000u, (1u << 26) - 1}) {
        const uint64_t g = mark_group(N);
        CHECK(g >= 64 && g * N <= 0xffffffffull && g * slot_words(N) <= 0xf0000000ull);
        CHECK((g + 1) * N > 0xffffffffull || (g + 1) * slot_words(N) > 0xf0000000ull);
    }
    CHECK(slot_words(1) == 8 && slot_words(256) == 8 && slot_words(257) == 16);

    std::unordered_map<uint64_t, FinishedQuery> done;
    done[2] = FinishedQuery();
    done[98] = FinishedQuery();
    cancel_queries({1, 2, 4}, queue, state, done);
    CHECK(queue.size() == 1 && queue[0].ticket == 5);
    CHECK(!state[0].busy && !state[2].busy && state[1].busy && state[3].busy);
    CHECK(done.size() == 1 && done.count(98) == 1);
    return 0;
}
"""


def test_failed_round_gives_its_queries_back(tmp_path):
    src, exe = tmp_path / "queue.cpp", tmp_path / "queue"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
