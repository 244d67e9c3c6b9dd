// Replayed one-shot host calls, on the stand-ins of fake_cuda.h.
#include <thread>

#include "fake_cuda.h"

#include "../../cvmatch_gb300/csrc/cvm_api.cpp"

namespace {

std::vector<uint8_t> frame(4096 * 4096 * 4), tpl(512 * 512 * 4);

int call(int w, int h, int tw, int th) {
    cvm_result r;
    return cvm_match(frame.data(), 4LL * w, w, h, tpl.data(), 4LL * tw, tw, th, &r);
}

// The capture happens while another thread switches the autotuner off, or
// publishes a plan: size and launches stay on the plan of the shape.
void plan_changes_during_the_capture(bool off) {
    cvm_set_form(CVM_FORM_FAST);
    cvm_set_autotune(1);
    const int w = 900, h = 700, tw = 40, th = 30;
    EXPECT(call(w, h, tw, th) == CVM_OK && call(w, h, tw, th) == CVM_OK);
    // the tuned plan: a small one; the other: the largest candidate
    const TuneKey key{w, h, tw, th, 1, 0, 4, CVM_FORM_FAST};
    const Plan small = plan_with(128, 128, tw, th, w - tw + 1, h - th + 1);
    const Plan large = plan_with(1024, 1024, tw, th, w - tw + 1, h - th + 1);
    EXPECT(g_tune.count(key) == 1);
    g_tune[key].plan = small;
    std::set<int> rows;
    fake::state().on_launch = [&](const char *name, const FftClass &fc) {
        if (!strcmp(name, "inv_rows")) rows.insert(fc.n);
    };
    fake::state().on_call = [&](const std::string &f) {
        if (f == "cudaHostAlloc") {
            if (off)
                g_autotune = 0;
            else
                g_tune[key].plan = large;
        }
        return cudaSuccess;
    };
    EXPECT(call(w, h, tw, th) == CVM_OK);
    EXPECT(fake::state().calls["cudaGraphLaunch"] == 1);
    EXPECT(rows == std::set<int>{128});
}

// Every call that queues work fails once, in every host-buffer entry point:
// an error return leaves nothing behind that still reads the caller's memory.
void errors_wait() {
    cvm_set_form(CVM_FORM_EXACT);
    const int w = 700, h = 300, tw = 40, th = 30;
    std::vector<float> map((size_t)(w - tw + 1) * (h - th + 1));
    std::vector<uint8_t> gray((size_t)w * h);
    cvm_matcher *m[2];
    for (int i = 0; i < 2; i++) {
        tpl[4 * i] = 7;
        EXPECT(cvm_matcher_new(tpl.data(), 4 * tw, tw, th, 4, &m[i]) == CVM_OK);
    }
    cvm_fleet *f;
    EXPECT(cvm_fleet_new(m, 2, &f) == CVM_OK);
    cvm_result r[2];
    int32_t xy[20], n;
    int c;
    const std::vector<std::function<int()>> entries = {
        [&] { return call(w, h, tw, th); },
        [&] { return cvm_match_gray_rgba(frame.data(), 4 * w, w, h, tpl.data(), 4 * tw, tw, th, r); },
        [&] { return cvm_match_map(frame.data(), 4 * w, w, h, tpl.data(), 4 * tw, tw, th, map.data()); },
        [&] { return cvm_match_map_peaks(frame.data(), 4 * w, w, h, tpl.data(), 4 * tw, tw, th, 0.5f, 2, 2, xy, 10, &n); },
        [&] { return cvm_matcher_find(m[0], frame.data(), 4 * w, w, h, r); },
        [&] { return cvm_fleet_find_all(f, frame.data(), 4 * w, w, h, r); },
        [&] { return cvm_rgba_to_gray(frame.data(), 4 * w, w, h, gray.data()); },
        [&] { return cvm_alpha_const(frame.data(), 4 * w, w, h, &c); },
    };
    auto &st = fake::state();
    const std::set<std::string> reads = {"ingest", "ingest_solo", "cudaMemcpy2DAsync", "cudaGraphLaunch"};
    int failed = 0;
    for (const auto &entry : entries)
        for (int replay = 0; replay < 2; replay++) {
            for (int k = replay ? 3 : 1; k > 0; k--) EXPECT(entry() == CVM_OK);
            for (int at = 0;; at++) {
                int i = 0;
                bool hit = false, reading = false;
                st.on_call = [&](const std::string &name) {
                    if (hit) return cudaSuccess;
                    if (i++ == at) {
                        hit = true;
                        st.synced.clear();
                        return cudaErrorUnknown;
                    }
                    reading = reading || reads.count(name);
                    return cudaSuccess;
                };
                const int rc = entry();
                st.on_call = nullptr;
                if (!hit) {
                    EXPECT(rc == CVM_OK);
                    break;
                }
                if (rc != CVM_OK && reading) {
                    failed++;
                    EXPECT(st.synced.count(thread_stream()) && st.synced.count(side_stream().st2));
                }
            }
        }
    EXPECT(failed > 60);
}

long graph_launches() { return fake::state().calls["cudaGraphLaunch"]; }

// Calls of one shape from ever new threads, one at a time: they share what is
// kept, and from the fourth on a thread's first call replays.
void threads_share() {
    cvm_set_form(CVM_FORM_EXACT);
    size_t after = 0;
    for (int i = 0; i < 24; i++) {
        std::thread([&] { EXPECT(call(700, 300, 40, 30) == CVM_OK); }).join();
        if (i >= 3) EXPECT(graph_launches() == i - 1);
        if (i == 3) after = fake::state().deviceBytes;
    }
    EXPECT(fake::state().calls["cudaGraphInstantiate"] == 1);
    EXPECT(fake::state().deviceBytes == after);
}

// Threads inside calls of one shape at the same time, a graph each: bounded.
void threads_bounded() {
    cvm_set_form(CVM_FORM_EXACT);
    for (int i = 0; i < 3; i++) EXPECT(call(1500, 700, 40, 30) == CVM_OK);
    const size_t one = fake::state().deviceBytes;
    std::vector<std::thread> t;
    std::atomic<int> left{64};
    for (int i = 0; i < 64; i++)
        t.emplace_back([&] {
            for (int k = 0; k < 4; k++) EXPECT(call(1500, 700, 40, 30) == CVM_OK);
            left--;
            while (left > 0) std::this_thread::yield();  // (a thread's end gives nothing back)
        });
    while (left > 0) std::this_thread::yield();
    EXPECT(fake::state().deviceBytes <= (size_t(1) << 30) + (64 << 20));
    for (auto &x : t) x.join();
    EXPECT(one > (16 << 20));
    EXPECT(fake::state().deviceBytes <= (size_t(1) << 30) + (64 << 20));
}

// More shapes than are kept, in turn: no capture pushes another out in vain;
// shapes no longer called make room.
void shapes_in_turn() {
    cvm_set_form(CVM_FORM_EXACT);
    for (int round = 0; round < 12; round++)
        for (int k = 0; k < 40; k++) EXPECT(call(300 + 8 * k, 200, 20, 20) == CVM_OK);
    EXPECT(fake::state().calls["cudaGraphInstantiate"] <= 40);
    EXPECT(graph_launches() > 200);
    for (int k = 0; k < 400; k++) EXPECT(call(300, 200, 20, 20) == CVM_OK);
    const long n = fake::state().calls["cudaGraphInstantiate"];
    for (int k = 0; k < 3; k++) EXPECT(call(1000, 200, 20, 20) == CVM_OK);
    EXPECT(fake::state().calls["cudaGraphInstantiate"] == n + 1);
    for (int k = 0; k < 200; k++)
        for (int i = 0; i < 3; i++) EXPECT(call(640, 220 + k, 20, 20) == CVM_OK);
    EXPECT(fake::state().deviceBytes <= (size_t(1) << 30) + (64 << 20));
}

// Device memory runs out: the idle graphs' goes to the call that needs it.
void memory_given_back() {
    cvm_set_form(CVM_FORM_EXACT);
    for (int i = 0; i < 4; i++) EXPECT(call(700, 300, 40, 30) == CVM_OK);
    EXPECT(graph_launches() == 2);
    const size_t held = fake::state().deviceBytes;
    fake::state().on_call = [&](const std::string &f) {
        return f == "cudaMallocFromPoolAsync" && fake::state().deviceBytes >= held ? cudaErrorMemoryAllocation : cudaSuccess;
    };
    EXPECT(call(500, 300, 40, 30) == CVM_OK);
    EXPECT(fake::state().deviceBytes < held);
}

// Templates are staged beside a staged frame, and small ones beside others.
void staged_templates() {
    cvm_set_form(CVM_FORM_EXACT);
    auto pinned = [&](int w, int h, int tw, int th) {
        size_t before = 0, after = 0;
        for (auto &a : fake::state().pinned) before += a.second;
        for (int i = 0; i < 3; i++) EXPECT(call(w, h, tw, th) == CVM_OK);
        for (auto &a : fake::state().pinned) after += a.second;
        return after - before;
    };
    pinned(100, 90, 10, 10);  // (the thread's own slots)
    EXPECT(pinned(200, 200, 100, 100) > 200 * 200 * 4 + 100 * 100 * 4);
    EXPECT(pinned(1920, 1080, 80, 80) > 80 * 80 * 4);
    EXPECT(pinned(1920, 1080, 181, 181) < 4096);
}

}  // namespace

int main(int argc, char **argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "autotune_off")
        plan_changes_during_the_capture(true);
    else if (what == "plan_published")
        plan_changes_during_the_capture(false);
    else if (what == "errors")
        errors_wait();
    else if (what == "staged_templates")
        staged_templates();
    else if (what == "threads_share")
        threads_share();
    else if (what == "threads_bounded")
        threads_bounded();
    else if (what == "shapes_in_turn")
        shapes_in_turn();
    else if (what == "memory_given_back")
        memory_given_back();
    else
        return 2;
    return 0;
}
