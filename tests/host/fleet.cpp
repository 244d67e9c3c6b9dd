// Fleets' host logic, on the stand-ins of fake_cuda.h.
#include "fake_cuda.h"

#include "../../cvmatch_gb300/csrc/cvm_api.cpp"

namespace {

std::vector<uint8_t> frame(1920 * 1080 * 4);

cvm_fleet *fleet(int n, int size) {
    std::vector<uint8_t> tpl((size_t)size * size * 4);
    tpl[5] = 9;
    std::vector<cvm_matcher *> ms(n);
    for (auto &m : ms) EXPECT(cvm_matcher_new(tpl.data(), 4 * size, size, size, 4, &m) == CVM_OK);
    cvm_fleet *f;
    EXPECT(cvm_fleet_new(ms.data(), n, &f) == CVM_OK);
    EXPECT(cvm_fleet_set_form(f, CVM_FORM_FAST) == CVM_OK);
    return f;
}

int find(cvm_fleet *f, int w = 640, int h = 480) {
    std::vector<cvm_result> r(f->ms.size());
    return cvm_fleet_find_all(f, frame.data(), 4 * w, w, h, r.data());
}

// Plans are timed once, whatever source of den the fleets have.
void tuned_once() {
    char buf[1 << 14];
    for (int mode : {CVM_STATS_KERNEL, CVM_STATS_EPILOGUE, CVM_STATS_KERNEL}) {
        cvm_fleet *f = fleet(8, 20);
        EXPECT(cvm_fleet_set_stats(f, mode) == CVM_OK);
        EXPECT(find(f) == CVM_OK);
    }
    cvm_autotune_report(buf, sizeof buf);
    int n = 0;
    for (const char *p = buf; (p = strstr(p, "\"fleet\":true")); p++) n++;
    EXPECT(n == 1);
    EXPECT(fake::state().calls["inv_rows_table"] == 1);  // the on-demand fleet's own call, no trial
}

// Contents as the device would report them.
enum Content { camera, black, icons, gradient };
void show(Content c, int n, int size, int w = 640, int h = 480) {
    const double share[] = {0.04, 0.0, 0.6, 1.0};
    const unsigned long long steps = n * (((long long)(w - size + 1) * (h - size + 1) + 31) / 32);
    fake::state().poor = c == icons ? 40 : 0;
    fake::state().formed = [=](int source) { return source == CVM_STATS_EPILOGUE ? (unsigned long long)(share[c] * steps) : 0; };
}

// Calls whose den came on demand, of n.
int on_demand(cvm_fleet *f, int n) {
    int k = 0;
    for (int i = 0; i < n; i++) {
        const long before = fake::state().calls["inv_rows_table"];
        EXPECT(find(f) == CVM_OK);
        k += fake::state().calls["inv_rows_table"] > before;
    }
    return k;
}

void the_choice_follows() {
    cvm_set_autotune(0);
    for (Content first : {camera, black}) {
        cvm_fleet *f = fleet(32, 20);
        show(first, 32, 20);
        EXPECT(on_demand(f, 1) == 1);
        show(icons, 32, 20);
        EXPECT(on_demand(f, 1000) <= 8);
        show(camera, 32, 20);
        EXPECT(on_demand(f, 1000) >= 900);
        show(icons, 32, 20);
        EXPECT(on_demand(f, 1000) <= 200);
    }
    cvm_fleet *f = fleet(32, 20);
    show(gradient, 32, 20);
    EXPECT(on_demand(f, 4000) <= 60);
    show(camera, 32, 20);
    EXPECT(on_demand(f, 10000) >= 5000);
    // a small fleet starts with the kernel and is tried on demand, briefly
    f = fleet(2, 20);
    show(gradient, 2, 20);  // (all its steps form den)
    EXPECT(on_demand(f, 1) == 0);
    EXPECT(on_demand(f, 4000) <= 60);
    // said once, it stays
    f = fleet(8, 20);
    EXPECT(cvm_fleet_set_stats(f, CVM_STATS_EPILOGUE) == CVM_OK);
    show(icons, 8, 20);
    EXPECT(on_demand(f, 100) == 100);
}

// A first call inside a caller's capture samples nothing; a later call does.
void captured_first() {
    cvm_set_autotune(0);
    cvm_fleet *f = fleet(32, 20);
    show(icons, 32, 20);
    cvm_result r[32];
    cudaStream_t st;
    cudaStreamCreateWithFlags(&st, 0);
    cudaStreamBeginCapture(st, cudaStreamCaptureModeGlobal);
    EXPECT(cvm_fleet_find_all_device(f, frame.data(), 4 * 640, 640, 480, r, st) == CVM_OK);
    cudaGraph_t g;
    cudaStreamEndCapture(st, &g);
    EXPECT(fake::state().calls["den_poor"] == 0 && fake::state().calls["tally"] == 0);
    EXPECT(on_demand(f, 100) <= 4);
}

// A stream's graphs hold their fleet's spectra: they outlive the fleet's use at
// another size and in another form.
void a_streams_spectra() {
    cvm_set_autotune(0);
    cvm_fleet *f = fleet(8, 20);
    cvm_stream *s;
    EXPECT(cvm_stream_new(f, nullptr, 640, 480, &s) == CVM_OK);
    const std::map<char *, size_t> kept = fake::state().device;
    EXPECT(find(f, 320, 200) == CVM_OK);
    EXPECT(cvm_fleet_set_form(f, CVM_FORM_EXACT) == CVM_OK && find(f, 320, 200) == CVM_OK);
    for (const auto &a : kept) EXPECT(fake::inside(a.first, a.second));
    cvm_stream_free(s);
    cvm_fleet_free(f);
}

// A stream's graphs follow what its fleet chooses on the frames pushed, also
// when the fleet goes on to other sizes.
void a_stream_follows() {
    cvm_set_autotune(0);
    cvm_fleet *f = fleet(32, 20);
    show(camera, 32, 20);
    cvm_stream *s;
    EXPECT(cvm_stream_new(f, nullptr, 640, 480, &s) == CVM_OK);
    std::vector<cvm_result> r(32);
    auto pushed = [&](int n) {
        const long before = fake::state().calls["inv_rows_table"], graphs = fake::state().calls["cudaGraphLaunch"];
        for (int i = 0; i < n; i++) {
            EXPECT(cvm_stream_push(s, frame.data(), 4 * 640) == CVM_OK);
            EXPECT(cvm_stream_pull(s, r.data(), nullptr, nullptr) == CVM_OK);
        }
        EXPECT(fake::state().calls["cudaGraphLaunch"] - graphs > n * 8 / 10);
        return fake::state().calls["inv_rows_table"] - before;
    };
    pushed(100);
    show(icons, 32, 20);
    pushed(100);
    EXPECT(pushed(1000) == 0);
    show(camera, 32, 20);
    pushed(400);
    EXPECT(pushed(1000) > 0);  // the looks, and a capture before them
    int graphed = 0, launches = 0;
    EXPECT(cvm_stream_info(s, &graphed, &launches) == CVM_OK && graphed);
    // the fleet is used at another size meanwhile
    EXPECT(find(f, 320, 200) == CVM_OK);
    show(icons, 32, 20);
    pushed(200);
    EXPECT(find(f, 320, 200) == CVM_OK);
    pushed(200);
    cvm_stream_free(s);
}

// Only a call that times plans waits for the caller's stream.
void no_waiting() {
    cvm_result r[8];
    cudaStream_t st;
    cudaStreamCreateWithFlags(&st, 0);
    auto waits = [&](cvm_fleet *f) {
        fake::state().synced.clear();
        EXPECT(cvm_fleet_find_all_device(f, frame.data(), 4 * 640, 640, 480, r, st) == CVM_OK);
        return fake::state().synced.count(st) > 0;
    };
    EXPECT(!waits(fleet(3, 20)));                      // too few to tune
    EXPECT(waits(fleet(8, 20)));                       // tunes
    EXPECT(!waits(fleet(8, 20)));                      // tuned before
    cvm_set_autotune(0);
    EXPECT(!waits(fleet(7, 21)));
}

// Without coherent access to pageable memory a kernel reads a caller's frame
// only when all of it is page-locked.
void partly_locked() {
    auto &st = fake::state();
    st.pageable = 0;
    cvm_set_autotune(0);
    cvm_fleet *f = fleet(3, 20);
    cvm_stream *s;
    EXPECT(cvm_stream_new(f, nullptr, 640, 480, &s) == CVM_OK);
    std::vector<cvm_result> r(3);
    for (int locked : {0, 1, 2}) {  // none, half, all of the frame
        st.lockedFrom = reinterpret_cast<const char *>(frame.data());
        st.lockedTo = st.lockedFrom + (size_t)locked * 640 * 480 * 2;
        const long before = st.calls["ingest"];
        EXPECT(cvm_stream_push(s, frame.data(), 4 * 640) == CVM_OK);
        EXPECT(cvm_stream_pull(s, r.data(), nullptr, nullptr) == CVM_OK);
        EXPECT(find(f) == CVM_OK);
        EXPECT(st.calls["ingest"] - before == (locked == 2 ? 2 : 0));
    }
    cvm_stream_free(s);
}

}  // namespace

int main(int argc, char **argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "tuned_once")
        tuned_once();
    else if (what == "the_choice_follows")
        the_choice_follows();
    else if (what == "a_streams_spectra")
        a_streams_spectra();
    else if (what == "a_stream_follows")
        a_stream_follows();
    else if (what == "no_waiting")
        no_waiting();
    else if (what == "partly_locked")
        partly_locked();
    else if (what == "captured_first")
        captured_first();
    else
        return 2;
    return 0;
}
