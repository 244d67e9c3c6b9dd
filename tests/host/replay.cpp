// Replayed one-shot host calls, on the stand-ins of fake_cuda.h.
#include "fake_cuda.h"

#include "../../cvmatch_gb300/csrc/cvm_api.cpp"

namespace {

cudaError_t no_den(const MemberSet &, int, int *, cudaStream_t) { return cudaSuccess; }

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

}  // namespace

namespace cvm {
cudaError_t launch_den_poor(const MemberSet &ms, int n, int *poor, cudaStream_t st) { return no_den(ms, n, poor, st); }
}  // namespace cvm

int main(int argc, char **argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "autotune_off")
        plan_changes_during_the_capture(true);
    else if (what == "plan_published")
        plan_changes_during_the_capture(false);
    else
        return 2;
    return 0;
}
