// Fleets' host logic, on the stand-ins of fake_cuda.h.
#include "fake_cuda.h"

#include "../../cvmatch_gb300/csrc/cvm_api.cpp"

namespace cvm {
cudaError_t launch_den_poor(const MemberSet &, int, int *, cudaStream_t) { return cudaSuccess; }
}  // namespace cvm

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

// Plans are tuned apart for the two sources of den.
void tuned_per_source() {
    char buf[1 << 14];
    for (int mode : {CVM_STATS_KERNEL, CVM_STATS_EPILOGUE, CVM_STATS_KERNEL}) {
        cvm_fleet *f = fleet(8, 20);
        EXPECT(cvm_fleet_set_stats(f, mode) == CVM_OK);
        EXPECT(find(f) == CVM_OK);
    }
    cvm_autotune_report(buf, sizeof buf);
    int n = 0;
    for (const char *p = buf; (p = strstr(p, "\"fleet\":true")); p++) n++;
    EXPECT(n == 2);
}

}  // namespace

int main(int argc, char **argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "tuned_per_source")
        tuned_per_source();
    else
        return 2;
    return 0;
}
