// profile_events.h — the event pairs of an instrumented render.
#pragma once
#include <cuda_runtime.h>
#include <vector>

namespace ptx_host {

// One region of launches: its kernel class, the events around it, the kernels launched in it (n0:
// the launch count at its start).
struct ProfRec { int cls; cudaEvent_t a, b; int n0, n; };

// The regions of one render.  The list owns its events, so a render that fails leaves none.
class ProfList {
public:
    ProfList() = default;
    ~ProfList() {
        for (ProfRec& r : recs_) {
            if (r.a) cudaEventDestroy(r.a);
            if (r.b) cudaEventDestroy(r.b);
        }
    }
    ProfList(const ProfList&) = delete;
    ProfList& operator=(const ProfList&) = delete;
    void begin(int cls, int n0, cudaStream_t st) {
        recs_.push_back(ProfRec{cls, nullptr, nullptr, n0, 0});
        cudaEventCreate(&recs_.back().a);
        cudaEventCreate(&recs_.back().b);
        cudaEventRecord(recs_.back().a, st);
    }
    void end(int n, cudaStream_t st) {   // of the region begun last, after n launches in all
        cudaEventRecord(recs_.back().b, st);
        recs_.back().n = n - recs_.back().n0;
    }
    // Adds each region's time and launches to its class's (the stream is idle).
    void fold(float* ms, int* launches) const {
        for (const ProfRec& r : recs_) {
            float t = 0.0f;
            cudaEventElapsedTime(&t, r.a, r.b);
            ms[r.cls] += t;
            launches[r.cls] += r.n;
        }
    }

private:
    std::vector<ProfRec> recs_;
};

}  // namespace ptx_host
