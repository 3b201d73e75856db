// The one-launch closure of small matrices (closure_resident.cu), as closure.cu calls it.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/se.h"

namespace se {
namespace resident {

constexpr int kB = 64;  // block edge, in cells

// Largest C whose tiles all fit 148 SMs at once: 24 x 12 tiles of 64 x 128 cells, two per SM, in
// 16-bit lanes; 21 x 7 tiles of 64 x 192 cells in 32-bit lanes.
constexpr int max_candidates(int lane_bits) { return lane_bits == 16 ? 1536 : 1344; }

// Workspace bytes of the resident closure, 0 where it does not apply.
int64_t workspace_bytes(int C, int lane_bits);

// What a call holds of the GPU while its launch may be in flight: until the call has waited for its
// stream or, with `queued`, until an event behind the launch has come.
struct Hold {
    bool queued;
    void* flights = nullptr;
    void* flight = nullptr;
    explicit Hold(bool queues) : queued(queues) {}
    ~Hold();
    Hold(const Hold&) = delete;
    Hold& operator=(const Hold&) = delete;
};

// Queues the whole closure on s and sets *ran, or leaves *ran false where the resident form does
// not apply (size, workspace, device, a capturing stream, too little room beside those of other
// streams). The first two words of the workspace are the closure's flags, as in closure.cu.
// automatic: 16-bit lanes with the window chosen on the device; where none holds, word kWide is set
// and nothing is written to out. Where the CTAs were not all on the GPU in time, word kArrived has
// bit kGaveWay and nothing is written to out either.
se_status_t run(const uint32_t* d, int64_t ld, int C, uint32_t* out, int64_t ld_out, int lane_bits, uint32_t base,
                bool automatic, void* d_work, int64_t work_bytes, cudaStream_t s, Hold& hold, bool* ran);

constexpr int kWide = 4, kArrived = 5;
constexpr uint32_t kGaveWay = 0x80000000u;

// Whether a launch for C candidates is a single CTA, which cannot give way.
constexpr bool single_cta(int C) { return C <= kB; }

void set_start_limit(uint64_t ns);
void set_wait_limit(uint64_t ns);

}  // namespace resident
}  // namespace se
