// Error reporting shared by the host translation units of libakb.
#pragma once

#include <cstdint>
#include <string>

struct akb_model;

namespace akb {
// records msg as the thread's last error and returns code
int fail(int code, const std::string &msg);

// the fused step's part of akb_estimate_device_bytes and (of several instances)
// akb_estimate_batch_device_bytes
int64_t plan_device_bytes(int et, int rule, int law, int precision, int64_t N, int64_t E,
                          int ninst);
// before initFull: no plan of the fused step is built
void leave_out_plan(akb_model *m);
}  // namespace akb
