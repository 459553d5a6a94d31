// Sizes of the buffers that the host code lays out (test infrastructure, never
// part of the library).
#include "../../cadise_gb300/csrc/internal.h"

#include <cstdint>

extern "C" {

uint64_t ly_wavefront_bytes(uint64_t paths, int rows) {
    cg::WfBuffers w{};
    return cg::wf_layout(nullptr, size_t(paths), rows, &w);
}

}  // extern "C"
