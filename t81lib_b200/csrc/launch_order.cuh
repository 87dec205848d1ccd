// Order between the kernels that write weights and the decode-sized ones that read weights early.
//
// A streaming product is launched with programmatic stream serialization and fetches its weights before it waits for the kernel
// ahead of it, whose writes are sure to be visible only after that wait.  So the launch behind a kernel that wrote weights does
// without the attribute: it starts once that kernel is complete, and everything later follows it.
#pragma once

#include "common.cuh"

namespace t81b200 {

// Notes that a kernel just launched on the stream writes weights (limbs or codes).
void note_weights_written(cudaStream_t st);
// Whether that is so for a stream on which no streaming product has been launched since; takes the note away.
bool take_weights_written(cudaStream_t st);

}  // namespace t81b200
