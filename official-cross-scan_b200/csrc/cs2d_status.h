// The device-side status word of the library (0 = fine).  A kernel that gives up on a bounded wait records why here
// instead of spinning; the host reads and clears it through cs2d_device_status().
#pragma once

#include <cstddef>
#include <cstdio>

namespace cs2d {

enum { ERR_BULK_COPY_TIMEOUT = 1, ERR_STAGE_TIMEOUT = 2, ERR_WORKER_TIMEOUT = 4 };

// What the word says.
inline void status_text(char *text, size_t size, int status) {
    snprintf(text, size, "a kernel gave up on a bounded wait (status %d:%s%s%s); its outputs are invalid", status,
             (status & ERR_BULK_COPY_TIMEOUT) ? " bulk copy" : "", (status & ERR_STAGE_TIMEOUT) ? " staging warps" : "",
             (status & ERR_WORKER_TIMEOUT) ? " row workers" : "");
}

}  // namespace cs2d
