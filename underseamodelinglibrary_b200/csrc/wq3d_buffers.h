/*
 * wq3d_buffers.h -- device buffers that change size together.
 */
#pragma once

#include <cstddef>
#include <vector>

namespace wq3d {

/* a buffer (null: not made yet), its new size in bytes, and the new buffer */
struct Resize {
    void* old;
    size_t bytes;
    void* fresh;
};

/* Allocates every new buffer, or none: when one fails, those made before it
 * are released again and the old ones stay as they are, so whoever holds
 * their addresses (a captured graph, a descriptor) still may use them.
 * alloc(void** out, size_t bytes) returns 0 or an error code, which is
 * returned; release(void*) takes what alloc gave. */
template <class Alloc, class Release>
int make_all(std::vector<Resize>& buffers, Alloc alloc, Release release) {
    for (size_t k = 0; k < buffers.size(); ++k) {
        buffers[k].fresh = nullptr;
        const int rc = alloc(&buffers[k].fresh, buffers[k].bytes);
        if (rc) {
            for (size_t j = 0; j < k; ++j) {
                release(buffers[j].fresh);
                buffers[j].fresh = nullptr;
            }
            return rc;
        }
    }
    return 0;
}

}  // namespace wq3d
