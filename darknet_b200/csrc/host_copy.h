// Parallel copy of ordinary host memory into a page-locked staging ring, chunk by chunk, so that the chunks' transfers to
// the device overlap the copying of the later ones.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#include <memory>

namespace dnb {

class CopyPool;

// The process's pool of copying threads, made by its first holder (make) and joined when the last one lets go.  Null: there is
// none, or no memory for one.  What it uses is made by the uploads that need it.
std::shared_ptr<CopyPool> copy_pool(bool make);

// Uploads `bytes` from pageable `src`, a part of a batch of `of` bytes, to memory `dst` of the current device on `s`.  Returns once src has been read; the
// transfers are then enqueued.  Safe to call from several threads (callers take turns).  NOT_STAGED: nothing was done, the
// driver's own path is the one to take (no pool, or no page-locked memory or events to be had).  Throws nothing.
constexpr int NOT_STAGED = -1;
int upload_staged(CopyPool *pool, void *dst, const void *src, size_t bytes, size_t of, cudaStream_t s);

}  // namespace dnb
