// An allocation that memory kept for speed alone may stand in the way of.
#pragma once

#include "../../include/lattice_gpu.h"

namespace lat {

// alloc(), and again after each release() that gave something back, as long as it
// fails for want of memory.  The status of the last try.
template <class Alloc, class... Release>
int alloc_or_release(Alloc&& alloc, Release&&... release)
{
    int rc = alloc();
    ((rc = rc == LAT_ERR_NOMEM && release() ? alloc() : rc), ...);
    return rc;
}

}  // namespace lat
