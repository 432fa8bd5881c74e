// populate() of ps3d_gb300/csrc/host_pages.h behind a C entry.
#include "host_pages.h"

extern "C" int host_populate(void *p, unsigned long long bytes) { return ps3d::populate(p, bytes); }
