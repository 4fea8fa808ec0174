// Host build of OncePerDevice (qcware_unitair_gb300/csrc/once.h).
#include "once.h"

static gbsv::OncePerDevice once;
static int calls[128];

// Runs the device's work, which returns `rc`; returns what the call returns.
extern "C" int once_run(int device, int rc) {
  return once(device, [&]() {
    ++calls[device];
    return rc;
  });
}
extern "C" int once_calls(int device) { return calls[device]; }
