// What launch_failure_test.cu and its runtime (fake_cuda_runtime.cpp) share.
#pragma once

namespace fake {
extern int launches;    // launches asked for
extern int reject;      // number of the launch to reject
extern bool capturing;  // streams are being captured: nothing runs
void launched(int k, void** args);  // the test's model of launch k
} // namespace fake
