// Address of a network's tcgen05 timeout flag (device memory), for the test
// that sets it on the host's behalf.  handle: an ek_unet, whose first member is
// the network.
#include <memory>

#include "ek_unet.h"

namespace {
int *ek::UNet::*flag_member();
template <int *ek::UNet::*M>
struct Open {
  friend int *ek::UNet::*flag_member() { return M; }
};
// an explicit instantiation may name a private member
template struct Open<&ek::UNet::tc_err_>;
}  // namespace

extern "C" void *unet_timeout_flag(void *handle) {
  return reinterpret_cast<std::unique_ptr<ek::UNet> *>(handle)->get()->*flag_member();
}
