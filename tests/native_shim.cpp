// C entries into the C++ core for tests that the C ABI does not reach: error codes planted on the host
// in place of a device wait that gave up.
#include "../votca_gb300/csrc/handle.cuh"

extern "C" {

// The code a kernel of the handle's FP64 products would leave when a bounded wait gives up.
void shim_plant_error(bse_handle *h, int code) {
  vgb::GemmWorkspace &ws = h->kind == 0 ? h->bse->ws : h->kind == 1 ? h->dense->ws : h->uks->alpha.ws;
  *ws.error_slot() = code;
}

}  // extern "C"
