/* Calls between the library's own parts (not part of the C ABI). */
#ifndef MICSA_INTERNAL_H
#define MICSA_INTERNAL_H

#include "micsa.h"

#ifdef __cplusplus
extern "C" {
#endif

/* micsa_create for a context that runs side by side with others of the same
 * job or server: its launch shape is chosen among those that leave the SMs to
 * the other contexts' kernels while they wait. */
int micsa_create_shared(const micsa_config *cfg, micsa_ctx **out);

#ifdef __cplusplus
}
#endif
#endif
