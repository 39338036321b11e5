// The one-launch four-step kernel's FS_IN form: inverse from a permuted order.
#include "pcx_fs_launch.cuh"

PCX_FS_FORM(pcx_fs_in, FS_IN)
