// The one-launch four-step kernel's FS_OUT form: forward into a permuted order.
#include "pcx_fs_launch.cuh"

PCX_FS_FORM(pcx_fs_out, FS_OUT)
