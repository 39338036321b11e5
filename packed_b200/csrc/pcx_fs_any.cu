// The one-launch four-step kernel's FS_ANY form: any pack widths, short sources.
#include "pcx_fs_launch.cuh"

PCX_FS_FORM(pcx_fs_any, FS_ANY)
