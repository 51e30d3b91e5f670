// rsbd8g_one_k8.cu - the one-kernel sorts of 64-bit keys.
#include "rsbd8g_onelaunch.cuh"

RSBD8G_DEFINE_ONE(launch_one_k8, uint64_t)
