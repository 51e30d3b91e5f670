// rsbd8g_one_k4.cu - the one-kernel sorts of 32-bit keys.
#include "rsbd8g_onelaunch.cuh"

RSBD8G_DEFINE_ONE(launch_one_k4, uint32_t)
