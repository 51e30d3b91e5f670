// rsbd8g_one_k2.cu - the one-kernel sorts of 16-bit keys.
#include "rsbd8g_onelaunch.cuh"

RSBD8G_DEFINE_ONE(launch_one_k2, uint16_t)
