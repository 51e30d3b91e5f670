// rsbd8g_one_k1.cu - the one-kernel sorts of 8-bit keys.
#include "rsbd8g_onelaunch.cuh"

RSBD8G_DEFINE_ONE(launch_one_k1, uint8_t)
