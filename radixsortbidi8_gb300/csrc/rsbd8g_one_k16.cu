// rsbd8g_one_k16.cu - the one-kernel sorts of 128-bit keys.
#include "rsbd8g_onelaunch.cuh"

RSBD8G_DEFINE_ONE(launch_one_k16, rsbd8g::KeyU128)
