// rsbd8g_one_x87.cu - the one-kernel sorts of x87 keys.
#include "rsbd8g_onelaunch.cuh"

RSBD8G_DEFINE_ONE(launch_one_x87, rsbd8g::KeyX87)
