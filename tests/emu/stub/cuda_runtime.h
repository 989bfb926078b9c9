// TEST INFRASTRUCTURE: stands in for the CUDA runtime header when the kernels' device
// code is compiled for the host (tests/emu/simt_emu.cpp).
#pragma once
#include "../simt.h"
