// Internal types shared by the host launchers and the kernels.
#pragma once
#include <stdint.h>

#include "../../include/pyexner_b200.h"

#define PXB_MAX_SED 8
