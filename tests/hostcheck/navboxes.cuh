// navboxes.cuh -- navboxes.cu, once in a file that takes several of its users.
#pragma once
#include "navboxes.cu"
