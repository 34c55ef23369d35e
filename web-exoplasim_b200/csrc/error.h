// Errors of the engine: a C-ABI status code and its message, thrown inside
// the library and turned into the call's return value at its C entry.
#pragma once
#include <cuda_runtime_api.h>

#include <stdexcept>
#include <string>

#include "../../include/exogcm.h"

namespace exogcm {

struct Error : std::runtime_error {
  int code;
  Error(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};

inline void check(cudaError_t e, const char* what) {
  if (e != cudaSuccess) throw Error(EXOGCM_EDEVICE, std::string(what) + ": " + cudaGetErrorString(e));
}

}  // namespace exogcm
