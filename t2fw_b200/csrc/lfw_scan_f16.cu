#define T2FW_LFW_SCAN_DEFINE
#include "lfw_scan.cuh"

namespace t2fw {
namespace lfw_scan {
T2FW_LFW_SCAN_TYPE(__half)
}  // namespace lfw_scan
}  // namespace t2fw
