#include "fd3_xpass64.cuh"
namespace fd3 {
template int launch_x64<16,16>(const X64Args&, X64Shape);
}
