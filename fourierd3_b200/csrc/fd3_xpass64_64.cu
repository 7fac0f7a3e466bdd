#include "fd3_xpass64.cuh"
namespace fd3 {
template int launch_x64<8,8>(const X64Args&, X64Shape);
}
