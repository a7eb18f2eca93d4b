// The kernel families with many instantiations, compiled in parallel: build.py compiles this file once
// per part with -DS2C_SPLIT -DS2C_PART=<part> and links the objects with lib.cu's.
#include "../../include/s2cnn_b200.h"

#include <algorithm>

#include "backend.h"
#include "host_math.h"
#include "tables.h"
#include "fft_device.h"
#include "so3_kernels.h"
#include "so3_fused_kernels.h"
#include "so3_relay_kernels.h"
#include "so3_mid_kernels.h"
#include "so3_mm_tc.h"

namespace s2c {

#define S2C_LENGTH(N)                                                                                \
  template int launch_so3_inv_fused<N>(long, int, size_t, stream_t, const InvFusedParams&);          \
  template int launch_so3_fwd_fused<N>(long, int, size_t, stream_t, const FwdFusedParams&);          \
  template int launch_so3_relay_fused<N>(long, int, size_t, stream_t, const RelayParams&);
#define S2C_MID(N)                                                                  \
  template int launch_so3_fwd_mid<N>(long, int, size_t, stream_t, const MidParams&); \
  template int launch_so3_inv_mid<N>(long, int, size_t, stream_t, const MidParams&);
#define S2C_TC_OP(OP) \
  template int launch_so3_mm_tc<OP>(const char*, long, bool, bool, stream_t, const MmTcParams&);

#if S2C_PART == 0
S2C_LENGTH(32)
#elif S2C_PART == 1
S2C_LENGTH(30)
#elif S2C_PART == 2
S2C_LENGTH(28) S2C_LENGTH(2) S2C_LENGTH(4)
#elif S2C_PART == 3
S2C_LENGTH(26) S2C_LENGTH(6)
#elif S2C_PART == 4
S2C_LENGTH(24) S2C_LENGTH(8) S2C_LENGTH(10)
#elif S2C_PART == 5
S2C_LENGTH(22) S2C_LENGTH(12) S2C_LENGTH(14)
#elif S2C_PART == 6
S2C_LENGTH(20) S2C_LENGTH(16) S2C_LENGTH(18)
#elif S2C_PART == 7
S2C_TC_OP(kTcFwd) S2C_TC_OP(kTcGradX)
#elif S2C_PART == 8
S2C_TC_OP(kTcGradY) S2C_TC_OP(kTcPlainCC) S2C_TC_OP(kTcPlainSC)
#elif S2C_PART == 9
S2C_MID(34) S2C_MID(38) S2C_MID(46) S2C_MID(58) S2C_MID(62)
#elif S2C_PART == 10
S2C_MID(36) S2C_MID(40) S2C_MID(42) S2C_MID(44) S2C_MID(48)
#elif S2C_PART == 11
S2C_MID(50) S2C_MID(52) S2C_MID(54) S2C_MID(56) S2C_MID(60)
#endif

}  // namespace s2c
