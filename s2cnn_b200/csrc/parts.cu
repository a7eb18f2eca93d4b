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
#include "so3_cluster_kernels.h"
#include "so3_mid_kernels.h"
#include "s2_kernels.h"
#include "so3_small_kernels.h"
#include "so3_mm_tc.h"

namespace s2c {

#define S2C_LENGTH(N)                                                                                \
  template int launch_so3_inv_fused<N>(long, int, size_t, stream_t, const InvFusedParams&);          \
  template int launch_so3_fwd_fused<N>(long, int, size_t, stream_t, const FwdFusedParams&);          \
  template int launch_so3_inv_cl<N>(long, int, size_t, stream_t, const ClInvParams&);                \
  template int launch_so3_fwd_cl<N>(long, int, size_t, stream_t, const ClFwdParams&);                \
  template int launch_so3_relay_cl<N>(long, int, size_t, stream_t, const ClRelayParams&);
#define S2C_RELAY(N) \
  template int launch_so3_relay_fused<N>(long, int, size_t, stream_t, const RelayParams&);
#define S2C_MID(N)                                                                  \
  template int launch_so3_fwd_mid<N>(long, int, size_t, stream_t, const MidParams&); \
  template int launch_so3_inv_mid<N>(long, int, size_t, stream_t, const MidParams&);
#define S2C_SMALL(N)                                                                     \
  template int launch_so3_fwd_small<N>(long, int, size_t, stream_t, const SmallParams&);   \
  template int launch_so3_inv_small<N>(long, int, size_t, stream_t, const SmallParams&);   \
  template int launch_so3_relay_small<N>(long, int, size_t, stream_t, const SmallParams&);
#define S2C_TC_OP(OP) \
  template int launch_so3_mm_tc<OP>(const char*, long, bool, bool, stream_t, const MmTcParams&);

#define S2C_S2(N)                                                                          \
  template int launch_s2_fwd_fused<N>(long, int, size_t, stream_t, const S2FwdFusedParams&); \
  template int launch_s2_fwd_rows<N>(long, int, size_t, stream_t, const S2RowsParams&);      \
  template int launch_s2_inv_rows<N>(long, int, size_t, stream_t, const S2RowsParams&);

#if S2C_PART == 0
S2C_LENGTH(32)
#elif S2C_PART == 1
S2C_LENGTH(30)
#elif S2C_PART == 2
S2C_LENGTH(28) S2C_LENGTH(2) S2C_RELAY(2) S2C_LENGTH(4) S2C_RELAY(4)
#elif S2C_PART == 3
S2C_LENGTH(26) S2C_LENGTH(6) S2C_RELAY(6)
#elif S2C_PART == 4
S2C_LENGTH(24) S2C_LENGTH(8) S2C_RELAY(8) S2C_LENGTH(10) S2C_RELAY(10)
#elif S2C_PART == 5
S2C_LENGTH(22) S2C_LENGTH(12) S2C_RELAY(12) S2C_LENGTH(14) S2C_RELAY(14)
#elif S2C_PART == 6
S2C_LENGTH(20) S2C_RELAY(20) S2C_LENGTH(16) S2C_RELAY(16) S2C_LENGTH(18) S2C_RELAY(18)
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
#elif S2C_PART == 12
S2C_S2(2) S2C_S2(4) S2C_S2(18) S2C_S2(20) S2C_S2(34) S2C_S2(36) S2C_S2(50) S2C_S2(52) S2C_S2(66)
S2C_S2(68) S2C_S2(88) S2C_S2(90) S2C_S2(108) S2C_S2(110) S2C_S2(128)
#elif S2C_PART == 13
S2C_S2(6) S2C_S2(16) S2C_S2(22) S2C_S2(32) S2C_S2(38) S2C_S2(48) S2C_S2(54) S2C_S2(64) S2C_S2(70)
S2C_S2(84) S2C_S2(92) S2C_S2(104) S2C_S2(112) S2C_S2(126)
#elif S2C_PART == 14
S2C_S2(8) S2C_S2(14) S2C_S2(24) S2C_S2(30) S2C_S2(40) S2C_S2(46) S2C_S2(56) S2C_S2(62) S2C_S2(72)
S2C_S2(80) S2C_S2(96) S2C_S2(102) S2C_S2(114) S2C_S2(124)
#elif S2C_PART == 15
S2C_S2(10) S2C_S2(12) S2C_S2(26) S2C_S2(28) S2C_S2(42) S2C_S2(44) S2C_S2(58) S2C_S2(60) S2C_S2(76)
S2C_S2(78) S2C_S2(98) S2C_S2(100) S2C_S2(116) S2C_S2(120)
#elif S2C_PART == 16
S2C_SMALL(32) S2C_SMALL(30) S2C_SMALL(24) S2C_SMALL(18)
#elif S2C_PART == 17
S2C_SMALL(28) S2C_SMALL(26) S2C_SMALL(22) S2C_SMALL(20)
#endif

}  // namespace s2c
