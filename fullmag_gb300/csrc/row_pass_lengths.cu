// row_pass_lengths.cu -- row pass kernels of a few x half lengths; compiled once per group
// (FM_GROUP, build.py), so that the groups build in parallel.
#include "row_pass.cuh"

namespace fm {

#if FM_GROUP == 0
#define FM_GROUP_LENGTHS(F) F(16) F(20) F(24)
#elif FM_GROUP == 1
#define FM_GROUP_LENGTHS(F) F(28) F(32) F(40)
#elif FM_GROUP == 2
#define FM_GROUP_LENGTHS(F) F(48) F(56) F(64)
#elif FM_GROUP == 3
#define FM_GROUP_LENGTHS(F) F(80) F(96) F(112)
#elif FM_GROUP == 4
#define FM_GROUP_LENGTHS(F) F(128) F(160) F(192)
#elif FM_GROUP == 5
#define FM_GROUP_LENGTHS(F) F(224) F(256) F(320)
#elif FM_GROUP == 6
#define FM_GROUP_LENGTHS(F) F(384) F(448) F(512)
#elif FM_GROUP == 7
#define FM_GROUP_LENGTHS(F) F(640) F(768)
#else
#define FM_GROUP_LENGTHS(F) F(896) F(1024)
#endif

#define FM_ENTRY(n) \
    template <> \
    const RowKernels &row_kernels_of<n>() { \
        static const RowKernels k = row_kernels<n>(); \
        return k; \
    }
FM_GROUP_LENGTHS(FM_ENTRY)

}  // namespace fm
