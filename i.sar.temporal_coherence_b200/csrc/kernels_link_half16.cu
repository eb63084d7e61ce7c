/* The half-warp link kernel for stacks of up to 16 dates: the code of
 * kernels_link_half.cu with matrices of 16 columns, one row per lane.
 */
#define TC_LINK_COLS 16
#include "kernels_link_half.cu"
