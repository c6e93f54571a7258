// explicit instantiations of the vy_gemm kernels whose epilogue is the staged fp32 one (see gemm_kernel.cuh)
#include "gemm_kernel.cuh"
namespace vy {
template int launch_gemm<float, 32, false, false, false, WB_F32>(const VyGemm*, const GemmDev&);
template int launch_gemm<float, 64, false, false, false, WB_F32>(const VyGemm*, const GemmDev&);
template int launch_gemm<float, 128, false, false, false, WB_F32>(const VyGemm*, const GemmDev&);
template int launch_gemm<float, 192, false, false, false, WB_F32>(const VyGemm*, const GemmDev&);
template int launch_gemm<float, 256, false, false, false, WB_F32>(const VyGemm*, const GemmDev&);
}  // namespace vy
