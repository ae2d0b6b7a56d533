// The regions' intensities, shared by the integration and its adjoint.
#pragma once

#include "internal.cuh"

// loi_Planck, SOAP_integration.cu:205-212
__device__ __forceinline__ double soap_planck(double lambda0, double temp) {
    double c = 299792458.;
    double h = 6.62606896e-34;
    double k_b = 1.380e-23;
    double scale = 1e-10;
    return 2 * h * pow(c, 2) * 1. / pow(lambda0 * scale, 5) * 1. / (exp((h * c) / (lambda0 * k_b * temp * scale)) - 1);
}

// cell intensity I at pixel j (fast_intensity / fast_intensity_fac / the solar form)
__device__ __forceinline__ double soap_intensity(int type, double T, double lbk, double lj, double ssed, double fsed,
                                                 int solar, int t_norm_fac) {
    if (type == 0) {
        // fast_intensity with T_norm = (int)T: the Planck ratio is exactly 1 for whole temperatures
        const int tn = (int)T;
        const double ratio = ((double)tn == T) ? 1.0 : soap_planck(lj, T) / soap_planck(lj, (double)tn);
        return __dmul_rn(ratio, ssed);
    }
    if (solar) {
        const double ratio = ((double)t_norm_fac == T) ? 1.0 : soap_planck(lj, T) / soap_planck(lj, (double)t_norm_fac);
        return __dmul_rn(ratio, fsed);
    }
    return __dmul_rn(__dadd_rn(1.0, lbk), fsed);
}
