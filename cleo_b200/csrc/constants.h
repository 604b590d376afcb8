// constants.h — CLEO's dimensionless scales and physical constants, for device and host.
#pragma once

#include <cstdint>

namespace cleo {

// ---- constants: libs/cleoconstants.hpp:32-118 ----
constexpr double PI = 3.141592653589793238462643383279502884;
constexpr double DC_RGAS_UNIV = 8.314462618;
constexpr double DC_MR_WATER = 0.01801528;
constexpr double DC_MR_DRY = 0.028966216;
constexpr double DC_RGAS_DRY = DC_RGAS_UNIV / DC_MR_DRY;
constexpr double DC_RGAS_V = DC_RGAS_UNIV / DC_MR_WATER;
constexpr double DC_LATENT_V = 2500930.0;
constexpr double DC_CP_DRY = 1004.64;
constexpr double DC_CP_V = 1865.01;
constexpr double DC_C_L = 4192.664;
constexpr double DC_RHO_L = 998.203;
constexpr double DC_RHO_SOL = 2016.5;
constexpr double DC_MR_SOL = 0.05844277;
constexpr double DC_SURFSIGMA = 7.28e-2;
constexpr double W0 = 1.0;
constexpr double TIME0 = 1000.0;
constexpr double COORD0 = TIME0 * W0;
constexpr double VOL0 = COORD0 * COORD0 * COORD0;
constexpr double CP0 = DC_CP_DRY;
constexpr double MR0 = DC_MR_DRY;
constexpr double R0 = 1e-6;
constexpr double P0 = 100000.0;
constexpr double TEMP0 = 273.15;
constexpr double RHO0 = P0 / (CP0 * TEMP0);
constexpr double MASS0 = R0 * R0 * R0 * RHO0;
constexpr double MASS0grams = MASS0 * 1000;
constexpr double F0 = TIME0 / (RHO0 * R0 * R0);
constexpr double Mr_ratio = DC_MR_WATER / DC_MR_DRY;
constexpr double Cp_dry = DC_CP_DRY / CP0;
constexpr double Cp_v = DC_CP_V / CP0;
constexpr double C_l = DC_C_L / CP0;
constexpr double Latent_v = DC_LATENT_V / (TEMP0 * CP0);
constexpr double Rgas_dry = DC_RGAS_DRY / CP0;
constexpr double Rgas_v = DC_RGAS_V / CP0;
constexpr double Rho_l = DC_RHO_L / RHO0;
constexpr double Rho_sol = DC_RHO_SOL / RHO0;
constexpr double Mr_sol = DC_MR_SOL / MR0;
constexpr double IONIC = 2.0;
constexpr double surfconst = 4.0 * DC_SURFSIGMA * PI * R0 * R0;
constexpr uint32_t OOB = 0xFFFFFFFFu;
constexpr double DBLMAX = 1.7976931348623157e308;

}  // namespace cleo
