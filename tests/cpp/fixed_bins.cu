// The fixed-point FP64 bins (cp3_fixed.cuh) on the host, one call for a whole grid; the number
// of bins that asked for the FP64 path is returned (-1: bad model).
#include <string>
#include <vector>

#include "cp3_fixed.cuh"
#include "cp3_host.hpp"

using namespace cp3;

static constexpr TrigTable kTable = make_trig_table();

extern "C" void fixed_trig(long long* out) { std::memcpy(out, &kTable, sizeof kTable); }

extern "C" int fixed_atmos(const double* mix, int knutype, int anti, const double* cz, int nc,
                           const double* en, int ne, const double* radii, const double* rho,
                           const double* ye, int n, double height_km, int refine, double* out) {
    OscParams p;
    build_osc_params(MixingInput{mix[0], mix[1], mix[2], mix[3], knutype, mix[4], mix[5]}, anti, &p);
    EarthModel model;
    std::string msg;
    TrajectoryTable t;
    if (make_earth_model(radii, rho, nullptr, nullptr, ye, n, false, &model, &msg) ||
        build_trajectories(model, cz, nc, height_km * 1e5, &t, &msg))
        return -1;
    int ncls = 1, outside = 0;
    for (int m : t.maxlayers) ncls = m + 1 > ncls ? m + 1 : ncls;
    std::vector<int2> tab((size_t)ncls * kFxFields + kFxExtra);
    int2* ext = tab.data() + (size_t)ncls * kFxFields;
    std::vector<FxClass> cls(ncls);
    for (int ie = 0; ie < ne; ie++) {
        for (int c = 0; c < ncls; c++) {
            // the FP64 vectors stand for the device's double-float ones, rounded as those are
            double u[2][3], dmv[3];
            const double E = en[ie], rho_e = c ? model.rho[c - 1] * model.ye[c - 1] : 0.0;
            rotated_layer_f64(&p, E, rho_e, u, dmv);
            fx_class_f64(u, dmv, E, cls[c]);
            if (refine) {
                for (int i = 0; i < 3; i++)
                    for (int k = 1; k < 3; k++)
                        cls[c].U[i][k] = fx_split((fx_from_double(u[k - 1][i]) >> 16) * 65536);  // 2^-46
                fx_third(cls[c].U);
                if (!fx_refine(&p, E, 1.0 / E, rho_e, cls[c])) fx_class_f64(u, dmv, E, cls[c]);
            }
            fx v[13], row[9];
            if (c < 2) {
                fx_rows(cls[c].U, p.w, row);
                for (int f = 0; f < 9; f++) ext[(c ? kFxV1 : kFxV0) + f] = make_int2(row[f].h, row[f].l);
            }
            if (c == 0) {
                fx_coefficients(row, v);
                for (int f = 0; f < 13; f++) ext[kFxVac + f] = make_int2(v[f].h, v[f].l);
            }
        }
        for (int c = 0; c < ncls; c++) {
            int2* d = tab.data() + (size_t)c * kFxFields;
            for (int q = 0; q < 2; q++) {
                const long long b = fx_bits(cls[c].rate[q]);
                d[kFxRates + q] = make_int2((int)b, (int)(b >> 32));
            }
            if (c + 1 == ncls) break;
            fx R[3][3];
            fx_rotation(cls[c + 1].U, cls[c].U, R);
            for (int f = 0; f < 9; f++) d[f] = make_int2(R[f / 3][f % 3].h, R[f / 3][f % 3].l);
        }
        const FxColumn col{tab.data(), ext, 1, (size_t)kFxFields};
        for (int ic = 0; ic < nc; ic++) {
            long long P[4];
            outside += !fx_bin(col, t.len_km.data() + t.offset[ic], t.maxlayers[ic],
                               reinterpret_cast<const longlong2*>(&kTable), P);
            fx_store(P, out + (size_t)ic * ne + ie, (size_t)nc * ne);
        }
    }
    return outside;
}
