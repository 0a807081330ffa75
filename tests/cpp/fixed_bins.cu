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
                           const double* ye, int n, double height_km, double* out) {
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
            double u[2][3], dmv[3], u0[3];
            rotated_layer_f64(&p, en[ie], c ? model.rho[c - 1] * model.ye[c - 1] : 0.0, u, dmv);
            fx_class(u, dmv, en[ie], cls[c], u0);
            fx v[13];
            if (c < 2) {
                fx_rows(u0, u, p.w, v);
                for (int f = 0; f < 9; f++) ext[(c ? kFxV1 : kFxV0) + f] = make_int2(v[f].h, v[f].l);
            }
            if (c == 0) {
                fx_vacuum(u, p.w, v);
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
