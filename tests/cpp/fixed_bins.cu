// The fixed-point FP64 bins (cp3_fixed.cuh) on the host, one call for a whole grid; the number
// of bins that asked for the FP64 path is returned (-1: bad model).
#include <algorithm>
#include <string>
#include <vector>

#include "cp3_fixed.cuh"
#include "cp3_host.hpp"

using namespace cp3;

static constexpr TrigTable kTable = make_trig_table();

// One energy's column of the table (launch_table_fx) from its solved classes.
static void fill_column(const OscParams& p, const std::vector<FxClass>& cls, int2* tab, int2* ext) {
    for (size_t c = 0; c < cls.size(); c++) {
        fx v[13], row[9];
        if (c < 2) {
            fx_rows(cls[c].U, p.w, row);
            for (int f = 0; f < 9; f++) ext[(c ? kFxV1 : kFxV0) + f] = make_int2(row[f].h, row[f].l);
        }
        if (c == 0) {
            fx_coefficients(row, v);
            for (int f = 0; f < 13; f++) ext[kFxVac + f] = make_int2(v[f].h, v[f].l);
        }
        int2* d = tab + c * kFxFields;
        for (int q = 0; q < 2; q++) {
            const long long b = fx_bits(cls[c].rate[q]);
            d[kFxRates + q] = make_int2((int)b, (int)(b >> 32));
        }
        if (c + 1 == cls.size()) break;
        fx R[3][3];
        fx_rotation(cls[c + 1].U, cls[c].U, R);
        for (int f = 0; f < 9; f++) d[f] = make_int2(R[f / 3][f % 3].h, R[f / 3][f % 3].l);
    }
}

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
        }
        fill_column(p, cls, tab.data(), ext);
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

// The bins whose layers are solved in place: densities per segment (poly: the quadratic
// coefficients a, b, c), with nb > 0 production-height averaging (prob [2][3][nc][nb][ne], edges
// in km).
extern "C" int fixed_inline(const double* mix, int knutype, int anti, const double* cz, int nc,
                            const double* en, int ne, const double* radii, const double* a,
                            const double* b, const double* c, const double* ye, int n, int poly,
                            double height_km, int nb, const double* prob, const double* edges, double* out) {
    OscParams p;
    build_osc_params(MixingInput{mix[0], mix[1], mix[2], mix[3], knutype, mix[4], mix[5]}, anti, &p);
    EarthModel model;
    std::string msg;
    TrajectoryTable t;
    if (make_earth_model(radii, a, b, c, ye, n, poly != 0, &model, &msg) ||
        build_trajectories(model, cz, nc, height_km * 1e5, &t, &msg))
        return -1;
    std::vector<double> sh;
    if (nb) production_height_shifts(cz, nc, height_km * 1e5, edges, nb, &sh);
    const longlong2* trig = reinterpret_cast<const longlong2*>(&kTable);
    const FxW w = fx_w(p.w);
    int outside = 0;
    for (int ie = 0; ie < ne; ie++) {
        auto layer = [&](double rho_e, FxClass& k) {
            double u[2][3], dmv[3];
            rotated_layer_f64(&p, en[ie], rho_e, u, dmv);
            fx_class_f64(u, dmv, en[ie], k);
        };
        FxClass k0;
        layer(0.0, k0);
        FxAir air;
        std::memcpy(air.U, k0.U, sizeof air.U);
        fx_rows(k0.U, p.w, air.row);
        fx_coefficients(air.row, air.coef);
        air.rate[0] = k0.rate[0], air.rate[1] = k0.rate[1];
        std::vector<FxClass> cls;
        for (int c = 0; c <= *std::max_element(t.maxlayers.begin(), t.maxlayers.end()) && !poly; c++) {
            cls.emplace_back();
            layer(c ? model.rho[c - 1] * model.ye[c - 1] : 0.0, cls.back());
        }
        std::vector<int2> tab(cls.size() * kFxFields + kFxExtra);
        int2* ext = tab.data() + cls.size() * kFxFields;
        fill_column(p, cls, tab.data(), ext);
        const FxColumn col{tab.data(), ext, 1, (size_t)kFxFields};
        for (int ic = 0; ic < nc; ic++) {
            const double *len = t.len_km.data() + t.offset[ic], *rho = t.rho_e.data() + t.offset[ic];
            auto solve = [&](int l, FxClass& k) { layer(rho[l], k); };
            double* o = out + (size_t)ic * ne + ie;
            const size_t plane = (size_t)nc * ne;
            if (nb == 0) {
                long long P[4];
                outside += !fx_bin_inline(solve, [&]() { return air; }, w, len, t.maxlayers[ic], trig, P);
                fx_store(P, o, plane);
                continue;
            }
            std::vector<double> mid(nb), wid(nb);
            for (int q = 0; q < nb; q++) {
                const double h0 = sh[(size_t)ic * (nb + 1) + q], h1 = sh[(size_t)ic * (nb + 1) + q + 1];
                mid[q] = t.air_cm[ic] == 0.0 ? 0.0 : 0.5 * (h0 + h1) / kKm2Cm;
                wid[q] = t.air_cm[ic] == 0.0 ? 0.0 : (h1 - h0) / kKm2Cm;
            }
            unsigned int bad = 0;
            long long sum[3][3][2] = {};
            unsigned long long total[3] = {};
            for (int part = 0; part < 3; part++) {  // the heights in three shares, as on the device
                FxShift one;
                fx_shift_sums(air.rate, part, 3, nb, prob + (((size_t)anti * 3 * nc + ic) * nb) * ne + ie,
                              (size_t)nc * nb * ne, ne, mid.data(), wid.data(), trig, bad, one);
                for (int j = 0; j < 3; j++) {
                    total[j] += one.total[j];
                    for (int q = 0; q < 6; q++) sum[q >> 1][j][q & 1] += one.value(q >> 1, j, q & 1);
                }
            }
            cfx rows[2][3];
            long long P[3][2];
            fx_check_weights(total, bad);
            if (poly)
                fx_air_rows(solve, [&]() { return air; }, w, len, t.maxlayers[ic], trig, bad, rows);
            else
                fx_air_rows(col, len, t.maxlayers[ic], trig, bad, rows);
            for (int j = 0; j < 3; j++) {
                cfx f[3];
                for (int q = 0; q < 3; q++) f[q] = cfx{fx_split(sum[q][j][0]), fx_split(sum[q][j][1])};
                fx_average(j, rows, air.row, air.rate, len[0], trig, f, bad, P[j]);
            }
            outside += (bad >> 20) != 0;
            for (int j = 0; j < 3; j++) {
                o[(size_t)(3 * j) * plane] = fx_to_double(P[j][0]);
                o[(size_t)(3 * j + 1) * plane] = fx_to_double(P[j][1]);
                o[(size_t)(3 * j + 2) * plane] = fx_to_double((1LL << 62) - P[j][0] - P[j][1]);
            }
        }
    }
    return outside;
}

extern "C" long long fixed_negated(long long v) { return fx_value(fx_neg(fx_split(v))); }

// x as a float pair (0 where it is refused), one over it, and a fixed-point number from a pair.
extern "C" int fixed_pair(double x, float* pair, double* reciprocal) {
    df d;
    if (!fx_float_pair(x, d)) return 0;
    pair[0] = d.hi, pair[1] = d.lo;
    *reciprocal = fx_reciprocal(x, d);
    return 1;
}
extern "C" long long fixed_from_pair(float hi, float lo) { return fx_value(fx_from_pair(hi, lo)); }

// A row's segment lengths (km) and electron densities, as the bins take them; their number.
extern "C" int fixed_segments(double cz, const double* radii, const double* rho, const double* ye, int n,
                              double height_km, double* len, double* rho_e) {
    EarthModel model;
    std::string msg;
    TrajectoryTable t;
    if (make_earth_model(radii, rho, nullptr, nullptr, ye, n, false, &model, &msg) ||
        build_trajectories(model, &cz, 1, height_km * 1e5, &t, &msg))
        return -1;
    const int m = t.maxlayers[0] + 1;
    for (int l = 0; l < m; l++) {
        len[l] = t.len_km[t.offset[0] + l];
        rho_e[l] = l ? model.rho[l - 1] * model.ye[l - 1] : 0.0;
    }
    return m;
}
