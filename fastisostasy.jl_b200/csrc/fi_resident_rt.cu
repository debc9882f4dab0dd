// fi_resident_rt.cu -- the resident step kernel for any radix schedule, its shared-memory
// layout and the choice among its builds.
#include "fi_resident.cuh"

namespace fi {

bool res_layout(int nx, int ny, int Mx, int My, int K, int same_plan, int h, int B_cols, int ncols, int h_conv,
                int B_conv, int grid, size_t budget, ResLayout* L) {
    const size_t rowf = (size_t)nx * 4, capU = capU_of(h), npi = (capU + 1) / 2, np = (h + 1) / 2;
    size_t off = 0;
    auto take = [&](size_t bytes) -> int {
        const int o = (int)off;
        off += al16(bytes);
        return o;
    };
    L->twx = take((size_t)nx * 8);
    L->twy = same_plan ? L->twx : take((size_t)ny * 8);
    L->tice = K > 0 && K <= TICE_MAX ? take((size_t)K * 8) : -1;
    L->P1 = take(capU * rowf * 2);
    const size_t f = al16(np * rowf * 2);
    size_t scratch = al16((size_t)2 * B_cols * (ny + 1) * 8);
    const size_t others[] = {ws_cols(ny, B_cols), ws_conv_rows(Mx, h_conv), ws_conv_cols(My, B_conv)};
    for (size_t q : others) scratch = q > scratch ? q : scratch;
    // moments of the whole tile at once where they fit, else of an even number of rows at a time
    size_t ms = 0;
    for (L->chunk = h;; L->chunk = (L->chunk / 2 + 1) / 2 * 2) {
        ms = al16(3 * capM_of(L->chunk) * rowf);
        const size_t fft = al16(npi * rowf * 2);
        ms = fft > ms ? fft : ms;
        if (ms + f < scratch) ms = al16(scratch - f);
        if (off + ms + f <= budget) break;
        if (L->chunk <= 2) return false;
    }
    L->MS = take(ms);
    L->F = take(f);
    auto opt = [&](size_t bytes) -> int { return off + al16(bytes) <= budget ? take(bytes) : -1; };
    // in order of what a place in shared memory saves
    L->P0 = opt(capU * rowf * 2);
    L->KA0 = L->KA1 = -1;
    if (off + 2 * al16(capU * rowf) <= budget) {
        L->KA0 = take(capU * rowf);
        L->KA1 = take(capU * rowf);
    }
    L->KB = opt(capU * rowf);
    L->D = opt(capM_of(h) * rowf);
    L->KC = opt(h * rowf);
    L->visc = opt(h * rowf);
    L->mult = ncols <= grid ? opt((size_t)B_cols * ny * 4) : -1;
    L->ue = L->dz = L->Ha = L->Hb = -1;
    if (off + 2 * al16(h * rowf) <= budget) {
        L->ue = take(h * rowf);
        L->dz = take(h * rowf);
    }
    if (off + 2 * al16(h * rowf) <= budget) {
        L->Ha = take(h * rowf);
        L->Hb = take(h * rowf);
    }
    L->bytes = (int)off;
    L->all = L->P0 >= 0 && L->KA0 >= 0 && L->KB >= 0 && L->KC >= 0 && L->D >= 0 && L->visc >= 0 && L->mult >= 0 &&
             L->ue >= 0 && L->Ha >= 0 && L->chunk >= h;
    return true;
}

// Compiled sequence pairs: the tuned schedules of the square grids 64, 96, 128, 192, 256 and 350
// (fi_resident_small.cu, fi_resident_large.cu: every buffer resident) and of 512 and 1024, whose
// tiles do not fit whole.
const void* resident_small(int seq);
const void* resident_large(int seq, int all);

const void* resident_kernel(int seqx, int seqy, int all) {
    const void* k = nullptr;
    if (seqx == seqy && seqx != 0) {
        if (all) k = resident_small(seqx);
        if (!k) k = resident_large(seqx, all);
    }
    if (k) return k;
    return all ? (const void*)k_resident<0, 0, 1> : (const void*)k_resident<0, 0, 0>;
}

}  // namespace fi
