// sweep_scratch_bytes for an image of plain numbers.
#include "iwpp_engine.cuh"

extern "C" __attribute__((visibility("default"))) size_t scratch_bytes(size_t marker, size_t mask, long long pitch,
                                                                      int w, int h, int dtype, int conn) {
    iwpp::ImgDesc d{};
    d.marker = reinterpret_cast<unsigned char*>(marker);
    d.mask = reinterpret_cast<const unsigned char*>(mask);
    d.pitch_m = d.pitch_k = pitch;
    d.W = w;
    d.H = h;
    d.dtype = dtype;
    d.conn = conn;
    return iwpp::sweep_scratch_bytes(d);
}
