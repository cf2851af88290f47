// The single post passes' tap positions on the host: how many pixels of a w x h image take their taps without
// clamps, and how many of those have a tap whose four texels are not inside by a quarter of the margin (or whose
// position is NaN): what is left of it is for the roundings another compiler would make.
#include "post_taps.h"

namespace {

struct Checked {
    float w, h;
    mutable bool bad;
    float operator()(float u, float v) const {
        const float x = u * w - 0.5f, y = v * h - 0.5f;
        const float mx = w / 4194304.0f, my = h / 4194304.0f;
        if (!(x >= mx && x < w - 1.0f - mx && y >= my && y < h - 1.0f - my)) bad = true;
        return 0.0f;
    }
};

}  // namespace

extern "C" void scan_god_rays(int w, int h, float sun_x, float sun_y, long long* inside, long long* bad) {
    const mm::post::TapArea area{(float)w, (float)h};
    *inside = *bad = 0;
    for (int y = 0; y < h; ++y)
        for (int x = 0; x < w; ++x) {
            float px, py, u, v;
            mm::post::frag(x, y, w, h, &px, &py, &u, &v);
            if (!mm::post::god_ray_inside(area, sun_x, sun_y, px, py)) continue;
            Checked taps{(float)w, (float)h, false};
            mm::post::god_ray_term(sun_x, sun_y, taps, px, py, 0.0f);
            ++*inside;
            *bad += taps.bad;
        }
}

extern "C" void scan_radial(int w, int h, float sun_x, float sun_y, long long* inside, long long* bad) {
    const mm::post::TapArea area{(float)w, (float)h};
    *inside = *bad = 0;
    for (int y = 0; y < h; ++y)
        for (int x = 0; x < w; ++x) {
            float px, py, u, v;
            mm::post::frag(x, y, w, h, &px, &py, &u, &v);
            if (!mm::post::radial_inside(area, sun_x, sun_y, px, py)) continue;
            Checked taps{(float)w, (float)h, false};
            mm::post::radial_term(sun_x, sun_y, taps, px, py);
            ++*inside;
            *bad += taps.bad;
        }
}
