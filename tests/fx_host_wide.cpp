// The line transforms of fx_host.cpp with eight pairs per block (the layout
// that fx_lines chooses where it fills the warps better).
#include "fx_host.cpp"

extern "C" void fx_line_wide(int n, int inverse, int, const double *a, const double *b, double *oa, double *ob)
{
    if (first_radix(n) == 8) line<8, 3>(n, inverse, a, b, oa, ob);
    else line<4, 3>(n, inverse, a, b, oa, ob);
}
