// How many images of a batch one launch takes whose kernel counts their rows,
// `rows` an image, in an int (a 64-bit row index would cost it a 64-bit
// division a thread).
#pragma once
#include <limits.h>

inline int images_per_launch(int images, long long rows) {
    const long long most = rows > 0 ? INT_MAX / rows : INT_MAX;
    const long long n = images < most ? images : most;
    return n > 1 ? (int)n : 1;
}
