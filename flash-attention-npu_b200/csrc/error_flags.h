// Plain C++, also compiled by a CPU test.
#pragma once

namespace fa {

// The first code that any of n error flags holds.  Every flag is read, and with `clear` reset, whatever the ones before it
// held: a kernel whose flag stays set leaves without writing its output.
inline int first_error(int (*const* flags)(bool), int n, bool clear) {
    int first = 0;
    for (int i = 0; i < n; ++i) {
        const int code = flags[i](clear);
        if (!first) first = code;
    }
    return first;
}

}  // namespace fa
