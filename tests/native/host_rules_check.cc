// Checks of csrc/host_rules.inl.  argv[1] names the check; exit status 0 = it held.
#include <cstdio>
#include <string>

#include "../../lmz_b200/csrc/host_rules.inl"

#define NEED(c)                                                          \
    do {                                                                 \
        if (!(c)) {                                                      \
            fprintf(stderr, "line %d: %s\n", __LINE__, #c);             \
            return 1;                                                    \
        }                                                                \
    } while (0)

static int size_classes()
{
    size_t last = 0, classes = 0;
    for (size_t n = 1; n < ((size_t)1 << 33); n += n / 37 + 1) {
        const size_t c = size_class(n);
        NEED(c >= n && c >= last && c % 4096 == 0);
        NEED(c <= n + n / 8 || c < n + 4096);
        NEED(size_class(c) == c && size_class(c + 1) > c);
        classes += c != last;
        last = c;
    }
    NEED(classes <= 8 * 34);
    for (int k = 12; k < 63; k++) NEED(size_class((size_t)1 << k) == (size_t)1 << k);
    for (size_t back = 0; back < 3; back++) NEED(size_class(SIZE_MAX - back) >= SIZE_MAX - back);
    NEED(size_class(((size_t)1 << 63) + 1) > (size_t)1 << 63);
    return 0;
}

int main(int argc, char **argv)
{
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "size classes") return size_classes();
    fprintf(stderr, "no such check\n");
    return 2;
}
