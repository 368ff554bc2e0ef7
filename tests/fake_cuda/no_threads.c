/* Preloaded: a system that has no more threads to give (the limit on a user's processes does not hold for root). */
#include <errno.h>
int pthread_create(void *t, const void *a, void *(*f)(void *), void *x) {
    (void)t;
    (void)a;
    (void)f;
    (void)x;
    return EAGAIN;
}
