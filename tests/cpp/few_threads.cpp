// Preloaded library: pthread_create fails once gnd_test_threads more threads have been started
// (-1: any number).
#include <dlfcn.h>
#include <pthread.h>

#include <cerrno>

extern "C" {
int gnd_test_threads = -1;

int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* arg) {
    if (gnd_test_threads == 0) return EAGAIN;
    if (gnd_test_threads > 0) --gnd_test_threads;
    using Create = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
    return reinterpret_cast<Create>(dlsym(RTLD_NEXT, "pthread_create"))(t, a, f, arg);
}
}
