// The mixed variant's plasticity update (precompute<float, double>) against the FP64 one on the
// same FP32 inputs, over yield limits [cy, sy] and families of singular values. Every sample
// counts; whether it must yield is the FP64 side's to say. Per limits and family, "name value"
// pairs in units of 2^-24, a NaN kept: err, the largest difference of Fe and, where FP64
// clamps, of Re (absolute, over max(1, sy)) and of Jp and Je (relative); rot, the largest
// difference of Re where it does not; and yields, the share of samples that FP64 clamps.
#include "mpm_math.cuh"
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>

using namespace mpm;

static void rotation(std::mt19937_64& g,double* R)
{
    std::normal_distribution<double> n(0.,1.);
    double w=n(g),x=n(g),y=n(g),z=n(g);
    const double s=1./std::sqrt(w*w+x*x+y*y+z*z);w*=s;x*=s;y*=s;z*=s;
    const double M[9]={1-2*(y*y+z*z),2*(x*y-w*z),2*(x*z+w*y),2*(x*y+w*z),1-2*(x*x+z*z),2*(y*z-w*x),2*(x*z-w*y),2*(y*z+w*x),1-2*(x*x+y*y)};
    std::memcpy(R,M,sizeof(M));
}
static void worst(double& a,double b){if(!(b<=a)) a=b;}

int main()
{
    const struct {const char* name;double cy,sy;} limits[]={{"snow",.975,1.0075},{"wide",.5,2.},{"rigid",.99995,1.00005},{"point",1.,1.},
                                                            {"low",.6,.8},{"high",1.2,1.5},{"crossed",1.05,.95}};
    const char* names[]={"mixed_sides","lower","upper","pair","spread","inverted"};
    for(const auto& L:limits) for(int mode=0;mode<6;++mode){
        const float cy=(float)L.cy,sy=(float)L.sy;
        std::mt19937_64 g(17+mode);
        std::uniform_real_distribution<double> u(-1.,1.);
        double err=0,rot=0;int yields=0;const int N=4000;
        for(int it=0;it<N;++it){
            double A[9],B[9],s[3],F[9];
            rotation(g,A);rotation(g,B);
            for(double& x:s){
                const double r=u(g);
                x=mode==0?.5*(cy+sy)*(1+.05*r):mode==1?cy+3e-7*r:mode==2?sy+3e-7*r:mode==3?1+.1*r:std::exp(1.2*r);}
            if(mode==3) s[1]=s[0]+1e-7*u(g);
            if(mode==5){s[0]=1.1+.2*u(g);s[1]=1.1+.2*u(g);s[2]=-.6+.2*u(g);}
            for(int i=0;i<3;++i) for(int j=0;j<3;++j) F[3*i+j]=A[3*i]*s[0]*B[3*j]+A[3*i+1]*s[1]*B[3*j+1]+A[3*i+2]*s[2]*B[3*j+2];
            float Fm[9],Rm[9],lam,mu,Je,Jp=1.f+.1f*(float)u(g);
            double Fx[9],Rx[9],lx,mx,Jx,Jq=Jp;
            for(int k=0;k<9;++k){Fm[k]=(float)F[k];Fx[k]=Fm[k];}
            precompute<float,double>(Fm,Jp,1e4f,2e4f,1,0.f,cy,sy,10.f,Rm,lam,mu,Je);
            precompute<double,double>(Fx,Jq,1e4,2e4,1,0.,(double)cy,(double)sy,10.,Rx,lx,mx,Jx);
            bool clamps=false;
            for(int k=0;k<9;++k) clamps|=Fx[k]!=(double)(float)F[k];
            yields+=clamps;
            const double unit=std::ldexp(1.,24),big=std::fmax(1.,(double)sy);
            worst(err,std::fabs(Jp-Jq)/std::fabs(Jq)*unit);worst(err,std::fabs(Je-Jx)/std::fabs(Jx)*unit);
            for(int k=0;k<9;++k){worst(err,std::fabs(Fm[k]-Fx[k])/big*unit);worst(clamps?err:rot,std::fabs(Rm[k]-Rx[k])*unit);}}
        std::printf("%s_%s_err %.4f %s_%s_rot %.4f %s_%s_yields %.4f ",L.name,names[mode],err,L.name,names[mode],rot,L.name,names[mode],yields/(double)N);}
    // near a rotation (polar_near): Re and Je, and the share of samples that it takes
    for(int mode=0;mode<3;++mode){
        std::mt19937_64 g(41+mode);
        std::uniform_real_distribution<double> u(-1.,1.);
        const double strain=mode==0?1e-7:mode==1?1e-3:0.007;
        double err=0;int taken=0;const int N=8000;
        for(int it=0;it<N;++it){
            double A[9],B[9],s[3],F[9];
            rotation(g,A);rotation(g,B);
            for(double& x:s) x=1+strain*u(g);
            for(int i=0;i<3;++i) for(int j=0;j<3;++j) F[3*i+j]=A[3*i]*s[0]*B[3*j]+A[3*i+1]*s[1]*B[3*j+1]+A[3*i+2]*s[2]*B[3*j+2];
            float Ff[9],R[9],Rm[9],lam,mu,Je,Jp=1.f;double Fx[9],Rx[9],lx,mx,Jx,Jq=1.;
            for(int k=0;k<9;++k){Ff[k]=(float)F[k];Fx[k]=Ff[k];}
            if(!polar_near(Ff,POLAR_SERIES_MAX*POLAR_SERIES_MAX,R)) continue;
            ++taken;
            precompute<float,double>(Ff,Jp,1e4f,2e4f,0,0.f,.975f,1.0075f,10.f,Rm,lam,mu,Je);
            precompute<double,double>(Fx,Jq,1e4,2e4,0,0.,.975,1.0075,10.,Rx,lx,mx,Jx);
            worst(err,std::fabs(Je-Jx)*std::ldexp(1.,24));
            for(int k=0;k<9;++k){worst(err,std::fabs(R[k]-Rx[k])*std::ldexp(1.,24));worst(err,std::fabs(Rm[k]-Rx[k])*std::ldexp(1.,24));}}
        const char* n=mode==0?"series_rigid":mode==1?"series_light":"series_limit";
        std::printf("%s_err %.4f %s_taken %.4f ",n,err,n,taken/(double)N);}
    std::printf("\n");
    return 0;
}
